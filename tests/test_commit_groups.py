"""Which column sizes of a tree are transformed together before they are hashed (the header's rule, as host code): small ones in one go, so that
the tree's launches follow one another; large ones by themselves."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zk_inference_prover_b200", "csrc", "host")
LIMIT = 1 << 13


@pytest.fixture(scope="module")
def group(tmp_path_factory):
    d = tmp_path_factory.mktemp("groups")
    src, so = d / "g.cpp", d / "g.so"
    src.write_text('#include "commit_groups.hpp"\nextern "C" size_t group(const size_t* words, size_t n) { return zk::commit_group(words, n); }\n')
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.group.restype = ctypes.c_size_t
    return lambda words: lib.group((ctypes.c_size_t * len(words))(*words), ctypes.c_size_t(len(words)))


@pytest.mark.parametrize("words,want", [([2 << 7, 1 << 6, 1 << 5], 3),  # a tree of ten columns of 2^6 ... 2^4 rows over three trees
                                       ([1], 1), ([LIMIT], 1), ([LIMIT - 1, 1], 2), ([LIMIT, 1], 1), ([LIMIT // 2, LIMIT // 2, 1], 2),
                                       ([1 << 28, 1, 1], 1), ([16, LIMIT, 16], 1)])
def test_small_sizes_are_a_group(group, words, want):
    assert group(words) == want


def test_every_size_is_in_one_group(group):
    words, at, sizes = [3 << k for k in range(24, 3, -1)], 0, []
    while at < len(words):
        sizes.append(group(words[at:]))
        assert sizes[-1] == 1 or sum(words[at:at + sizes[-1]]) <= LIMIT
        at += sizes[-1]
    assert at == len(words) and sizes[0] == 1 and sizes[-1] > 6
