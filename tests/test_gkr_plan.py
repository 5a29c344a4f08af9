"""How the batched GKR driver takes a layer's rounds, from their terms alone (the header's rule, as host code): rounds are taken ahead of
the transcript only where what that saves makes up for the large rounds among them."""
import ctypes
import os
import random
import subprocess
from collections import Counter

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zk_inference_prover_b200", "csrc")
GRID = 148


@pytest.fixture(scope="module")
def look_from(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, so = d / "p.cpp", d / "p.so"
    src.write_text('#include "gkr_batch.hpp"\nextern "C" int look_from(const size_t* terms, int n, unsigned grid) { return zk::gkr_look_from(terms, n, grid); }\n')
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    return lambda terms, grid=GRID: lib.look_from((ctypes.c_size_t * len(terms))(*terms), len(terms), grid)


def _layers(logs):
    """The terms of every round of every layer of a batch: an instance of 2^log fractions has layers of 1 ... log - 1 rounds."""
    of = sorted(Counter(logs).items())
    for n in range(1, max(logs)):
        # at this layer an instance has as many variables fewer than the tallest as it is shorter
        yield [sum(count for lg, count in of if n - (max(logs) - lg) >= n - j) << (n - j - 1) for j in range(n)]


def _pieces(terms, j, grid):
    return 8 * terms[j + 1] / (512 * (grid - 1)) if j + 1 < len(terms) else 0


@pytest.mark.parametrize("logs", [[16] + [14] * 500, [14] + [13] * 300, [16] + [10] * 500, [12] + [8] * 582, [16] * 3 + [13] * 60 + [11] * 200])
def test_no_large_rounds_ahead_where_shorter_instances_enter(look_from, logs):
    ahead = 0
    for terms in _layers(logs):
        first = look_from(terms)
        for j in range(first, len(terms)) if first >= 0 else ():
            assert _pieces(terms, j, GRID) <= 8, (terms, first, j)  # some 45,000 cycles, for 16,000 of an ordinary round
            ahead += 1
    assert ahead > 20  # the small rounds of the batch are


def test_rounds_that_only_fall_are_ahead_from_the_first_small_one(look_from):
    for terms in _layers([10 + i % 4 for i in range(34)]):
        if len(terms) >= 2:
            assert look_from(terms) == next(j for j, t in enumerate(terms) if 4 * t <= 2 * GRID * 512)
    assert look_from([1]) == -1 and look_from([2, 1]) == 0 and look_from([2, 1], grid=1) == -1
    assert look_from([1 << 20, 1 << 19]) == -1


def test_what_is_saved_makes_up_for_the_large_rounds(look_from):
    rng = random.Random(11)
    for _ in range(60):
        logs = [rng.randint(2, 22) for _ in range(rng.randint(1, 4))] + [rng.randint(2, 16)] * rng.choice([0, 1, 30, 300, 4000])
        grid = rng.choice([2, 20, 66, 132, 148])
        for terms in _layers(logs):
            first = look_from(terms, grid)
            if first < 0:
                continue
            assert 0 <= first <= len(terms) - 2
            cost = sum(max(9500, 4500 + 5000 * _pieces(terms, j, grid)) for j in range(first, len(terms)))
            assert cost <= 16000 * (len(terms) - first) + 1 + (10000 if first == 0 and len(terms) <= 16 else 0)  # (no table of eq then)
            # a sum of 16-bit halves takes 2^16 additions; a piece makes at most 64 of them to one counter
            assert all(64 * (_pieces(terms, j, grid) + 1) < 1 << 16 for j in range(first, len(terms)))


def test_the_table_of_eq_counts(look_from):
    """Ahead from the first round on a layer needs no table: worth a first round that alone is not, where the terms' indices are short enough."""
    halves = lambda *first: list(first) + [max(1, first[-1] >> k) for k in range(1, 15 - len(first) + 1)]
    assert look_from(halves(16384, 24576)) == 0 and look_from(halves(1024, 31232)) == 0
    assert look_from(halves(32768, 49152)) == 2  # too large even so
    assert look_from(halves(24576, 24576, 16384)) == 0
