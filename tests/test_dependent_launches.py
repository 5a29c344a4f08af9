"""Kernels that may start while the grid before them still runs (programmatic dependent launches): what that grid may be writing must not
be read through read-only loads, which are defined only for memory that nobody writes during the kernel. Read from the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zk_inference_prover_b200", "csrc")
# Tables that no kernel writes: the inverse twiddles, and what the host staged before the chain (column addresses, a proof's layers).
TABLES = {"itw", "cols", "layers"}


def _kernels():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
            for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\((.*?)\)\s*\{(.*?)\n\}", text, flags=re.S):
                yield name, m.group(1), m.group(2), m.group(3)


DEPENDENT = [k for k in _kernels() if "follow_previous()" in k[3] or "griddepcontrol.wait" in k[3]]


def test_the_dependent_kernels_are_found():
    assert {k[1] for k in DEPENDENT} >= {"merkle_layer_quad_kernel", "merkle_levels_kernel", "merkle_top_kernel", "fold_line_kernel2", "fold_line_kernel4",
                                        "fold_circle_kernel2", "fold_circle_kernel4", "tower_kernel", "res_round_kernel", "res_chain_kernel"}
    text = "".join(open(os.path.join(CSRC, f)).read() for f in os.listdir(CSRC) if f.endswith(".cu"))
    launched = set(re.findall(r"launch_following\(ctx, (\w+)", text)) | set(re.findall(r'launch\.run\("[^"]*", (\w+)', text))
    assert launched <= {k[1] for k in DEPENDENT}


@pytest.mark.parametrize("kernel", DEPENDENT, ids=lambda k: k[1])
def test_plain_loads_of_what_the_grid_before_may_write(kernel):
    _, name, params, body = kernel
    read_only = {p.split()[-1] for p in re.split(r",\s*", params) if re.search(r"const\b.*\*\s*__restrict__", p)}
    assert read_only <= TABLES, (name, read_only - TABLES)
    for arg in re.findall(r"__ldg\((.*)", body):
        assert any(t in arg for t in TABLES), (name, arg)
