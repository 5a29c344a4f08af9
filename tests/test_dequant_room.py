"""What the dequantize kernel wants in a thread block's shared memory, from its sources: the normalisation and the product table have room beside the
counters at every accumulator window that its components use."""
import os
import re

import pytest

from zk_inference_prover_b200.witness_cases import dequant_case, mul_table, norm_table

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zk_inference_prover_b200", "csrc", "witness_gen.cu")).read()
LOGS = {k: int(v) for k, v in re.findall(r"(DEQ_(?:NORM|FRAC|MUL)_LOG) = (\d+)", SRC)}


@pytest.mark.parametrize("kmax", [13, 14, 16, 19, 22])
@pytest.mark.parametrize("per_row", [4, 16, 32])
def test_tables_of_the_chain_variant_have_room(kmax, per_row):
    cfg = dequant_case(1, 1, tokens=1, chunks=2, per_row=per_row, kmax=kmax)["cfg"]
    counters = sum(4 << LOGS[k] for k in ("DEQ_NORM_LOG", "DEQ_FRAC_LOG", "DEQ_MUL_LOG")) + 4 * cfg["n_r8"]
    pointers = 8 * per_row * (cfg["per_slot"] + cfg["chan_w"])
    assert counters + pointers + 4 * len(norm_table(kmax, 1)) + 2 * len(mul_table()) <= 227 * 1024
