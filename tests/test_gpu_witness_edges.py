"""The witness generators at the sizes and layouts where they change how they run, cell for cell against the oracle: groups of more
than 256 rows and more groups than a thread block has threads, weights that can be loaded sixteen at a time and at no alignment,
residual-stream columns evenly spaced in one allocation, enough rows for two teams of warps, more columns than fit shared memory."""
import numpy as np
import pytest

from test_freivalds import test_freivalds_device_matches_oracle as freivalds_matches_oracle
from test_witness_gen import test_dequant_matches_oracle as dequant_matches_oracle
from test_witness_pre import run_residual_stream
from zk_inference_prover_b200 import witness_cases as wc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,n_in,n_outs,chunks", [(3, 5, [64, 48], 4), (2, 3, [514, 513], 257), (5, 4, [899], 300), (1, 1200, [7, 5], 1),
                                                      (2, 2, [33, 1], 256), (7, 2049, [18], 2), (1, 1, [3], 2)])
def test_freivalds_edges(ctx, oracle, tokens, n_in, n_outs, chunks):
    freivalds_matches_oracle(ctx, oracle, tokens, n_in, n_outs, chunks)


class _EvenColumns:
    """A context whose allocations of one size lie in one buffer, a fixed distance apart."""

    def __init__(self, ctx, words, count, descending):
        self._ctx, self._words, self._left = ctx, words, list(range(count))
        self._buf, self._down = ctx.alloc(words * count).zero(), descending

    def __getattr__(self, name):
        return getattr(self._ctx, name)

    def alloc(self, words):
        if words != self._words or not self._left:
            return self._ctx.alloc(words)
        at = self._left.pop(-1 if self._down else 0)
        outer = self

        class View:
            ptr = outer._buf.view(at * words)

            def zero(self):
                return self

            def download(self):
                return outer._buf.download()[at * words:(at + 1) * words]

        return View()


@pytest.mark.parametrize("even", [None, False, True])
@pytest.mark.parametrize("shape,n,log_rows,live_rows,kind,sticky,spread", [("pairs", 8, 13, 8000, 0, True, 130), ("pairs", 8, 13, 8192, 1, True, 30),
                                                                         ("tree", 40, 12, 4096, 0, False, 100), ("pairs", 4, 3, 7, 0, True, 9)])
def test_residual_stream_edges(ctx, oracle, even, shape, n, log_rows, live_rows, kind, sticky, spread):
    pad = 64 if shape == "tree" else None
    case = wc.residual_stream_case(77 + n + log_rows, shape, n, log_rows, live_rows, pad=pad, un=(0, 0), kind=kind, sticky=sticky, kmax=13, spread=spread)
    c = ctx if even is None else _EvenColumns(ctx, 1 << log_rows, case["n_cols"], even)
    got, want = run_residual_stream(c, case), oracle.witness_residual_stream(case)
    for k in want:
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("variant,tokens,chunks,per_row", [(1, 4, 4, 330), (0, 2, 4, 500), (1, 64, 64, 1)])
def test_dequant_edges(ctx, oracle, variant, tokens, chunks, per_row):
    dequant_matches_oracle(ctx, oracle, variant, tokens, chunks, per_row, 16, 1, 1, False)
