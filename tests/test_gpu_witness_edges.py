"""The witness generators at the sizes and layouts where they change how they run, cell for cell against the oracle: groups of more
than 256 rows and more groups than a thread block has threads, weights that can be loaded sixteen at a time and at no alignment,
residual-stream columns evenly spaced in one allocation, enough rows for two teams of warps, more columns than fit shared memory."""
import numpy as np
import pytest

from test_freivalds import test_freivalds_device_matches_oracle as freivalds_matches_oracle
from test_witness_gen import run_dequant
from test_witness_gen import test_dequant_matches_oracle as dequant_matches_oracle
from test_witness_pre import run_residual_stream
from zk_inference_prover_b200 import witness_cases as wc
from zk_inference_prover_b200.witness_cases import dequant_case

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


@pytest.mark.parametrize("log_rows,kmax,change", [(6, 21, None), (5, 13, "table"), (5, 13, "operands"), (14, 13, None)])
def test_residual_stream_wide_values(ctx, oracle, log_rows, kmax, change):
    """Tables too large for a counter a row; table rows and operands that 32 bits do not hold the sum of; rows for more passes than teams."""
    case = wc.residual_stream_case(5 + log_rows, "pairs", 16, log_rows, (1 << log_rows) - 3, un=(1, 2) if change == "operands" else (0, 0), kind=0, sticky=True, kmax=kmax, spread=9)
    rng = np.random.default_rng(log_rows)
    if change == "table":
        rows = case["norm3"].reshape(-1, 3)
        at = rng.integers(1, len(rows), len(rows) // 2)
        rows[at, rng.integers(0, 3, at.size)] = rng.choice(np.array([255, 256, 65535, 65536, 1 << 20], np.uint32), at.size)
    if change == "operands":
        for images in case["un2"]:
            at = rng.integers(0, images.size, images.size // 2)
            images[at] = rng.choice(np.array([0, 131071, 131072, -131072, -131073, 1 << 20, (1 << 30) - 1, -(1 << 29)], np.int64), at.size)
            images[1::2] = rng.choice(np.array([0, 1, 254, 300, (1 << 20) - 1, 1 << 20, 1 << 29], np.int64), images.size // 2)
    got, want = run_residual_stream(ctx, case), oracle.witness_residual_stream(case)
    for k in want:
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("variant,per_row,kmax,wide_row", [(1, 7, 16, False), (1, 8, 13, False), (1, 8, 13, True), (0, 16, 13, False)])
def test_dequant_tables_in_shared_memory(ctx, oracle, variant, per_row, kmax, wide_row):
    """Slots enough a thread block for the tables to be brought there; a row that does not fit a word keeps them in memory."""
    case = dequant_case(7 + per_row, variant, 256, 256, per_row, kmax, 1, 0, False)
    if wide_row:
        case["norm3"].reshape(-1, 3)[300] = (256, 65536, 1)
    got = run_dequant(ctx, case)
    want = oracle.witness_dequant(case["acc"], case["jx"], case["jw"], case["sx"], case["sw"], case["norm3"], case["mul2"], case["n_base"], case["n_pre"], case["cfg"])
    want["want"][:] = 0
    for k in ("counts", "m_norm", "m_frac", "m_mul", "m_r8", "pre", "base"):
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("kmax", [14, 16, 19])
def test_dequant_tables_beside_the_counters(ctx, oracle, kmax):
    """Both tables in shared memory beside fraction counters that two and more rows share."""
    case = dequant_case(40 + kmax, 1, 256, 256, 16, kmax, 1, 0, False)
    got = run_dequant(ctx, case)
    want = oracle.witness_dequant(case["acc"], case["jx"], case["jw"], case["sx"], case["sw"], case["norm3"], case["mul2"], case["n_base"], case["n_pre"], case["cfg"])
    want["want"][:] = 0
    for k in ("counts", "m_norm", "m_frac", "m_mul", "m_r8", "pre", "base"):
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("n", [11, 12])
@pytest.mark.parametrize("kmax,sticky,even", [(13, True, None), (13, False, True), (16, True, False), (16, False, None)])
def test_residual_stream_around_the_fraction_counters(ctx, oracle, n, kmax, sticky, even):
    """352 and 384 additions a thread block: fewer and more counters of the fraction table, shared by several rows and one each."""
    case = wc.residual_stream_case(90 + n + kmax, "pairs", n, 5, 32, kind=0, sticky=sticky, kmax=kmax, spread=9)
    got, want = run_residual_stream(ctx if even is None else _EvenColumns(ctx, 32, case["n_cols"], even), case), oracle.witness_residual_stream(case)
    for k in want:
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("even", [None, False, True])
@pytest.mark.parametrize("shape,n,log_rows,live_rows,kind,sticky,spread", [("tree", 40, 4, 16, 0, True, 20), ("tree", 40, 2, 3, 0, False, 20), ("pairs", 8, 1, 2, 1, True, 9)])
def test_residual_stream_of_fewer_rows_than_lanes(ctx, oracle, even, shape, n, log_rows, live_rows, kind, sticky, spread):
    """Over several levels of additions, whose barriers take whole warps."""
    test_residual_stream_edges(ctx, oracle, even, shape, n, log_rows, live_rows, kind, sticky, spread)
