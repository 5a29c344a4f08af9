"""Calls whose pointer tables take a large part of the staging ring (2^20 slots): every table of a call stays in place until the call's
kernels have read it, wherever in the ring the call before has left off, and a call whose tables do not fit together is refused."""
import numpy as np
import pytest

from util import m31_column

pytestmark = pytest.mark.gpu


def _columns(buf, n, words):
    return (np.uint64(buf.ptr) + np.uint64(4 * words) * np.arange(n, dtype=np.uint64)).tolist()


@pytest.mark.parametrize("n_cols", [1 << 17, 300001, 350000, 1 << 19])
def test_extension_of_many_columns_wherever_the_ring_stands(zkb, oracle, n_cols):
    ctx = zkb.Context(device=0, max_log_size=8)
    vals = m31_column(77, 4 * n_cols)
    src = ctx.upload(vals)
    outs = [ctx.alloc(8 * n_cols) for _ in range(2)]
    want = None
    for k in range(4):  # the source's table is found in the ring, or not; the destination's fits behind it, or not
        out = outs[k & 1].zero()
        ctx.lde_cols(_columns(src, n_cols, 4), 2, _columns(out, n_cols, 8), 3)
        got = out.download().reshape(n_cols, 8)
        if want is None:
            want = got
            some = [0, 1, n_cols // 2, n_cols - 1]
            assert (got[some] == oracle.evaluate_cols(vals.reshape(n_cols, 4)[some], 2, 3)).all()
        assert (got == want).all(), k
    ctx.close()


def test_more_columns_than_the_ring_holds_are_refused(zkb):
    ctx = zkb.Context(device=0, max_log_size=8)
    n = (1 << 19) + 1
    src, out = ctx.alloc(4 * n).zero(), ctx.alloc(8 * n).zero()
    with pytest.raises(zkb.ZkbError):
        ctx.lde_cols(_columns(src, n, 4), 2, _columns(out, n, 8), 3)
    assert not out.download().any()
    ctx.close()


def test_a_decommitment_of_more_columns_than_the_ring_takes_together(zkb, oracle):
    """600,001 columns of two sizes: each size's tables fit the ring, all of them do not, so the decommitment's plan brings them along."""
    logs = [[3] * 300000 + [2] * 300000, [4]]
    at = np.cumsum([0] + [1 << lg for tree in logs for lg in tree])
    vals, flat = m31_column(78, int(at[-1])), range(len(at) - 1)
    cols = [vals[at[i]:at[i + 1]] for i in flat]
    kw = dict(pow_bits=0, log_blowup=1, n_queries=2)
    want = oracle.pcs_prove([cols[:-1], cols[-1:]], **kw)
    ctx = zkb.Context(device=0, max_log_size=8)
    buf = ctx.upload(vals)
    ptrs = [buf.ptr + 4 * int(at[i]) for i in flat]
    got = ctx.pcs_prove_device([ptrs[:-1], ptrs[-1:]], [lg for tree in logs for lg in tree], **kw)
    assert len(got) == len(want) and (got == want).all()
    ctx.close()
