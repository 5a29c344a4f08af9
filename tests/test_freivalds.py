"""The Freivalds attention-witness component: columns (scatter) and Horner accumulators.

CPU: the oracle's restatement of prover/src/gadgets/freivalds/{trace,claims}.rs is pinned to the
identity the component exists to prove: the claim of matrix m equals
sum_{t,i} s^t rv^i (X W_m)[t, i] with the integer product X W_m computed independently.
GPU: zkb_freivalds_scatter / zkb_freivalds_acc against the oracle, every cell."""
import numpy as np
import pytest

from util import P, qm31_array


def layout(n_in, n_out_max, tokens, chunks):
    """FreivaldsLayout for a given chunk count (prover/src/gadgets/freivalds/layout.rs:22-46)."""
    pk = -(-n_out_max // chunks)
    pq = -(-tokens // chunks)
    rows = n_in * chunks
    log_rows = max(4, (rows - 1).bit_length())
    return (log_rows, n_in, chunks, (1 << log_rows) - rows), pq, pk


def _case(seed, tokens, n_in, n_outs):
    rng = np.random.default_rng(seed)
    qx = rng.integers(-128, 128, (tokens, n_in), dtype=np.int8)
    qws = [rng.integers(-128, 128, (n_in, no), dtype=np.int8) for no in n_outs]
    return qx, qws


def _qm31_pow_sum(oracle, coeffs_2d, s, rv):
    """sum_{t,i} s^t rv^i c[t,i] over QM31 for an integer matrix c."""
    acc = np.zeros(4, np.uint32)
    sp = oracle.secure_powers(s, coeffs_2d.shape[0])
    rp = oracle.secure_powers(rv, coeffs_2d.shape[1])
    for t in range(coeffs_2d.shape[0]):
        row = np.zeros(4, np.uint32)
        for i in range(coeffs_2d.shape[1]):
            c = int(coeffs_2d[t, i]) % P
            term = oracle.qm31_mul(rp[i], [c, 0, 0, 0])
            row = ((row.astype(np.uint64) + term) % P).astype(np.uint32)
        acc = ((acc.astype(np.uint64) + oracle.qm31_mul(sp[t], row)) % P).astype(np.uint32)
    return acc


@pytest.mark.parametrize("tokens,n_in,n_outs,chunks", [(5, 6, [7, 5], 4), (3, 8, [8], 2), (9, 4, [4, 6, 2], 3), (1, 16, [5], 1)])
def test_oracle_claims_are_the_freivalds_identity(oracle, tokens, n_in, n_outs, chunks):
    qx, qws = _case(11, tokens, n_in, n_outs)
    grid, pq, pk = layout(n_in, max(n_outs), tokens, chunks)
    base, pre, m_r8, off = oracle.freivalds_columns(qx, qws, grid, pq, pk)
    assert off == 0 and m_r8.sum() == pq << grid[0]
    s, rv = qm31_array(21, 1)[0], qm31_array(22, 1)[0]
    cols, claims = oracle.freivalds_acc(base, pre, len(qws), grid, pq, pk, s, rv)
    for m, w in enumerate(qws):
        y = qx.astype(np.int64) @ w.astype(np.int64)
        assert (claims[m] == _qm31_pow_sum(oracle, y, s, rv)).all()
    # the last committed row of acc_m carries the claim (coset row rows-1 sits at index coset_perm(rows-1))
    last = oracle.coset_perm((1 << grid[0]) - 1, grid[0])
    for m in range(len(qws)):
        assert (cols[8 + 8 * m:12 + 8 * m, last] == claims[m]).all()


# groups of 32 to 256 rows, a power of two (with and without lead rows), and what lies around that; then 2^19 rows, where the inner products go from two
# rows a thread to four at eight columns a matrix and from one tile of columns to two above 64, and where scan and split go in one with groups
# of 256 rows (the last two: with a quarter of lead rows, and a group more of them)
BLOCKS = [(5, 16, [70, 33], 32), (5, 15, [70], 32), (8, 12, [300], 64), (40, 100, [256, 100, 31], 256), (3, 17, [600], 128), (2, 20, [520], 512), (9, 8, [64], 32),
          (9, 60, [64], 33), (9, 2048, [1792, 100], 256), (300, 2047, [2048, 100], 256), (3, 2600, [8500], 128), (3, 1536, [300, 300, 20], 256), (3, 1535, [2048], 256)]


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,n_in,n_outs,chunks", BLOCKS)
def test_freivalds_device_matches_oracle_in_blocks(ctx, oracle, tokens, n_in, n_outs, chunks):
    test_freivalds_device_matches_oracle(ctx, oracle, tokens, n_in, n_outs, chunks)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,n_in,n_outs,chunks", [(5, 6, [7, 5], 4), (3, 8, [8], 2), (9, 4, [4, 6, 2], 3), (1, 16, [5], 1),
                                                      (32, 64, [64, 48, 64], 16), (17, 128, [96], 64)])
def test_freivalds_device_matches_oracle(ctx, oracle, tokens, n_in, n_outs, chunks):
    qx, qws = _case(12, tokens, n_in, n_outs)
    grid, pq, pk = layout(n_in, max(n_outs), tokens, chunks)
    rows = 1 << grid[0]
    n_mats = len(qws)
    want_base, want_pre, want_m, want_off = oracle.freivalds_columns(qx, qws, grid, pq, pk)
    d_qx = ctx.upload_bytes(qx)
    d_qw = [ctx.upload_bytes(w) for w in qws]
    base = [ctx.alloc(rows) for _ in range(pq)]
    pre = [ctx.alloc(rows) for _ in range(n_mats * pk + 4)]
    m_r8 = ctx.alloc(256).zero()
    off = ctx.alloc(2).zero()
    ctx.freivalds_scatter(d_qx.ptr, [w.ptr for w in d_qw], n_outs, grid, pq, pk, n_in, tokens, [b.ptr for b in base],
                          [p.ptr for p in pre], m_r8.ptr, 256, off.ptr)
    assert (np.stack([b.download() for b in base]) == want_base).all()
    assert (np.stack([p.download() for p in pre]) == want_pre).all()
    assert (m_r8.download() == want_m).all()
    assert int(off.download()[0]) == want_off
    s, rv = qm31_array(31, 1)[0], qm31_array(32, 1)[0]
    want_cols, want_claims = oracle.freivalds_acc(want_base, want_pre, n_mats, grid, pq, pk, s, rv)
    out = [ctx.alloc(rows) for _ in range((1 + 2 * n_mats) * 4)]
    claims = ctx.freivalds_acc([b.ptr for b in base], [p.ptr for p in pre[:n_mats * pk]], grid, pq, pk, n_mats, s, rv, [o.ptr for o in out])
    assert (np.stack([o.download() for o in out]) == want_cols).all()
    assert (claims == want_claims).all()


# 2^19 rows, 256 to a group: the one pass over scan and split with few lead rows, with almost half of them and with columns that it does not take, the
# four-row inner products with columns on 8 bytes and without; 2^20 rows; shorter groups. shift: words by which the columns miss 16 bytes
@pytest.mark.gpu
@pytest.mark.parametrize("tokens,n_in,n_outs,chunks,shift_in,shift_out", [
    (9, 1100, [2048, 300], 256, 0, 0), (300, 1025, [2048], 256, 2, 0), (3, 2049, [300], 256, 0, 0), (3, 2047, [2048], 256, 1, 0), (3, 2047, [2048], 256, 0, 1),
    (3, 1536, [2048, 2000], 256, 1, 1), (3, 1536, [2048], 256, 3, 2), (3, 4095, [1024], 128, 1, 2)])
def test_freivalds_accumulators_at_2_19_rows(ctx, oracle, tokens, n_in, n_outs, chunks, shift_in, shift_out):
    qx, qws = _case(13, tokens, n_in, n_outs)
    grid, pq, pk = layout(n_in, max(n_outs), tokens, chunks)
    rows, n_mats = 1 << grid[0], len(qws)
    base, pre, _, _ = oracle.freivalds_columns(qx, qws, grid, pq, pk)
    s, rv = qm31_array(33, 1)[0], qm31_array(34, 1)[0]
    want_cols, want_claims = oracle.freivalds_acc(base, pre, n_mats, grid, pq, pk, s, rv)

    def at(shift, words):  # on the device, `shift` words behind a 16-byte boundary, in one buffer
        buf = ctx.upload(np.concatenate([np.zeros(shift, np.uint32)] + [np.concatenate([w, np.zeros(4, np.uint32)]) for w in words]))
        return buf, [buf.ptr + 4 * (shift + k * (rows + 4)) for k in range(len(words))]

    keep_b, d_base = at(shift_in, base)
    keep_p, d_pre = at(shift_in, pre[:n_mats * pk])
    keep_o, d_out = at(shift_out, np.zeros_like(want_cols))
    ctx.profile_begin()
    claims = ctx.freivalds_acc(d_base, d_pre, grid, pq, pk, n_mats, s, rv, d_out)
    ran = ctx.profile_end()
    assert ("freivalds_scan_out_kernel" in ran) == (chunks == 256 and shift_out == 0)
    assert ("freivalds_inner_quad_kernel" in ran) == (pk >= 8 and shift_in % 2 == 0)
    assert (keep_o.download()[shift_out:].reshape(-1, rows + 4)[:, :rows] == want_cols).all()
    assert (claims == want_claims).all()
