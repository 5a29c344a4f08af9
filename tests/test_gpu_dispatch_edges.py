"""Proofs at the sizes where the library changes how it runs them, word for word against the oracle: FRI layers that fit the
one-launch tail (2^10 values), those that many thread blocks take in one launch (2^15) and those above, last layers it interpolates and those it leaves to the host; GKR instances around
the layer sizes one CTA takes (2^13 entries), passes of one term per lane, of several and of more than the small form's limit;
batches whose towers take one launch (2^10 entries) and two; samples whose quotient lines are worked out on the host and on the
device (from 512 on, in pieces of 1,024); trees hashed on a second stream, quotients planned on a second thread, decommitments of a few
cells and of many; a few instances on both sides of the choice of driver."""
import numpy as np
import pytest

from util import m31_column, qm31_array
from zk_inference_prover_b200 import ZkbError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n", [1, 2, 3, 8, 9, 10, 11])
@pytest.mark.parametrize("kw", [
    dict(pow_bits=4, log_blowup=1, log_last_layer=0, n_queries=3),
    dict(pow_bits=0, log_blowup=2, log_last_layer=2, n_queries=5),
    dict(pow_bits=6, log_blowup=1, log_last_layer=3, n_queries=2),
    dict(pow_bits=1, log_blowup=4, log_last_layer=2, n_queries=4),
])
def test_pcs_proof_around_the_fri_tail(ctx, oracle, log_n, kw):
    if log_n < kw["log_last_layer"] + 1:
        pytest.skip("the last layer would be larger than the first fold")
    trees = [[m31_column(6000 + 10 * log_n + c, 1 << log_n) for c in range(3)]]
    want = oracle.pcs_prove(trees, **kw)
    got = ctx.pcs_prove_host(trees, **kw)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("log_n", [1, 2, 3, 6, 7, 8, 9, 10, 12, 13, 14, 15])
def test_gkr_single_instance_around_the_chain(ctx, oracle, kind, log_n):
    if kind == 2 and log_n == 1:
        pytest.skip("a multiplicities layer of two entries is not an input the protocol has")
    n = 1 << log_n
    den = qm31_array(7000 + log_n, n, nonzero=True)
    num = qm31_array(7100 + log_n, n) if kind == 1 else m31_column(7200 + log_n, n) if kind == 2 else None
    want = oracle.gkr_prove([(kind, num, den)], 0x5EED0004, verify=True)
    nb, db = ctx.upload(num) if num is not None else None, ctx.upload(den)
    got = ctx.gkr_prove_device([(kind, nb.ptr if nb else 0, db.ptr, n)], 0x5EED0004)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("kind,log_n,value", [(k, n, None) for k in (0, 1, 2, 3) for n in (4, 5, 11)] + [(0, 2, 1), (0, 7, 0), (0, 11, 1), (1, 3, 1), (1, 10, 1), (1, 11, 0)])
def test_gkr_single_instance_a_round_ahead(ctx, oracle, kind, log_n, value):
    """Layers that are taken whole, the one above them, and constant ones, whose round polynomials are of low degree or nothing."""
    n = 1 << log_n
    den = qm31_array(7000 + log_n, n, nonzero=True)
    num = qm31_array(7100 + log_n, n) if kind == 1 else m31_column(7200 + log_n, n) if kind == 2 else None
    if value is not None:
        den = np.zeros_like(den)
        den[:, 0] = value
        num = np.zeros_like(num) if num is not None else None
    want = oracle.gkr_prove([(kind, num, den)], 0x5EED0016, verify=True)
    nb, db = ctx.upload(num) if num is not None else None, ctx.upload(den)
    got = ctx.gkr_prove_device([(kind, nb.ptr if nb else 0, db.ptr, n)], 0x5EED0016)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("log_n,n_inst", [(5, 431), (5, 432), (5, 433), (9, 365), (9, 377)])
def test_gkr_batch_around_what_a_launch_carries(ctx, oracle, log_n, n_inst):
    """16 + 64 rounds + 4 instances words of a layer's description: 2,000 at most go with the launch, more are copied."""
    inst, dev, keep = [], [], []
    for i in range(n_inst):
        n = 1 << (log_n if i == 3 else 2 + i % 3)
        den = qm31_array(7300 + i, n, nonzero=True)
        inst.append((3, None, den))
        keep.append(ctx.upload(den))
        dev.append((3, 0, keep[-1].ptr, n))
    want = oracle.gkr_prove(inst, 0x5EED0017, verify=True)
    got = ctx.gkr_prove_device(dev, 0x5EED0017)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("spec", [{16: 1, 13: 40}, {14: 1, 11: 120, 3: 2}, {15: 2, 12: 30, 9: 300}])
def test_gkr_batch_with_rounds_that_grow(ctx, oracle, spec):
    """Shorter instances that enter make a round large again: small rounds, large ones and small ones in a layer, those ahead of the transcript last."""
    inst, dev, keep = [], [], []
    for log_n, count in spec.items():
        for i in range(count):
            n, kind = 1 << log_n, (3, 0, 1, 2)[len(inst) % 4]
            at = 7600 + 3 * len(inst)
            den = qm31_array(at, n, nonzero=True)
            num = qm31_array(at + 1, n) if kind == 1 else m31_column(at + 2, n) if kind == 2 else None
            inst.append((kind, num, den))
            keep += [ctx.upload(num) if num is not None else None, ctx.upload(den)]
            dev.append((kind, keep[-2].ptr if num is not None else 0, keep[-1].ptr, n))
    want = oracle.gkr_prove(inst, 0x5EED0018, verify=True)
    got = ctx.gkr_prove_device(dev, 0x5EED0018)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("log_n", [2, 9, 10, 11, 12])
def test_gkr_batch_around_the_tower_launches(ctx, oracle, log_n):
    inst, dev, keep = [], [], []
    for k, kind in enumerate([0, 3, 1, 2, 0, 3, 1]):  # more than the driver of a few instances takes
        n = 1 << max(1 + (kind == 2), log_n - k // 4 * (log_n - 1))
        den = qm31_array(7300 + 10 * log_n + k, n, nonzero=True)
        num = qm31_array(7400 + 10 * log_n + k, n) if kind == 1 else m31_column(7500 + 10 * log_n + k, n) if kind == 2 else None
        inst.append((kind, num, den))
        keep.append((ctx.upload(num) if num is not None else None, ctx.upload(den)))
        dev.append((kind, keep[-1][0].ptr if keep[-1][0] else 0, keep[-1][1].ptr, n))
    want = oracle.gkr_prove(inst, 0x5EED0005, verify=True)
    got = ctx.gkr_prove_device(dev, 0x5EED0005)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("n_cols", [382, 383, 2200])
def test_pcs_proof_around_the_line_kernel(ctx, oracle, n_cols):
    # 511, 512 entries (a column with two samples has three); more than 1,024 of a size; the last tree holds the tallest column
    trees = [[m31_column(6500 + c, 1 << (3 if c % 2 else 4)) for c in range(n_cols)], [m31_column(6400, 1 << 5)]]
    kw = dict(pow_bits=0, log_blowup=1, log_last_layer=0, n_queries=3, two_sample_every=6)
    want = oracle.pcs_prove(trees, **kw)
    got = ctx.pcs_prove_host(trees, **kw)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("log_n", [0, 1, 9, 10, 11, 12, 22])
@pytest.mark.parametrize("shift", [0, 1])
def test_eval_at_point_around_its_kernels(ctx, oracle, log_n, shift):
    # up to 2^10 coefficients a warp a column; above, chunks of 2^11 by 16-byte loads or, for columns that do not start on 16 bytes, folded
    n = 1 << log_n
    cols = [m31_column(6300 + 10 * log_n + c, n) for c in range(3)]
    at = [c * (n + 4 - n % 4) + shift for c in range(3)]
    flat = np.zeros(at[2] + n, np.uint32)
    for a, c in zip(at, cols):
        flat[a:a + n] = c
    buf, point = ctx.upload(flat), qm31_array(6390, 2).ravel()
    got = ctx.eval_at_point_cols([buf.ptr + 4 * a for a in at], log_n, point)
    assert (got == np.stack([oracle.eval_at_point(c, point) for c in cols])).all()


@pytest.mark.parametrize("shape,kw", [
    # a tree before the last whose short layers are a chain of 64 blocks of sixteen columns is hashed on a second stream: 63, 64, the first
    # of two, one whose layers are not all short
    ([[4] * 600 + [5] * 424, [6] * 8], dict(n_queries=20)),
    ([[4] * 608 + [5] * 416, [6] * 8], dict(n_queries=20)),
    ([[5] * 1100 + [3] * 40, [4] * 1100, [7] * 3], dict(pow_bits=2, log_blowup=2, n_queries=20, two_sample_every=7)),
    ([[4] * 3, [13] * 2 + [12] * 1040, [14]], dict(n_queries=5)),
    # 8,191 and 8,192 samples: from there on the quotient plan is made on another thread
    ([[4] * 8189, [5] * 2], dict(n_queries=3)),
    ([[4] * 8190, [5] * 2], dict(n_queries=3)),
    # a decommitment of more than 2^20 cells: a launch per block
    ([[7] * 8300, [8] * 2], dict(n_queries=250)),
])
def test_pcs_proof_of_many_device_columns(ctx, oracle, shape, kw):
    kw = {"pow_bits": 0, "log_blowup": 1, **kw}
    trees = [[m31_column(6700 + 100 * t + c, 1 << lg) for c, lg in enumerate(logs)] for t, logs in enumerate(shape)]
    want = oracle.pcs_prove(trees, **kw)
    flat = np.concatenate([c for t in trees for c in t])
    at = np.cumsum([0] + [len(c) for t in trees for c in t])
    for _ in range(2):  # the second pass finds tables, blocks and buffers of the first
        buf = ctx.upload(flat)
        ptrs = iter([buf.ptr + 4 * int(a) for a in at[:-1]])
        got = ctx.pcs_prove_device([[next(ptrs) for _ in t] for t in trees], [lg for t in shape for lg in t], **kw)
        assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("n_inst,log_n", [(2, 12), (2, 13), (3, 12), (3, 13), (4, 5)])
def test_gkr_few_instances_around_the_choice_of_driver(ctx, oracle, n_inst, log_n):
    inst, dev, keep = [], [], []
    for k in range(n_inst):
        kind, n = (3, 0, 1, 3)[k], 1 << (log_n - k)
        den = qm31_array(7600 + 10 * log_n + k, n, nonzero=True)
        num = qm31_array(7700 + 10 * log_n + k, n) if kind == 1 else None
        inst.append((kind, num, den))
        keep.append((ctx.upload(num) if num is not None else None, ctx.upload(den)))
        dev.append((kind, keep[-1][0].ptr if keep[-1][0] else 0, keep[-1][1].ptr, n))
    want = oracle.gkr_prove(inst, 0x5EED0006, verify=True)
    got = ctx.gkr_prove_device(dev, 0x5EED0006)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("child_log,levels", [(19, 9), (20, 3), (20, 4), (21, 9), (23, 7)])
def test_merkle_levels_around_the_split_launches(ctx, oracle, child_log, levels):
    # from 2^20 children on three levels a launch, the others in the next
    below = m31_column(7800 + child_log, 8 << child_log).reshape(-1, 8)
    buf = ctx.upload(below)
    outs = [ctx.alloc(8 << (child_log - j)) for j in range(1, levels + 1)]
    ctx.merkle_levels(child_log, buf.ptr, [o.ptr for o in outs])
    for j, o in enumerate(outs, 1):
        below = oracle.commit_on_layer(child_log - j, below, [], m31=True)
        assert (o.download(shape=(-1, 8)) == below).all(), j


@pytest.mark.parametrize("n_cols,log_n,blowup,shift,two", [(63, 19, 1, 0, 0), (64, 19, 1, 0, 0), (64, 18, 2, 0, 5), (64, 19, 1, 1, 0), (2100, 13, 2, 0, 0), (100, 19, 1, 2, 3)])
def test_pcs_proof_around_the_numerators_of_coefficients(ctx, oracle, n_cols, log_n, blowup, shift, two):
    # wide and tall groups' numerators come from the coefficients, unless these do not start on 16 bytes
    trees = [[m31_column(7900 + c, 1 << log_n) for c in range(n_cols)]]
    kw = dict(pow_bits=0, log_blowup=blowup, log_last_layer=0, n_queries=3, two_sample_every=two)
    want = oracle.pcs_prove(trees, **kw)
    buf = ctx.upload(np.concatenate([np.zeros(shift, np.uint32)] + trees[0]))
    got = ctx.pcs_prove_device([[buf.ptr + 4 * (shift + (c << log_n)) for c in range(n_cols)]], [log_n] * n_cols, **kw)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("log_n,n_cols", [(1, 40), (2, 31), (2, 32), (5, 600), (9, 33), (10, 1500), (13, 100), (19, 34)])
def test_numerators_split_over_columns(ctx, oracle, log_n, n_cols):
    # as long as the rows alone do not fill the GPU, in pieces of sixteen columns and more; 24 pieces are added up by eight warps
    cols = [m31_column(8000 + c, 1 << log_n) for c in range(n_cols)]
    point, values, rands = oracle.secure_circle_mul(24680), qm31_array(8101, n_cols), qm31_array(8102, n_cols)
    want, _ = oracle.quot_numerators(cols, point, np.arange(n_cols, dtype=np.uint32), values, rands)
    lc = np.stack([oracle.line_coeffs(point, values[k], rands[k]) for k in range(n_cols)])
    bufs, outs = [ctx.upload(c) for c in cols], [ctx.alloc(1 << log_n) for _ in range(4)]
    ctx.quot_numerators([b.ptr for b in bufs], log_n, np.arange(n_cols, dtype=np.uint32), lc[:, 1, :], lc[:, 2, :], [o.ptr for o in outs])
    assert (np.stack([o.download() for o in outs]) == want).all()


@pytest.mark.parametrize("n_acc", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("log_n", [3, 4, 9])
def test_quotients_combined_several_rows_a_thread(ctx, oracle, n_acc, log_n):
    accs = [([m31_column(8200 + 10 * a + q, 1 << (log_n - a % 3)) for q in range(4)], log_n - a % 3) for a in range(n_acc)]
    first, points = qm31_array(8300, n_acc), np.stack([oracle.secure_circle_mul(13579 + 977 * a) for a in range(n_acc)])
    want = oracle.quot_combine([np.stack(c) for c, _ in accs], first, points, log_n)
    keep = [[ctx.upload(x) for x in c] for c, _ in accs]
    outs = [ctx.alloc(1 << log_n) for _ in range(4)]
    ctx.quot_combine([b.ptr for k in keep for b in k], [lg for _, lg in accs], first, points, log_n, [o.ptr for o in outs])
    assert (np.stack([o.download() for o in outs]) == want).all()


@pytest.mark.parametrize("log_n,n_cols", [(14, 2), (15, 1), (15, 300), (16, 150), (17, 5), (17, 300), (18, 299)])
def test_eval_at_point_in_runs_of_chunks(ctx, oracle, log_n, n_cols):
    # one run of sixteen chunks a column, runs of sixteen, and of 32 and 64 where there are two for every SM
    cols = [m31_column(8400 + 7 * log_n + c, 1 << log_n) for c in range(n_cols)]
    bufs, point = [ctx.upload(c) for c in cols], qm31_array(8390, 2).ravel()
    got = ctx.eval_at_point_cols([b.ptr for b in bufs], log_n, point)
    assert (got == np.stack([oracle.eval_at_point(c, point) for c in cols])).all()


@pytest.mark.parametrize("log_n,n_cols", [(4, 3), (5, 1), (5, 33), (6, 17), (7, 9), (8, 5), (8, 700), (9, 2), (9, 301)])
@pytest.mark.parametrize("blowup", [1, 2, 4])
def test_transforms_of_short_columns(ctx, oracle, log_n, n_cols, blowup):
    # 2^5 to 2^9 words: a CTA a column and, of many columns, several to a warp, the last warp's not all there; extensions into that range and out of it
    vals = np.stack([m31_column(8600 + c, 1 << log_n) for c in range(n_cols)])
    cols = [ctx.upload(v) for v in vals]
    ctx.ifft_cols([c.ptr for c in cols], log_n)
    coeffs = oracle.interpolate_cols(vals, log_n)
    assert (np.stack([c.download() for c in cols]) == coeffs).all()
    outs = [ctx.alloc(1 << (log_n + blowup)) for _ in range(n_cols)]
    ctx.lde_cols([c.ptr for c in cols], log_n, [o.ptr for o in outs], log_n + blowup)
    assert (np.stack([o.download() for o in outs]) == oracle.evaluate_cols(coeffs, log_n, log_n + blowup)).all()


@pytest.mark.parametrize("with_prev", [False, True])
@pytest.mark.parametrize("log_size,ncols", [(0, 64), (3, 63), (3, 65), (4, 80), (5, 81), (6, 95), (7, 96), (13, 64), (13, 97), (14, 64), (2, 1000)])
def test_merkle_layers_of_many_columns(ctx, oracle, log_size, ncols, with_prev):
    # many columns: a warp brings the blocks of sixteen nodes; even and odd numbers of blocks, whole and partial last ones
    cols = [m31_column(8700 + c, 1 << log_size) for c in range(ncols)]
    prev = m31_column(8690, 16 << log_size).reshape(-1, 8) if with_prev else None
    bufs, pb, out = [ctx.upload(c) for c in cols], ctx.upload(prev) if with_prev else None, ctx.alloc(8 << log_size)
    for m31 in (False, True):
        ctx.merkle_layer(log_size, pb.ptr if pb else 0, [b.ptr for b in bufs], out.ptr, m31_out=m31)
        assert (out.download(shape=(-1, 8)) == oracle.commit_on_layer(log_size, prev, cols, m31=m31)).all()


@pytest.mark.parametrize("log_n,n_cols,runs", [(15, 1, True), (16, 39, False), (16, 40, True), (18, 9, False), (18, 10, True), (20, 2, False), (20, 3, True)])
def test_eval_at_point_where_runs_begin(ctx, oracle, log_n, n_cols, runs):
    # one run a column, or eighty runs of sixteen chunks
    cols = [m31_column(8450 + c, 1 << log_n) for c in range(n_cols)]
    bufs, point = [ctx.upload(c) for c in cols], qm31_array(8395, 2).ravel()
    ctx.profile_begin()
    got = ctx.eval_at_point_cols([b.ptr for b in bufs], log_n, point)
    assert ("eval_runs_kernel" in ctx.profile_end()) == runs
    assert (got == np.stack([oracle.eval_at_point(c, point) for c in cols])).all()


@pytest.mark.parametrize("log_size,ncols,chain", [(0, 95, False), (0, 96, True), (8, 95, False), (11, 95, False), (11, 96, True), (11, 129, True), (12, 1535, False),
                                                  (12, 1536, True), (13, 143, False), (13, 144, True)])
def test_merkle_layers_where_the_loader_warp_begins(ctx, oracle, log_size, ncols, chain):
    cols = [m31_column(9000 + c, 1 << log_size) for c in range(ncols)]
    bufs, out = [ctx.upload(c) for c in cols], ctx.alloc(8 << log_size)
    ctx.profile_begin()
    ctx.merkle_layer(log_size, 0, [b.ptr for b in bufs], out.ptr, m31_out=True)
    assert ("merkle_layer_chain_kernel" in ctx.profile_end()) == chain
    assert (out.download(shape=(-1, 8)) == oracle.commit_on_layer(log_size, None, cols, m31=True)).all()


@pytest.mark.parametrize("log_n,n_cols", [(1, 40), (2, 39), (2, 41), (13, 39), (13, 40), (16, 40), (17, 47), (17, 49), (18, 111), (18, 112)])
def test_numerators_where_the_split_begins(ctx, oracle, log_n, n_cols):
    # 40 entries; 48 and 112 where the rows leave room for four pieces and for two
    test_numerators_split_over_columns(ctx, oracle, log_n, n_cols)


@pytest.mark.parametrize("n_acc", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("log_n,row_begin,n_rows", [(16, 0, 1 << 16), (17, 0, 1 << 17), (18, 1 << 16, (1 << 17) + 2), (18, 1 << 16, (1 << 17) + 4), (18, 8, (1 << 17) - 2), (4, 8, 2)])
def test_quotients_of_many_rows_combined(ctx, oracle, n_acc, log_n, row_begin, n_rows):
    # from 2^17 rows on several a thread, a shard's rows too unless they are not a multiple of four
    import ctypes as C

    accs = [([m31_column(9100 + 10 * a + q, 1 << (log_n - a % 3)) for q in range(4)], log_n - a % 3) for a in range(n_acc)]
    first, points = qm31_array(9200, n_acc), np.stack([oracle.secure_circle_mul(24680 + 977 * a) for a in range(n_acc)])
    want = oracle.quot_combine([np.stack(c) for c, _ in accs], first, points, log_n)[:, row_begin:row_begin + n_rows]
    keep = [ctx.upload(x[row_begin >> (log_n - lg):]) for c, lg in accs for x in c]  # a shard holds its own rows
    outs = [ctx.alloc(n_rows) for _ in range(4)]
    ptrs = lambda bufs: (C.c_void_p * len(bufs))(*[b.ptr for b in bufs])
    logs = np.array([lg for _, lg in accs], np.int32)
    at = lambda a: np.ascontiguousarray(a).ctypes.data_as(C.c_void_p)
    first, points = np.ascontiguousarray(first, np.uint32), np.ascontiguousarray(points, np.uint32)
    ctx._check(ctx.lib.zkb_quot_combine_rows(ctx.h, C.c_int(n_acc), ptrs(keep), at(logs), at(first), at(points), C.c_int(log_n), C.c_size_t(row_begin), C.c_size_t(n_rows), ptrs(outs)))
    assert (np.stack([o.download() for o in outs]) == want).all()


@pytest.mark.parametrize("n_cols,log_n,blowup,shift,two", [(247, 17, 1, 0, 0), (248, 17, 1, 0, 0), (248, 17, 1, 1, 0), (248, 17, 1, 2, 3), (104, 18, 2, 0, 5)])
def test_pcs_proof_where_the_numerators_of_coefficients_begin(ctx, oracle, n_cols, log_n, blowup, shift, two):
    # 24 M words and 28 columns of evaluations saved: 248 columns of 2^17 at blow-up 2
    test_pcs_proof_around_the_numerators_of_coefficients(ctx, oracle, n_cols, log_n, blowup, shift, two)


@pytest.mark.parametrize("log_n,n_cols,short", [(5, 2047, False), (5, 2048, True), (6, 2051, True), (7, 2049, True), (8, 1023, False), (8, 1024, True), (9, 511, False), (9, 513, True)])
def test_transforms_where_short_columns_share_a_warp(ctx, oracle, log_n, n_cols, short):
    vals = np.stack([m31_column(9300 + c, 1 << log_n) for c in range(n_cols)])
    flat = ctx.upload(vals)
    ptrs = [flat.ptr + 4 * (c << log_n) for c in range(n_cols)]
    ctx.profile_begin()
    ctx.ifft_cols(ptrs, log_n)
    assert any("short" in name for name in ctx.profile_end()) == short
    coeffs = oracle.interpolate_cols(vals, log_n)
    assert (flat.download(shape=vals.shape) == coeffs).all()
    outs = ctx.alloc(n_cols << (log_n + 1))
    ctx.lde_cols(ptrs, log_n, [outs.ptr + 4 * (c << (log_n + 1)) for c in range(n_cols)], log_n + 1)
    assert (outs.download(shape=(n_cols, -1)) == oracle.evaluate_cols(coeffs, log_n, log_n + 1)).all()


@pytest.mark.parametrize("log_rows,kw", [(9, {}), (10, {}), (10, dict(log_last_layer=2)), (11, {}), (13, dict(log_last_layer=9)), (15, {}), (16, {}), (17, {}), (17, dict(log_last_layer=14))])
def test_fri_layers_of_many_ctas(ctx, oracle, log_rows, kw):
    """First layers of 2^10 ... 2^18 values: none, some and all of the middle ones in one launch, the last one above and below where that ends."""
    trees = [[m31_column(9100 + log_rows, 1 << log_rows), m31_column(9200, 1 << (log_rows - 3))], [m31_column(9300 + log_rows, 1 << log_rows)]]
    kw = dict(pow_bits=4, log_blowup=1, n_queries=9, **kw)
    want = oracle.pcs_prove(trees, **kw)
    got = ctx.pcs_prove_host(trees, **kw)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("kw", [dict(log_last_layer=9), {}])
def test_fri_reports_a_wait_that_ran_out(ctx, oracle, monkeypatch, kw):
    """Thread blocks that give up their first wait: of one layer, after which nobody waits for them, and of several. The context proves on."""
    trees, kw = [[m31_column(9400, 1 << 10)]], dict(pow_bits=4, log_blowup=1, n_queries=9, **kw)
    monkeypatch.setenv("ZKB_FRI_MID", "impatient")
    with pytest.raises(ZkbError) as e:
        ctx.pcs_prove_host(trees, **kw)
    assert e.value.code == -4
    monkeypatch.delenv("ZKB_FRI_MID")
    want, got = oracle.pcs_prove(trees, **kw), ctx.pcs_prove_host(trees, **kw)
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("spec", [{5: 2, 3: 1}, {12: 2, 9: 30}, {16: 1, 13: 40}, {6: 500, 2: 3}])
def test_gkr_batch_whose_launch_is_refused(ctx, oracle, monkeypatch, spec):
    """Layers whose thread blocks can not all be resident are planned again, as launches, after what was planned had been staged: rounds ahead of the
    transcript from the first one on (no eq table there yet) and from a later one, words that the launch carries and words that are copied."""
    inst, dev, keep = [], [], []
    for log_n, count in spec.items():
        for i in range(count):
            n, kind = 1 << log_n, (3, 0, 1, 2)[len(inst) % 4]
            at = 9500 + 3 * len(inst)
            den = qm31_array(at, n, nonzero=True)
            num = qm31_array(at + 1, n) if kind == 1 else m31_column(at + 2, n) if kind == 2 else None
            inst.append((kind, num, den))
            keep += [ctx.upload(num) if num is not None else None, ctx.upload(den)]
            dev.append((kind, keep[-2].ptr if num is not None else 0, keep[-1].ptr, n))
    want = oracle.gkr_prove(inst, 0x5EED0019, verify=True)
    monkeypatch.setenv("ZKB_GKR_DRIVER", "batch")
    monkeypatch.setenv("ZKB_GKR_ROUNDS", "refused")
    ctx.profile_begin()
    got = ctx.gkr_prove_device(dev, 0x5EED0019)
    prof, layers = ctx.profile_end(), max(spec)
    assert prof["gkr_batch_step_kernel"][1] == sum(r + 1 for r in range(1, layers))  # every layer went that way
    assert len(got) == len(want) and (got == want).all()


@pytest.mark.parametrize("log_rows,kw", [(10, {}), (10, dict(log_last_layer=9)), (11, dict(log_last_layer=2)), (15, {}), (16, dict(log_last_layer=12))])
def test_fri_layers_of_many_ctas_refused(ctx, oracle, monkeypatch, log_rows, kw):
    """The middle layers as launches, none before them and one, with and without last layers in a launch behind them."""
    monkeypatch.setenv("ZKB_FRI_MID", "refused")
    ctx.profile_begin()
    test_fri_layers_of_many_ctas(ctx, oracle, log_rows, kw)
    assert "fri_mid_kernel" not in ctx.profile_end()
