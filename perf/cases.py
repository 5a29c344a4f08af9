"""What a user of this library has it do: whole proofs (commitment scheme, STARK, lookup arguments, composed segments), the
trait operators called one by one as a Rust backend calls them, and the device witness generators.

`listed()` names twelve cases, `draw()` gives more from the same ranges, `prepare()` builds what a program holds before the
call, `run()` is one pass through the public entry points, `work()` the bytes and operations it cannot do without."""
import math

import numpy as np
import torch

import zk_inference_prover_b200 as zkb
from zk_inference_prover_b200 import air
from zk_inference_prover_b200 import witness_cases

P = (1 << 31) - 1
MAX_LOG = 24  # the tallest domain any case uses: a segment's 2^23-row table at blow-up 2

# Operations of the two building blocks: a circle-FFT butterfly (one modular product, sum and difference) and a Blake2s
# compression (80 half-rounds of 12 additions, xors and rotations).
BUTTERFLY_OPS, COMPRESS_OPS = 10.5, 960


def listed():
    return [
        # The smallest statement somebody proves: ten short columns. Latency and launches only.
        dict(name="pcs 10 x 2^8", kind="pcs", cols=10, log_rows=8, spread=0, trees=1, log_blowup=2, queries=3, pow_bits=10, host=False),
        # The headline workload of the benchmark: 256 columns of 2^20 rows, blow-up 4, trace on the device.
        dict(name="pcs 256 x 2^20", kind="pcs", cols=256, log_rows=20, spread=0, trees=1, log_blowup=2, queries=3, pow_bits=10, host=False),
        # The same call for a prover whose witness is made on the host: the trace comes from page-locked host memory.
        dict(name="pcs host 64 x 2^20", kind="pcs", cols=64, log_rows=20, spread=0, trees=1, log_blowup=2, queries=3, pow_bits=10, host=True),
        # The backend traits called one by one, as the Rust prover does, on an odd column count.
        dict(name="operators 33 x 2^16", kind="operators", cols=33, log_rows=16, log_blowup=1),
        # A statement of several components of different heights, proved with compiled constraints.
        dict(name="stark 3 components", kind="stark", components=3, cols=100, log_rows=16, log_blowup=1, queries=20, pow_bits=10, specialised=True),
        # Lookup arguments: one short instance, a batch of mixed instances, and the 2^24-fraction benchmark.
        dict(name="gkr 2^10", kind="gkr", instances=1, log_rows=10, spread=0, layer="singles"),
        dict(name="gkr batch of 34", kind="gkr", instances=34, log_rows=13, spread=3, layer="mixed"),
        dict(name="gkr 2^24", kind="gkr", instances=1, log_rows=24, spread=0, layer="multiplicities"),
        # Composed decode segments, the product's unit of work: the microbenchmark's size and a full layer segment.
        dict(name="segment micro", kind="segment", tiles=8, tile_log=7, mat_log=8, width=544, table_log=22),
        dict(name="segment layer", kind="segment", tiles=64, tile_log=11, mat_log=13, width=4480, table_log=23),
        # The witness side: the Freivalds component of a 4096 x 4096 product, and a layer's generated columns.
        dict(name="freivalds 4096 x 4096", kind="freivalds", n_in=4096, n_out=4096, tokens=32, chunks=256, mats=2),
        dict(name="witness 512 x 4096", kind="witness", tokens=512, chunks=256, per_row=16, adds=128, stream_log=15, table_log=23),
    ]


def _between(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["pcs", "pcs", "pcs", "operators", "stark", "gkr", "gkr", "segment", "segment", "freivalds", "witness"])
    if kind == "pcs":
        log_rows = rng.randint(6, 20)
        spread = rng.choice([0, 0, rng.randint(1, min(8, log_rows - 4))])
        return dict(kind=kind, cols=_between(rng, 2, 256), log_rows=log_rows, spread=spread, trees=rng.choice([1, 1, 2, 3]),
                    log_blowup=rng.choice([1, 2]), queries=rng.choice([3, 20, 70, 100]), pow_bits=rng.choice([0, 5, 10]), host=rng.random() < 0.3)
    if kind == "operators":
        return dict(kind=kind, cols=_between(rng, 4, 200), log_rows=rng.randint(6, 19), log_blowup=rng.choice([1, 2]))
    if kind == "stark":
        return dict(kind=kind, components=rng.randint(1, 4), cols=_between(rng, 10, 160), log_rows=rng.randint(10, 18), log_blowup=rng.choice([1, 2]),
                    queries=rng.choice([3, 20, 70]), pow_bits=rng.choice([0, 10]), specialised=rng.random() < 0.7)
    if kind == "gkr":
        layer = rng.choice(["singles", "multiplicities", "generic", "product", "mixed"])
        if rng.random() < 0.5:
            return dict(kind=kind, instances=1, log_rows=rng.randint(4, 23), spread=0, layer=layer)
        return dict(kind=kind, instances=_between(rng, 2, 300), log_rows=rng.randint(6, 16), spread=rng.randint(0, 4), layer=layer)
    if kind == "segment":
        return dict(kind=kind, tiles=_between(rng, 2, 60), tile_log=rng.randint(6, 11), mat_log=rng.randint(8, 13), width=_between(rng, 300, 4400),
                    table_log=rng.randint(14, 22))
    if kind == "freivalds":
        return dict(kind=kind, n_in=_between(rng, 64, 4096), n_out=_between(rng, 64, 4096), tokens=rng.randint(1, 64),
                    chunks=rng.choice([4, 13, 32, 100, 256]), mats=rng.randint(1, 3))
    return dict(kind=kind, tokens=1 << rng.randint(3, 9), chunks=1 << rng.randint(3, 8), per_row=rng.randint(1, 16), adds=_between(rng, 4, 128),
                stream_log=rng.randint(6, 15), table_log=rng.randint(10, 23))


# ---- what a program keeps: one context, compiled constraint programs, the closed-form tables -------------------------------
_kept = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _context():
    return _keep("context", lambda: zkb.Context(device=0, max_log_size=MAX_LOG))


def _program(cols, specialised):
    def make():
        prog = _context().air_compile(air.wide_fibonacci(air.ExprEvaluator(), cols).source())
        return prog.specialize() if specialised else prog

    return _keep(("program", cols, specialised), make)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _words(g, n, low=0, high=P):
    """n uniform field elements on the device (as int32: the values fit 31 bits)."""
    return torch.randint(low, high, (n,), generator=g, device="cuda", dtype=torch.int32)


def _empty(n):
    return torch.empty(int(n), device="cuda", dtype=torch.int32)


def _pieces(t, sizes):
    """Device addresses of consecutive runs of `sizes` words of tensor t."""
    out, at = [], t.data_ptr()
    for n in sizes:
        out.append(at)
        at += 4 * n
    return out


def _felts(seed, n):
    """n secure field elements as host words (challenges and points)."""
    return np.random.default_rng(seed).integers(1, P, (n, 4)).astype(np.uint32)


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["run"] = _RUN[case["kind"]]
    state["ctx"] = _context()
    torch.cuda.synchronize()
    return state


def run(state):
    return state["run"](state, state["ctx"])


def tolerance(case):
    return "exact"  # field elements, hashes and counts


def work(case):
    return _WORK[case["kind"]](case)


# ---- polynomial commitment proofs --------------------------------------------------------------------------------------------
def _pcs_shape(case):
    """The trees' column heights: the columns are dealt to the trees in turn; heights run over [log_rows - spread, log_rows] and
    the last tree's first column is the tallest."""
    trees = [[] for _ in range(min(case["trees"], case["cols"]))]
    for c in range(case["cols"]):
        trees[(c + 1) % len(trees)].append(case["log_rows"] - (c // len(trees)) * 5 % (case["spread"] + 1))
    trees[-1][0] = case["log_rows"]
    return trees


def _proof_room(trees, log_blowup, queries):
    """A buffer that holds any proof of this shape. How long one is depends on its challenges (queries that fall together, shared
    paths; a lifted column is opened at its queries and along the paths), so a program that keeps proofs of one shape keeps them in
    buffers of the longest, the rest zero."""
    cols, height = sum(len(t) for t in trees), max(max(t) for t in trees) + log_blowup
    return np.zeros(1024 + 16 * cols + 2 * queries * (cols + 8 * height * (len(trees) + 2 * height)), np.uint32)


def _into(room, words):
    room[:len(words)] = words
    return room


def _pcs_prepare(case, seed):
    ctx, trees = _context(), _pcs_shape(case)
    logs = [l for t in trees for l in t]
    trace = _words(_gen(seed), sum(1 << l for l in logs))
    config = dict(pow_bits=case["pow_bits"], log_blowup=case["log_blowup"], log_last_layer=0, n_queries=case["queries"])
    room = _proof_room(trees, case["log_blowup"], case["queries"])
    if case["host"]:
        pinned = torch.empty(trace.numel(), dtype=torch.int32, pin_memory=True)
        pinned.copy_(trace)
        words, at, cols = pinned.numpy().view(np.uint32), 0, []
        for t in trees:
            cols.append([])
            for l in t:
                cols[-1].append(words[at:at + (1 << l)])
                at += 1 << l
        return dict(host=cols, keep=pinned, config=config, room=room)
    work_copy = torch.empty_like(trace)
    ptrs, flat = [], iter(_pieces(work_copy, [1 << l for l in logs]))
    for t in trees:
        ptrs.append([next(flat) for _ in t])
    return dict(host=None, trace=trace, work=work_copy, ptrs=ptrs, logs=logs, config=config, room=room)


def _pcs_run(s, ctx):
    if s["host"] is not None:
        return _into(s["room"], ctx.pcs_prove_host(s["host"], **s["config"]))
    # the proof consumes its trace: the copy stands for the trace's arrival
    ctx.d2d(s["work"].data_ptr(), s["trace"].data_ptr(), 4 * s["trace"].numel())
    return _into(s["room"], ctx.pcs_prove_device(s["ptrs"], s["logs"], **s["config"]))


def _commit_ops(trees, log_blowup):
    """Interpolation, extension and hashing of the trees of a commitment, then FRI's trees over the tallest domain."""
    ops = 0.0
    for t in trees:
        for l in set(t):
            n, count = 1 << l, t.count(l)
            ops += BUTTERFLY_OPS * count * (n / 2 * l + (n << log_blowup) / 2 * l)
            ops += COMPRESS_OPS * (n << log_blowup) * (1 + (count - 1) // 16)
        ops += COMPRESS_OPS * (2 << (max(t) + log_blowup))
    return ops + COMPRESS_OPS * (4 << (max(max(t) for t in trees) + log_blowup))


def _pcs_work(case):
    trees = _pcs_shape(case)
    return {"bytes": 4 * sum(1 << l for t in trees for l in t), "flops": _commit_ops(trees, case["log_blowup"])}


# ---- the traits' operators one by one ------------------------------------------------------------------------------------------
def _operators_prepare(case, seed):
    n, log_out = 1 << case["log_rows"], case["log_rows"] + case["log_blowup"]
    N, cols = 1 << log_out, case["cols"]
    s = dict(case=case, log_out=log_out, trace=_words(_gen(seed), cols * n), coeffs=_empty(cols * n), evals=_empty(cols * N),
             hashes=_empty(16 * N), numerators=_empty(4 * N), quotients=_empty(4 * N), folds=torch.zeros(4 * N + 64, device="cuda", dtype=torch.int32),
             zeros=torch.zeros(2 * N, device="cuda", dtype=torch.int32), fri_hashes=_empty(16 * N), points=_felts(seed, 2), alphas=_felts(seed + 1, log_out + 1), lines=_felts(seed + 2, 2 * cols))
    s["coeff_ptrs"], s["eval_ptrs"] = _pieces(s["coeffs"], [n] * cols), _pieces(s["evals"], [N] * cols)
    s["layers"] = _pieces(s["hashes"], [8 << k for k in range(log_out, -1, -1)])
    return s


def _pieces_at(at, log_rows):
    """The four coordinate columns of a FRI layer, each on a 16-byte boundary."""
    return [at + k * max(16, 4 << log_rows) for k in range(4)]


def _operators_run(s, ctx):
    case, log_out = s["case"], s["log_out"]
    N, cols, log_n = 1 << log_out, case["cols"], case["log_rows"]
    ctx.d2d(s["coeffs"].data_ptr(), s["trace"].data_ptr(), 4 * s["trace"].numel())
    ctx.ifft_cols(s["coeff_ptrs"], log_n)
    ctx.lde_cols(s["coeff_ptrs"], log_n, s["eval_ptrs"], log_out)
    ctx.merkle_layer(log_out, 0, s["eval_ptrs"], s["layers"][0])
    for k in range(1, log_out + 1):
        ctx.merkle_layer(log_out - k, s["layers"][k - 1], [], s["layers"][k])
    samples = ctx.eval_at_point_cols(s["coeff_ptrs"], log_n, s["points"].reshape(-1))
    num = _pieces(s["numerators"], [N] * 4)
    ctx.quot_numerators(s["eval_ptrs"], log_out, list(range(cols)), s["lines"][:cols], s["lines"][cols:], num)
    quo = _pieces(s["quotients"], [N] * 4)
    ctx.quot_combine(num, [log_out], s["alphas"][0], s["points"].reshape(-1), log_out, quo)
    # FRI: the circle fold into a zeroed line, then line folds, each layer with its own tree
    ctx.d2d(s["folds"].data_ptr(), s["zeros"].data_ptr(), 8 * N)
    at, log_layer = s["folds"].data_ptr(), log_out - 1
    layer = _pieces_at(at, log_layer)
    ctx.fold_circle_into_line(layer, quo, log_out, s["alphas"][1])
    nodes = s["fri_hashes"].data_ptr()
    while log_layer > 0:
        ctx.merkle_layer(log_layer, 0, layer, nodes)
        for k in range(log_layer - 1, -1, -1):
            ctx.merkle_layer(k, nodes, [], nodes + (32 << (k + 1)))
            nodes += 32 << (k + 1)
        nodes += 32
        at = layer[3] + max(16, 4 << log_layer)
        log_layer -= 1
        folded = _pieces_at(at, log_layer)
        ctx.fold_line(folded, layer, log_layer + 1, s["alphas"][log_out - log_layer])
        layer = folded
    written = (nodes - s["fri_hashes"].data_ptr()) // 4
    return dict(coeffs=s["coeffs"], evals=s["evals"], tree=s["hashes"][:16 * N - 8], samples=samples, quotients=s["quotients"],
                folds=s["folds"], fri=s["fri_hashes"][:written])


def _operators_work(case):
    n, N = 1 << case["log_rows"], 1 << (case["log_rows"] + case["log_blowup"])
    return {"bytes": 4 * case["cols"] * (2 * n + N) + 4 * N * (16 + 4 + 4 + 16), "flops": _commit_ops([[case["log_rows"]] * case["cols"]], case["log_blowup"])}


# ---- STARK proofs of wide Fibonacci components -----------------------------------------------------------------------------------
def _stark_shape(case):
    """(columns, log rows) of the components: each next one a quarter as high and five columns narrower, none below 2^6 rows."""
    return [(max(5, case["cols"] - 5 * k), max(6, case["log_rows"] - 2 * k)) for k in range(case["components"])]


def _stark_prepare(case, seed):
    g, shape = _gen(seed), _stark_shape(case)
    trace = []
    for cols, log_rows in shape:  # every row its own sequence from two random values: a trace the constraints accept
        a, b = (_words(g, 1 << log_rows).long() for _ in range(2))
        rows = [a, b]
        for _ in range(2, cols):
            a, b = b, (a * a % P + b * b % P) % P
            rows.append(b)
        trace.append(torch.stack(rows).to(torch.int32).reshape(-1))
    trace = torch.cat(trace)
    work_copy = torch.empty_like(trace)
    ptrs = _pieces(work_copy, [1 << l for c, l in shape for _ in range(c)])
    # the tallest component's columns first; the composition tree, which the call adds, is the last and tallest
    comps = [(_program(c, case["specialised"]), l, None) for c, l in shape]
    trees = [[l for c, l in shape for _ in range(c)], [case["log_rows"]] * 8]
    return dict(trace=trace, work=work_copy, ptrs=ptrs, components=comps, room=_proof_room(trees, case["log_blowup"], case["queries"]),
                config=dict(pow_bits=case["pow_bits"], log_blowup=case["log_blowup"], log_last_layer=0, n_queries=case["queries"]))


def _stark_run(s, ctx):
    ctx.d2d(s["work"].data_ptr(), s["trace"].data_ptr(), 4 * s["trace"].numel())
    words, committed, from_constraints, _ms = ctx.stark_prove_multi(s["components"], [[], [], s["ptrs"], []], **s["config"])
    return _into(s["room"], words), committed, from_constraints


def _stark_work(case):
    shape = _stark_shape(case)
    trees = [[l for c, l in shape for _ in range(c)], [case["log_rows"]] * 8]
    constraints = sum(10.0 * c * (2 << l) for c, l in shape)
    return {"bytes": 4 * sum(c << l for c, l in shape), "flops": _commit_ops(trees, case["log_blowup"]) + constraints}


# ---- lookup arguments ----------------------------------------------------------------------------------------------------------------
_LAYERS = {"product": (zkb.GKR_GRAND_PRODUCT, 0), "generic": (zkb.GKR_LOGUP_GENERIC, 4), "multiplicities": (zkb.GKR_LOGUP_MULTIPLICITIES, 1),
           "singles": (zkb.GKR_LOGUP_SINGLES, 0)}


def _gkr_shape(case):
    """(layer kind, numerator words an entry, log entries) of the instances."""
    order = ["singles", "singles", "multiplicities", "generic", "product"] if case["layer"] == "mixed" else [case["layer"]]
    return [_LAYERS[order[i % len(order)]] + (max(1, case["log_rows"] - i * 3 % (case["spread"] + 1)),) for i in range(case["instances"])]


def _gkr_instances(g, shape):
    den = _words(g, sum(4 << l for _k, _w, l in shape), low=1)
    num = _words(g, max(4, sum(w << l for _k, w, l in shape)))
    den_ptrs, num_ptrs = _pieces(den, [4 << l for _k, _w, l in shape]), _pieces(num, [w << l for _k, w, l in shape])
    return [(k, n if w else 0, d, 1 << l) for (k, w, l), n, d in zip(shape, num_ptrs, den_ptrs)], (den, num)


def _gkr_prepare(case, seed):
    shape = sorted(_gkr_shape(case), key=lambda x: -x[2])  # tallest first: every column starts on a 16-byte boundary
    instances, keep = _gkr_instances(_gen(seed), shape)
    return dict(instances=instances, keep=keep)


def _gkr_run(s, ctx):
    return ctx.gkr_prove_device(s["instances"], 0x5EED0004)


def _gkr_ops(logs):
    """Building the layers (three secure products a pair) and the rounds on them (about twelve a quadruple, halving)."""
    return sum((3 + 12 + 12) * 30.0 * (1 << l) for l in logs)


def _gkr_work(case):
    shape = _gkr_shape(case)
    return {"bytes": sum((4 + w) * 4 << l for _k, w, l in shape), "flops": _gkr_ops([l for _k, _w, l in shape])}


# ---- composed segments -----------------------------------------------------------------------------------------------------------------
def _segment_shape(case):
    """The trees of one composed segment and its lookup batches: components of (committed columns, interaction columns, log rows,
    lookups a row, repetitions), one opening proof for all of their columns and one lookup argument per family."""
    t, tl, ml, w, tb = case["tiles"], case["tile_log"], case["mat_log"], case["width"], case["table_log"]
    low = lambda l: max(4, l)
    families = {
        "key tiles": [(64, 16, tl, 64, t), (192, 24, low(tl - 2), 160, t), (64, 20, tl, 64, 1), (192, 28, low(tl - 2), 160, 1),
                      (64, 16, low(tl - 1), 64, 2 * t), (192, 24, low(tl - 3), 160, 2 * t), (64, 8, 5, 32, 1), (64, 8, 4, 32, 2)],
        "dequantize": [(242, 16, ml, 96, 2), (242, 16, low(ml - 2), 96, 1), (146, 12, low(ml - 2), 128, 1), (212, 16, min(tb, ml + 2), 84, 2)],
        "outputs": [(146, 20, ml, 112, 1)],
        "freivalds": [(2, 32, min(tb, ml + 4), 2, 1), (2, 16, min(tb, ml + 4), 2, 1), (1, 24, min(tb, ml + 6), 1, 1)],
        "residual stream": [(w, 16, low(min(10, tl)), w * 2 // 5, 2), (w // 8, 8, 5, w // 20 + 1, 2), (w // 3, 12, low(min(10, tl)), w // 6 + 1, 4),
                            (w // 2, 8, low(min(8, tl)), w // 5 + 1, 2)],
    }
    plain = [(112, 168, ml, 1), (112, 168, low(ml - 2), 1), (116, 176, ml, 2), (1, 4, tb, 1)] + [(1, 4, l, 2) for l in range(4, min(tb, 18))]
    links = [(0, 16, l, 1) for l in range(4, min(tb, 12))]
    trees, batches = [[], []], []
    for comps in families.values():
        batch = []
        for base, inter, log_rows, lookups, times in comps:
            trees[0] += [log_rows] * (base * times)
            trees[1] += [log_rows] * (inter * times)
            # a component's lookups are split along the binary digits of their number
            batch += [log_rows + b for b in range(lookups.bit_length()) if lookups >> b & 1] * times
        batches.append(sorted(batch, reverse=True))
    for base, inter, log_rows, times in plain + links:
        trees[0] += [log_rows] * (base * times)
        trees[1] += [log_rows] * (inter * times)
    trees.append([min(tb, 16)] * max(2, t * 8))  # boundary columns
    trees.append([max(l for tree in trees for l in tree)] * 8)  # the composition columns
    return trees, batches


def _segment_prepare(case, seed):
    ctx, g = _context(), _gen(seed)
    trees, batches = _segment_shape(case)
    logs = [l for t in trees for l in t]
    trace = _words(g, sum(1 << l for l in logs))
    work_copy = torch.empty_like(trace)
    flat = _pieces(work_copy, [1 << l for l in logs])
    ptrs, at = [], 0
    for t in trees:
        ptrs.append(flat[at:at + len(t)])
        at += len(t)
    instances, keep = [], []
    for b in batches:
        inst, held = _gkr_instances(g, [_LAYERS["singles"] + (l,) for l in b])
        instances.append(inst)
        keep.append(held)
    prepared = ctx.pcs_prepare(ptrs, logs, cap=1)
    prepared["out"] = _proof_room(trees, 1, 100)
    return dict(trace=trace, work=work_copy, prepared=prepared, instances=instances, keep=keep)


def _segment_run(s, ctx):
    ctx.d2d(s["work"].data_ptr(), s["trace"].data_ptr(), 4 * s["trace"].numel())
    # the prover's own parameters: blow-up 2, 100 queries, no proof of work
    ctx.pcs_prove_device(s["prepared"], None, pow_bits=0, log_blowup=1, log_last_layer=0, n_queries=100)
    return [s["prepared"]["out"]] + [ctx.gkr_prove_device(inst, 0x5EED0007 + i, cap=1 << 24) for i, inst in enumerate(s["instances"])]


def _segment_work(case):
    trees, batches = _segment_shape(case)
    logs = [l for b in batches for l in b]
    return {"bytes": 4 * sum(1 << l for t in trees for l in t) + 16 * sum(1 << l for l in logs), "flops": _commit_ops(trees, 1) + _gkr_ops(logs)}


# ---- witness generation ------------------------------------------------------------------------------------------------------------------
def _freivalds_layout(case):
    """(grid, columns of activations, columns of weights a matrix) for the case's chunk count."""
    rows = case["n_in"] * case["chunks"]
    log_rows = max(4, (rows - 1).bit_length())
    return (log_rows, case["n_in"], case["chunks"], (1 << log_rows) - rows), -(-case["tokens"] // case["chunks"]), -(-case["n_out"] // case["chunks"])


def _freivalds_prepare(case, seed):
    g = _gen(seed)
    grid, pq, pk = _freivalds_layout(case)
    R, mats = 1 << grid[0], case["mats"]
    ints = lambda *shape: torch.randint(-128, 128, shape, generator=g, device="cuda", dtype=torch.int8)
    s = dict(case=case, grid=grid, pq=pq, pk=pk, qx=ints(case["tokens"], case["n_in"]), qw=[ints(case["n_in"], case["n_out"]) for _ in range(mats)],
             base=_empty(pq * R), pre=_empty((mats * pk + 4) * R), acc=_empty((1 + 2 * mats) * 4 * R), counts=_empty(258),
             zeros=torch.zeros(258, device="cuda", dtype=torch.int32), felts=_felts(seed, 2))
    s["base_ptrs"], s["pre_ptrs"] = _pieces(s["base"], [R] * pq), _pieces(s["pre"], [R] * (mats * pk + 4))
    s["acc_ptrs"] = _pieces(s["acc"], [R] * ((1 + 2 * mats) * 4))
    return s


def _freivalds_run(s, ctx):
    case, counts = s["case"], s["counts"].data_ptr()
    ctx.d2d(counts, s["zeros"].data_ptr(), 4 * 258)
    ctx.freivalds_scatter(s["qx"].data_ptr(), [w.data_ptr() for w in s["qw"]], [case["n_out"]] * case["mats"], s["grid"], s["pq"], s["pk"], case["n_in"],
                          case["tokens"], s["base_ptrs"], s["pre_ptrs"], counts, 256, counts + 1024)
    claims = ctx.freivalds_acc(s["base_ptrs"], s["pre_ptrs"][:case["mats"] * s["pk"]], s["grid"], s["pq"], s["pk"], case["mats"], s["felts"][0],
                               s["felts"][1], s["acc_ptrs"])
    return dict(base=s["base"], pre=s["pre"], acc=s["acc"], counts=s["counts"], claims=claims)


def _freivalds_work(case):
    grid, pq, pk = _freivalds_layout(case)
    R, mats = 1 << grid[0], case["mats"]
    inputs = case["tokens"] * case["n_in"] + mats * case["n_in"] * case["n_out"]
    return {"bytes": inputs + 4 * R * (pq + mats * pk + 4 + (1 + 2 * mats) * 4), "flops": R * (8.0 * (pq + mats * pk) + 60.0 * (1 + 2 * mats))}


_KMAX = 13  # the widest accumulator window of the normalisation table used here


def _stream_program(adds):
    """The residual-stream component's program and tables for `adds` additions a row (its inputs are made on the device)."""
    return _keep(("stream", adds), lambda: witness_cases.residual_stream_case(9, "pairs", adds, 4, 1, kind=0, sticky=True, kmax=_KMAX, spread=8))


def _dequant_layout(case):
    return witness_cases.dequant_case(8, 1, tokens=1, chunks=16, per_row=case["per_row"], kmax=_KMAX, sticky=1, do_ref=0)


def _tables(case):
    """The closed-form tables on the device, which a program uploads once."""
    def make():
        rs = _stream_program(4)
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a).astype(np.int64).reshape(-1)).to(torch.int32).cuda()
        return dict(norm=up(witness_cases.norm_table(_KMAX, 1)), mul=up(witness_cases.mul_table()), smul=up(rs["smul3"]))

    return _keep("tables", make)


def _witness_prepare(case, seed):
    g, tables = _gen(seed), _tables(case)
    layout = _keep(("dequantize", case["per_row"]), lambda: _dequant_layout(case))
    tokens, n_out = case["tokens"], case["chunks"] * case["per_row"]
    rows = tokens * case["chunks"]
    cfg = dict(layout["cfg"], tokens=tokens, n_out=n_out, chunks=case["chunks"], log_rows=rows.bit_length() - 1)
    # accumulators of every magnitude the window holds, both signs
    magnitude = torch.randint(0, 1 << (_KMAX + 9), (tokens * n_out,), generator=g, device="cuda", dtype=torch.int64)
    magnitude >>= torch.randint(0, _KMAX + 9, magnitude.shape, generator=g, device="cuda", dtype=torch.int64)
    acc = (magnitude * (1 - 2 * torch.randint(0, 2, magnitude.shape, generator=g, device="cuda", dtype=torch.int64))).to(torch.int32)
    scale = lambda n: torch.stack([_words(g, n, 0, 128), _words(g, n, 100, 140)], 1).contiguous()
    # bf16 patterns of a narrow exponent range, so that additions keep and drop their smaller operand
    rs, stream_rows = _stream_program(case["adds"]), 1 << case["stream_log"]
    n = stream_rows * rs["n_leaves"]
    wit = (_words(g, n, 0, 2) << 15) | (_words(g, n, 119, 136) << 7) | _words(g, n, 0, 128)
    table_rows = 1 << case["table_log"]
    counters = [_words(g, table_rows, 0, 1000) for _ in range(4)]
    mult = {k: rs["m_len"][k] for k in ("pow", "norm", "val", "frac", "smul")}
    sizes = [cfg["n_norm"], cfg["n_frac"], cfg["n_mul"], cfg["n_r8"], 4] + list(mult.values()) + [4]
    sizes = [-(-v // 4) * 4 for v in sizes]
    s = dict(cfg=cfg, tables=tables, rs=rs, stream_log=case["stream_log"], table_log=case["table_log"], acc=acc, sx=scale(tokens), sw=scale(n_out), wit=wit,
             expmap=_words(g, 1 << 16, 0, 512), counters=counters, base=_empty(layout["n_base"] * rows), pre=_empty(layout["n_pre"] * rows),
             cols=_empty(rs["n_cols"] * stream_rows), out_pat=_empty(stream_rows * case["adds"]), out_nat=_empty(stream_rows * case["adds"] * 2),
             in_nat=_empty(n * 2), table=_empty(3 * table_rows), counts=_empty(sum(sizes)), zeros=torch.zeros(sum(sizes), device="cuda", dtype=torch.int32))
    s["base_ptrs"], s["pre_ptrs"] = _pieces(s["base"], [rows] * layout["n_base"]), _pieces(s["pre"], [rows] * layout["n_pre"])
    s["col_ptrs"], s["table_ptrs"] = _pieces(s["cols"], [stream_rows] * rs["n_cols"]), _pieces(s["table"], [table_rows] * 3)
    s["count_ptrs"], s["mult"] = _pieces(s["counts"], sizes), mult
    return s


def _witness_run(s, ctx):
    cfg, rs, t, c = s["cfg"], s["rs"], s["tables"], s["count_ptrs"]
    ctx.d2d(c[0], s["zeros"].data_ptr(), 4 * s["zeros"].numel())
    ctx.witness_dequant(cfg, s["acc"].data_ptr(), 0, 0, s["sx"].data_ptr(), s["sw"].data_ptr(), t["norm"].data_ptr(), t["mul"].data_ptr(), s["base_ptrs"],
                        s["pre_ptrs"], c[0], c[1], c[2], c[3], c[4], 0)
    mults = {k: (c[5 + i], n) for i, (k, n) in enumerate(s["mult"].items())}
    ctx.witness_residual_stream(rs["lowered_groups"], rs["lowered_slots"], rs["out_slot"], 0, True, _KMAX, t["norm"].data_ptr(), t["norm"].numel() // 3,
                                t["smul"].data_ptr(), t["smul"].numel() // 3, [], rs["n_val"], s["wit"].data_ptr(), 1 << s["stream_log"], s["stream_log"],
                                s["col_ptrs"], s["out_pat"].data_ptr(), s["out_nat"].data_ptr(), s["in_nat"].data_ptr(), mults, [], c[10])
    ctx.witness_tables(s["expmap"].data_ptr(), [x.data_ptr() for x in s["counters"]], s["table_log"], False, 2.0 ** 7, *s["table_ptrs"])
    return dict(base=s["base"], pre=s["pre"], cols=s["cols"], out_pat=s["out_pat"], out_nat=s["out_nat"], in_nat=s["in_nat"], table=s["table"],
                counts=s["counts"])


def _witness_work(case):
    layout, rs = _dequant_layout(case), _stream_program(case["adds"])
    rows, stream_rows = case["tokens"] * case["chunks"], 1 << case["stream_log"]
    words = rows * (layout["n_base"] + layout["n_pre"] + case["per_row"]) + stream_rows * (rs["n_cols"] + 3 * rs["n_leaves"] + 3 * case["adds"])
    words += 7 << case["table_log"]
    return {"bytes": 4 * words, "flops": 60.0 * (rows * case["per_row"] + stream_rows * case["adds"]) + 10.0 * (1 << case["table_log"])}


_PREPARE = dict(pcs=_pcs_prepare, operators=_operators_prepare, stark=_stark_prepare, gkr=_gkr_prepare, segment=_segment_prepare,
                freivalds=_freivalds_prepare, witness=_witness_prepare)
_RUN = dict(pcs=_pcs_run, operators=_operators_run, stark=_stark_run, gkr=_gkr_run, segment=_segment_run, freivalds=_freivalds_run, witness=_witness_run)
_WORK = dict(pcs=_pcs_work, operators=_operators_work, stark=_stark_work, gkr=_gkr_work, segment=_segment_work, freivalds=_freivalds_work,
             witness=_witness_work)
