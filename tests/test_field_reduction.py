"""The fold of a 64-bit sum of products to a residue, over the whole range of its argument: the header the kernels and the host code
share, and the copy of it that specialised constraint programs are compiled with, both as host code."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zk_inference_prover_b200", "csrc")
P = (1 << 31) - 1

SHARED = '#include "m31.cuh"\nusing namespace zk;\n'
EXPORTS = """
extern "C" unsigned reduce64(unsigned long long v) { return m31_reduce64(v); }
extern "C" void mul(const unsigned* a, const unsigned* b, unsigned* o) {
    qm31 x{{a[0], a[1], a[2], a[3]}}, y{{b[0], b[1], b[2], b[3]}}, r = qm31_mul(x, y);
    for (int k = 0; k < 4; k++) o[k] = r.c[k];
}
"""


def _prelude():
    """The field part of the specialised programs' prelude, with the device qualifiers made empty."""
    text = open(os.path.join(CSRC, "host", "air_jit.cpp")).read()
    body = re.search(r'R"SRC\((.*?)// core/utils', text, flags=re.S).group(1)
    return "#define __device__\n#define __forceinline__ inline\n" + body


@pytest.fixture(scope="module", params=["shared", "specialised"])
def field(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("field")
    src, so = d / "f.cpp", d / "f.so"
    src.write_text((SHARED if request.param == "shared" else _prelude()) + EXPORTS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.reduce64.argtypes, lib.reduce64.restype = [ctypes.c_uint64], ctypes.c_uint32
    return lib


# Operands of a secure product whose first coordinate adds four products up to 3 * 2^62 - 1: x0 y0 + (p - x1) y1 + x2 e0 + (p - x3) e1
# with e0 = 2 y2 - y3 and e1 = y2 + 2 y3.
E0, E1 = 2147483582, 1674196099
FIFTH = pow(5, -1, P)
X = [2147483509, P - 2147482779, 2147482864, P - 4188]
Y = [2147483064, 2147482825, (2 * E0 + E1) * FIFTH % P, (2 * E1 - E0) * FIFTH % P]


def _mul(x, y):
    def cm(a, b):
        return [(a[0] * b[0] - a[1] * b[1]) % P, (a[0] * b[1] + a[1] * b[0]) % P]

    ac, bd, ad, bc = cm(x[:2], y[:2]), cm(x[2:], y[2:]), cm(x[:2], y[2:]), cm(x[2:], y[:2])
    return [(ac[0] + 2 * bd[0] - bd[1]) % P, (ac[1] + 2 * bd[1] + bd[0]) % P, (ad[0] + bc[0]) % P, (ad[1] + bc[1]) % P]


def test_reduction_over_the_whole_range(field):
    assert X[0] * Y[0] + (P - X[1]) * Y[1] + X[2] * E0 + (P - X[3]) * E1 == 3 * (1 << 62) - 1
    vals = {0, (1 << 64) - 1}
    for c in [k << 62 for k in range(1, 4)] + [k * P * P for k in range(1, 5)] + [k << 31 for k in range(1, 4)] + [(k << 62) - (1 << 31) for k in range(1, 5)]:
        vals |= {c + d for d in range(-70, 71)}
    rng = np.random.default_rng(7)
    vals |= {int(v) for v in rng.integers(0, 1 << 64, 20000, dtype=np.uint64)}
    bad = [v for v in vals if 0 <= v < 1 << 64 and field.reduce64(v) != v % P]
    assert not bad, bad[:3]


def test_product_at_the_top_of_the_range(field):
    out = (ctypes.c_uint32 * 4)()
    for x, y in [(X, Y), (Y, X), ([P - 1] * 4, [P - 1] * 4), ([0] * 4, Y), ([0, 0, P - 1, 0], [0, 0, P - 1, P - 1])]:
        field.mul((ctypes.c_uint32 * 4)(*x), (ctypes.c_uint32 * 4)(*y), out)
        assert list(out) == _mul(x, y)


@pytest.mark.gpu
def test_product_at_the_top_of_the_range_on_the_device(ctx):
    """fix_first_variable of the two entries 0 and y at x is x y."""
    src = ctx.upload(np.array([[0] * 4, Y], np.uint32))
    dst = ctx.alloc(4)
    ctx.mle_fix_qm31(src.ptr, 2, np.array(X, np.uint32), dst.ptr)
    assert dst.download().tolist() == _mul(X, Y)


SIGNED = SHARED + """
extern "C" unsigned mul_signed(unsigned v, unsigned t) { return m31_mul_signed(v, m31_twice_signed(t)); }
extern "C" unsigned unsign(unsigned v) { return m31_unsign(v); }
"""


def test_signed_product_stays_in_range_and_in_its_class(tmp_path):
    (tmp_path / "s.cpp").write_text(SIGNED)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(tmp_path / "s.so"), str(tmp_path / "s.cpp")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "s.so"))
    lib.mul_signed.restype = lib.unsign.restype = ctypes.c_uint32
    half = 1 << 30
    rng = np.random.default_rng(3)
    vs = [-P, 1 - P, 2 - P, -half - 1, -half, 1 - half, -1, 0, 1, half - 1, half, half + 1, P - 1, P] + [int(x) for x in rng.integers(-P, P + 1, 200)]
    ts = [0, 1, half - 2, half - 1, half, half + 1, P - 2, P - 1] + [int(x) for x in rng.integers(0, P, 100)]
    for v in vs:
        for t in ts:
            q = lib.mul_signed(ctypes.c_uint32(v & 0xffffffff), ctypes.c_uint32(t))
            assert -P <= q - ((q >> 31) << 32) <= P - 1 and lib.unsign(ctypes.c_uint32(q)) == v * t % P


SUMS = SHARED + """
static qm31 q(const unsigned* a) { return {{a[0], a[1], a[2], a[3]}}; }
extern "C" void sums(const unsigned* x, const unsigned* y, const unsigned* z, int n, unsigned* o) {
    qm31_sum s = qm31_sum_zero();
    for (int k = 0; k < n; k++) s.add_product(q(x), q(y));
    const qm31 r[4] = {qm31_mul_add(q(x), q(y), q(z)), qm31_dot2(q(x), q(y), q(z), q(y)), qm31_dot2_m31(q(x), y[0], q(z), y[1]), s.value()};
    for (int k = 0; k < 16; k++) o[k] = r[k / 4].c[k % 4];
}
"""


def test_sums_of_products_at_the_top_of_the_range(tmp_path):
    (tmp_path / "s.cpp").write_text(SUMS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(tmp_path / "s.so"), str(tmp_path / "s.cpp")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "s.so"))
    rng = np.random.default_rng(4)
    top, word = [P - 1] * 4, lambda v: np.array(v, np.uint32).ctypes.data_as(ctypes.c_void_p)
    cases = [(X, Y, top), (top, top, top), ([0, 0, 0, 0], top, top), ([P - 1, 0, P - 1, 0], [P - 1, P - 1, 0, P - 1], [0] * 4)]
    cases += [tuple([int(v) for v in rng.integers(0, P, 4)] for _ in range(3)) for _ in range(200)]
    for x, y, z in cases:
        out = np.zeros(16, np.uint32)
        lib.sums(word(x), word(y), word(z), 5, out.ctypes.data_as(ctypes.c_void_p))
        xy, zy = _mul(x, y), _mul(z, y)
        want = [(a + b) % P for a, b in zip(xy, z)] + [(a + b) % P for a, b in zip(xy, zy)] + [(a * y[0] + b * y[1]) % P for a, b in zip(x, z)] + [5 * a % P for a in xy]
        assert out.tolist() == want
