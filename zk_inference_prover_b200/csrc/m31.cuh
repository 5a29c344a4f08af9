// Field arithmetic for the Circle-STARK operators: M31 (p = 2^31 - 1), CM31 = M31[i]/(i^2+1),
// QM31 = CM31[u]/(u^2 - 2 - i). Usable from device and host code.
//
// Every value stored to memory is canonical, i.e. in [0, p): the reference's backends compare and
// hash raw words (nitroo/crates/stwo/src/core/fields/m31.rs:58-60 gives the reduction,
// cm31.rs:44-52 and qm31.rs:80-88 the extension products). Products are accumulated unreduced in
// 64 bits and folded once per output coordinate, which is exact because 2^31 = 1 (mod p).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define ZK_HD __host__ __device__ __forceinline__
#else
#define ZK_HD inline
#endif

namespace zk {

constexpr uint32_t P = 0x7fffffffu;
constexpr uint64_t P_SQ = (uint64_t)P * (uint64_t)P;

ZK_HD uint32_t umin32(uint32_t a, uint32_t b) { return a < b ? a : b; }

// a, b in [0, p) -> canonical.
ZK_HD uint32_t m31_add(uint32_t a, uint32_t b) { uint32_t s = a + b; return umin32(s, s - P); }
ZK_HD uint32_t m31_sub(uint32_t a, uint32_t b) { uint32_t d = a - b; return umin32(d, d + P); }
ZK_HD uint32_t m31_neg(uint32_t a) { return a ? P - a : 0u; }
ZK_HD uint32_t m31_dbl(uint32_t a) { return m31_add(a, a); }

// Any 64-bit value to one below 2^34 of the same class: 2^32 = 2 (mod p), so the upper word enters doubled. On the device that is one wide
// multiply-add on the FMA pipe; masks, shifts and carries in its place are five instructions on the ALU pipe, which bounds field arithmetic here.
ZK_HD uint64_t m31_fold64(uint64_t v) {
#ifdef __CUDA_ARCH__
    uint64_t t;
    asm("mad.wide.u32 %0, %1, 2, %2;" : "=l"(t) : "r"((uint32_t)(v >> 32)), "l"((uint64_t)(uint32_t)v));
    return t;
#else
    return (v >> 32) * 2 + (uint32_t)v;
#endif
}
// Any 64-bit value -> canonical residue. The fold leaves at most 3 (2^32 - 1), whose parts of 31 and 3 bits add up to at most p + 5.
ZK_HD uint32_t m31_reduce64(uint64_t v) {
    const uint64_t t = m31_fold64(v);
    const uint32_t s = ((uint32_t)t & P) + (uint32_t)(t >> 31);
    return umin32(s, s - P);
}
// Product of two canonical values.
ZK_HD uint32_t m31_mul(uint32_t a, uint32_t b) {
    uint64_t p = (uint64_t)a * b;  // < 2^62
    uint32_t s = ((uint32_t)p & P) + (uint32_t)(p >> 31);
    return umin32(s, s - P);
}
ZK_HD uint32_t m31_sqr(uint32_t a) { return m31_mul(a, a); }

// Signed representatives. A word read as a signed integer in [-p, p - 1] stands for its residue; one add-and-minimum brings it back to
// [0, p) (m31_unsign), and a product takes it, or p, as it is.
//
// t2 is twice the representative of a factor in [-(2^30 - 1), 2^30 - 1] (m31_twice_signed). With v t2 + 2^31 = h 2^32 + l, l even,
// v t = h 2^31 + l / 2 - 2^30, congruent to h - 2^30 + l / 2: one product with the constant in its addend, one shift-and-add. For v in
// [-p, p] that lies in [-p, p - 1], since |v t2| <= (2^31 - 1) (2^31 - 2) puts h in [-2^30 + 1, 2^30 - 1].
ZK_HD uint32_t m31_twice_signed(uint32_t t) { return 2 * t + (t >> 30 ? 2u : 0u); }
ZK_HD uint32_t m31_mul_signed(uint32_t v, uint32_t t2) {
    const int64_t p = (int64_t)(int32_t)v * (int32_t)t2 + (((int64_t)1 << 31) - ((int64_t)1 << 62));
    return (uint32_t)((uint64_t)p >> 32) + ((uint32_t)p >> 1);
}
ZK_HD uint32_t m31_unsign(uint32_t v) { return umin32(v, v + P); }      // [-p, p - 1] -> [0, p)
ZK_HD uint32_t m31_reduce_sum(uint32_t v) { return umin32(v, v - P); }  // [0, 2p - 1] -> [0, p)
ZK_HD uint32_t m31_sqn(uint32_t v, int n) { for (int i = 0; i < n; i++) v = m31_sqr(v); return v; }
// v^(p-2): 37 multiplications, the addition chain of m31.rs:192-200.
ZK_HD uint32_t m31_inv(uint32_t v) {
    uint32_t t0 = m31_mul(m31_sqn(v, 2), v);
    uint32_t t1 = m31_mul(m31_sqn(t0, 1), t0);
    uint32_t t2 = m31_mul(m31_sqn(t1, 3), t0);
    uint32_t t3 = m31_mul(m31_sqn(t2, 1), t0);
    uint32_t t4 = m31_mul(m31_sqn(t3, 8), t3);
    uint32_t t5 = m31_mul(m31_sqn(t4, 8), t3);
    return m31_mul(m31_sqn(t5, 7), t2);
}

struct cm31 { uint32_t a, b; };
ZK_HD cm31 cm31_add(cm31 x, cm31 y) { return {m31_add(x.a, y.a), m31_add(x.b, y.b)}; }
ZK_HD cm31 cm31_sub(cm31 x, cm31 y) { return {m31_sub(x.a, y.a), m31_sub(x.b, y.b)}; }
ZK_HD cm31 cm31_mul(cm31 x, cm31 y) {
    uint64_t re = (uint64_t)x.a * y.a + (P_SQ - (uint64_t)x.b * y.b);
    uint64_t im = (uint64_t)x.a * y.b + (uint64_t)x.b * y.a;
    return {m31_reduce64(re), m31_reduce64(im)};
}
ZK_HD cm31 cm31_mul_m31(cm31 x, uint32_t y) { return {m31_mul(x.a, y), m31_mul(x.b, y)}; }
// 1/(a+bi) = (a-bi)/(a^2+b^2), cm31.rs:66-72
ZK_HD cm31 cm31_inv(cm31 x) {
    uint32_t n = m31_reduce64((uint64_t)x.a * x.a + (uint64_t)x.b * x.b);
    uint32_t ni = m31_inv(n);
    return {m31_mul(x.a, ni), m31_mul(m31_neg(x.b), ni)};
}

// c[0] + c[1] i + (c[2] + c[3] i) u
struct qm31 { uint32_t c[4]; };
ZK_HD qm31 qm31_zero() { return {{0, 0, 0, 0}}; }
ZK_HD qm31 qm31_one() { return {{1, 0, 0, 0}}; }
ZK_HD qm31 qm31_from_m31(uint32_t v) { return {{v, 0, 0, 0}}; }
ZK_HD qm31 qm31_add(qm31 x, qm31 y) {
    return {{m31_add(x.c[0], y.c[0]), m31_add(x.c[1], y.c[1]), m31_add(x.c[2], y.c[2]), m31_add(x.c[3], y.c[3])}};
}
ZK_HD qm31 qm31_sub(qm31 x, qm31 y) {
    return {{m31_sub(x.c[0], y.c[0]), m31_sub(x.c[1], y.c[1]), m31_sub(x.c[2], y.c[2]), m31_sub(x.c[3], y.c[3])}};
}
ZK_HD qm31 qm31_neg(qm31 x) { return {{m31_neg(x.c[0]), m31_neg(x.c[1]), m31_neg(x.c[2]), m31_neg(x.c[3])}}; }
ZK_HD qm31 qm31_dbl(qm31 x) { return qm31_add(x, x); }
ZK_HD qm31 qm31_mul_m31(qm31 x, uint32_t y) {
    return {{m31_mul(x.c[0], y), m31_mul(x.c[1], y), m31_mul(x.c[2], y), m31_mul(x.c[3], y)}};
}
ZK_HD bool qm31_eq(qm31 x, qm31 y) {
    return x.c[0] == y.c[0] && x.c[1] == y.c[1] && x.c[2] == y.c[2] && x.c[3] == y.c[3];
}
ZK_HD bool qm31_is_zero(qm31 x) { return (x.c[0] | x.c[1] | x.c[2] | x.c[3]) == 0; }
// (A + B u)(C + D u) = (AC + (2+i) BD) + (AD + BC) u, qm31.rs:80-88. (2+i) D = e0 + e1 i is formed first, so that every output
// coordinate is four 62-bit products and one fold: folding BD before it is multiplied by 2+i is two folds more, on the longest
// path (233 -> 319 G products/s over all SMs, latency 188 -> 163 cycles). Subtracted products take p - x for x. 4 p^2 < 2^64.
// What is in r is added: a canonical word or a folded sum, at most 3 (2^32 - 1) = 2^34 - 2^32 - 3; 4 p^2 = 2^64 - 2^34 + 4.
ZK_HD void qm31_add_products(uint64_t (&r)[4], qm31 x, qm31 y) {
    const uint32_t e0 = m31_sub(m31_dbl(y.c[2]), y.c[3]), e1 = m31_add(y.c[2], m31_dbl(y.c[3]));
    const uint32_t n1 = P - x.c[1], n3 = P - x.c[3];
    const uint64_t x0 = x.c[0], x1 = x.c[1], x2 = x.c[2], x3 = x.c[3];
    r[0] += x0 * y.c[0] + (uint64_t)n1 * y.c[1] + x2 * e0 + (uint64_t)n3 * e1;
    r[1] += x0 * y.c[1] + x1 * y.c[0] + x2 * e1 + x3 * e0;
    r[2] += x0 * y.c[2] + (uint64_t)n1 * y.c[3] + x2 * y.c[0] + (uint64_t)n3 * y.c[1];
    r[3] += x0 * y.c[3] + x1 * y.c[2] + x2 * y.c[1] + x3 * y.c[0];
}
ZK_HD qm31 qm31_reduce64(const uint64_t (&r)[4]) { return {{m31_reduce64(r[0]), m31_reduce64(r[1]), m31_reduce64(r[2]), m31_reduce64(r[3])}}; }
ZK_HD qm31 qm31_mul(qm31 x, qm31 y) {
    uint64_t r[4] = {0, 0, 0, 0};
    qm31_add_products(r, x, y);
    return qm31_reduce64(r);
}
// x y + z: the addition is an operand of the first multiply-add
ZK_HD qm31 qm31_mul_add(qm31 x, qm31 y, qm31 z) {
    uint64_t r[4] = {z.c[0], z.c[1], z.c[2], z.c[3]};
    qm31_add_products(r, x, y);
    return qm31_reduce64(r);
}
ZK_HD qm31 qm31_sqr(qm31 x) { return qm31_mul(x, x); }
// A sum of secure products, its coordinates folded (at most 3 (2^32 - 1)) and not reduced. Adding a product costs its sixteen multiply-adds and four folds; the
// reductions and additions that a product and a sum of its own would take, half of their ALU instructions, come once at the end.
struct qm31_sum {
    uint64_t c[4];
    ZK_HD void add_product(qm31 x, qm31 y) {
        qm31_add_products(c, x, y);
        for (int k = 0; k < 4; k++) c[k] = m31_fold64(c[k]);
    }
    ZK_HD qm31 value() const { return qm31_reduce64(c); }
};
ZK_HD qm31_sum qm31_sum_zero() { return {{0, 0, 0, 0}}; }
// x0 y0 + x1 y1
ZK_HD qm31 qm31_dot2(qm31 x0, qm31 y0, qm31 x1, qm31 y1) {
    qm31_sum s = qm31_sum_zero();
    s.add_product(x0, y0);
    qm31_add_products(s.c, x1, y1);
    return s.value();
}
ZK_HD qm31 qm31_dot2_m31(qm31 x0, uint32_t y0, qm31 x1, uint32_t y1) {
    return {{m31_reduce64((uint64_t)x0.c[0] * y0 + (uint64_t)x1.c[0] * y1), m31_reduce64((uint64_t)x0.c[1] * y0 + (uint64_t)x1.c[1] * y1),
             m31_reduce64((uint64_t)x0.c[2] * y0 + (uint64_t)x1.c[2] * y1), m31_reduce64((uint64_t)x0.c[3] * y0 + (uint64_t)x1.c[3] * y1)}};
}
ZK_HD qm31 qm31_mul_cm31(qm31 x, cm31 y) {
    cm31 a = cm31_mul({x.c[0], x.c[1]}, y), b = cm31_mul({x.c[2], x.c[3]}, y);
    return {{a.a, a.b, b.a, b.b}};
}
// (a + bu)^-1 = (a - bu) / (a^2 - (2+i) b^2), qm31.rs:118-127
ZK_HD qm31 qm31_inv(qm31 x) {
    cm31 a{x.c[0], x.c[1]}, b{x.c[2], x.c[3]};
    cm31 b2 = cm31_mul(b, b);
    cm31 ib2{m31_neg(b2.b), b2.a};
    cm31 denom = cm31_sub(cm31_mul(a, a), cm31_add(cm31_add(b2, b2), ib2));
    cm31 di = cm31_inv(denom);
    cm31 ra = cm31_mul(a, di), rb = cm31_mul({m31_neg(b.a), m31_neg(b.b)}, di);
    return {{ra.a, ra.b, rb.a, rb.b}};
}

// Circle group law over M31 (nitroo/crates/stwo/src/core/circle.rs:103-113).
struct cpoint { uint32_t x, y; };
ZK_HD cpoint cpoint_add(cpoint p, cpoint q) {
    uint64_t x = (uint64_t)p.x * q.x + (P_SQ - (uint64_t)p.y * q.y);
    uint64_t y = (uint64_t)p.x * q.y + (uint64_t)p.y * q.x;
    return {m31_reduce64(x), m31_reduce64(y)};
}
// pi(x) = 2x^2 - 1 (circle.rs:28-31)
ZK_HD uint32_t m31_double_x(uint32_t x) { uint32_t s = m31_sqr(x); return m31_sub(m31_add(s, s), 1u); }
ZK_HD qm31 qm31_double_x(qm31 x) { qm31 s = qm31_sqr(x); return qm31_sub(qm31_add(s, s), qm31_one()); }

}  // namespace zk
