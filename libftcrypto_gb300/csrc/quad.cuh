// quad.cuh — group operations with the four lanes of a quad on one point.
//
// Every formula of ge.cuh is rounds of four independent field operations:
// the four products (or squarings) of an addition (or doubling), then the
// four products that make it projective again.  Lane l of a quad does one of
// each round, and holds one coordinate of a point:
//
//   lane        0             1             2             3
//   p3          T             Y             Z             X
//   cached      T2d           Y+X           Z             Y-X
//   p1p1        X ("E")       Y ("H")       Z ("G")       T ("F")
//
// so that p1p1 to p3 is one product with the next lane's value: E H = T,
// H G = Y, G F = Z, F E = X.  The operands and the order of every field
// operation are those of ge.cuh, so coordinates are the same words.  All
// lanes of a warp run these together.
#pragma once
#include "ge.cuh"
#include "fe_inv.cuh"
#include "u4.cuh"

namespace ft {

// b where the mask is set, else a
FT_DEV void fe_pick(fe &h, const fe &a, const fe &b, uint32_t m)
{
#pragma unroll
    for (int k = 0; k < 8; ++k) h.v[k] = (a.v[k] & ~m) | (b.v[k] & m);
}

// all ones in the lanes l of `lanes`; opaque, so that a pick stays a pick (as a
// condition the compiler branches around each one's eight moves: a point's
// ladder 345 us against 244)
FT_DEV uint32_t quad_mask(int l, unsigned lanes)
{
    uint32_t m = 0u - (lanes >> l & 1u);
    asm volatile("" : "+r"(m));
    return m;
}

// Lanes trade values through shared memory, two uint4 a thread in one of two
// buffers in turn (`slot`): a value written once is read by any number of
// lanes, and one warp barrier orders it (a shuffle moves one word and brings a
// barrier of its own).
struct QuadX {
    uint4 *slot; // this thread's, buffer 0: [buffer][half][thread], 4 * threads uint4
    int stride;  // threads of the block
    int l;       // the lane's place in its quad
    uint32_t m0, m1, m03, m13, m23; // quad_mask of those lanes
    int flip = 0;
    FT_DEV QuadX(uint4 *buf, int threads)
        : slot(buf + threadIdx.x), stride(threads), l(threadIdx.x & 3), m0(quad_mask(l, 1)), m1(quad_mask(l, 2)),
          m03(quad_mask(l, 9)), m13(quad_mask(l, 10)), m23(quad_mask(l, 12))
    {
    }
    FT_DEV void put(const fe &v)
    {
        flip ^= 2 * stride;
        slot[flip] = u4_lo(v);
        slot[flip + stride] = u4_hi(v);
        __syncwarp();
    }
    // the value that lane `src` of the quad put last
    FT_DEV void get(fe &o, int src) const
    {
        const uint4 *q = slot + flip + src - l;
        fe_from_u4(o, q[0], q[stride]);
    }
};

// a + b for m = 0 (the words of fe_add), a - b for m = all ones (fe_sub's)
FT_DEV void fe_addsub(fe &h, const fe &a, const fe &b, uint32_t m)
{
    uint32_t r[8];
    (void)add_cc(m, 1u); // carry in: 1 to subtract (a + ~b + 1)
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = addc_cc(a.v[k], b.v[k] ^ m);
    uint32_t c = addc(0u, m);                // 1: carry to repay, -1: borrow, 0: neither
    const uint32_t s = (uint32_t)((int)c >> 31);
    r[0] = add_cc(r[0], 38u * c);
#pragma unroll
    for (int k = 1; k < 8; ++k) r[k] = addc_cc(r[k], s);
    c = addc(0u, s);
    r[0] += 38u * c;
#pragma unroll
    for (int k = 0; k < 8; ++k) h.v[k] = r[k];
}

// p1p1 to p3
FT_DEV void quad_p3(fe &v, QuadX &x)
{
    fe o;
    x.put(v);
    x.get(o, (x.l + 1) & 3);
    fe_mul(v, v, o);
}

// p3 (T unused) doubled, to p1p1 (ge_p2_dbl)
FT_DEV void quad_dbl(fe &v, QuadX &x)
{
    fe a, b, t, s;
    x.put(v);
    x.get(a, 3);
    x.get(b, 1);
    fe_add(t, a, b);
    fe_pick(t, v, t, x.m0);
    fe_sq(s, t); // (X+Y)^2, Y^2, Z^2, X^2
    x.put(s);
    x.get(a, 1);
    x.get(b, 3);
    x.get(t, 2);
    fe_add(t, t, t);           // 2 Z^2
    fe_addsub(v, a, b, x.m23); // lanes 0, 1: H; lanes 2, 3: G
    fe_pick(t, t, s, x.m0);
    fe_sub(t, t, v);           // lane 0: E, lane 3: F
    fe_pick(v, v, t, x.m03);
}

// Y + X in lane 1, Y - X in lane 3, v in the others
FT_DEV void quad_yx(fe &t, const fe &v, QuadX &x)
{
    fe o, a, b;
    x.put(v);
    x.get(o, x.l ^ 2);
    fe_pick(b, o, v, x.m1);
    fe_pick(a, v, o, x.m1);
    fe_addsub(o, b, a, ~x.m1);
    fe_pick(t, v, o, x.m13);
}

// p3 plus cached, to p1p1 (ge_add)
FT_DEV void quad_add(fe &v, const fe &q, QuadX &x)
{
    fe a, b, t, s;
    quad_yx(t, v, x);
    fe_mul(s, t, q); // T T2d, (Y+X)(Y+X)', Z Z', (Y-X)(Y-X)'
    x.put(s);
    x.get(b, x.l < 2 ? 1 : 2);
    x.get(a, x.l < 2 ? 3 : 0);
    fe_add(t, b, b);
    fe_pick(b, b, t, x.m23);
    fe_addsub(v, b, a, x.m03);
}

// p3 to cached (ge_p3_to_cached)
FT_DEV void quad_cached(fe &c, const fe &v, QuadX &x)
{
    fe t;
    quad_yx(t, v, x);
    fe_mul(c, v, fe_d2());
    fe_pick(c, t, c, x.m0);
}

// 1/z for the z that the four lanes of the quad hold alike (fe_inv): the
// division steps in all of them, and of the numbers f, g, d and e the one of
// the lane, 34,300 -> 24,000 cycles
FT_DEV void quad_inv(fe &out, const fe &z)
{
    const int l = threadIdx.x & 3;
    const uint32_t hi = quad_mask(l, 10), de = quad_mask(l, 12); // g and e; d and e
    fe c;
    fe_canon(c, z);
    int32_t x[INV_LIMBS], y[INV_LIMBS], g[INV_LIMBS];
    inv_limbs(g, c);
#pragma unroll
    for (int i = 0; i < INV_LIMBS; ++i) {
        const int32_t fg = (int32_t)((uint32_t)inv_p(i) & ~hi) | (int32_t)((uint32_t)g[i] & hi);
        x[i] = (int32_t)(((uint32_t)fg & ~de) | ((i == 0 ? 1u : 0u) & hi & de));
    }
    int32_t eta = -1;
#pragma unroll 1
    for (int round = 0; round < INV_ROUNDS; ++round) {
        const uint32_t w = (uint32_t)x[0] | (uint32_t)x[1] << 30;
        int32_t u, v, q, r;
        inv_steps(eta, __shfl_sync(0xffffffffu, w, 0, 4), __shfl_sync(0xffffffffu, w, 1, 4), u, v, q, r);
        // this lane's row of the matrix, its own number's factor first
        const int32_t a = (int32_t)(((uint32_t)u & ~hi) | ((uint32_t)r & hi));
        const int32_t b = (int32_t)(((uint32_t)v & ~hi) | ((uint32_t)q & hi));
#pragma unroll
        for (int i = 0; i < INV_LIMBS; ++i) y[i] = __shfl_xor_sync(0xffffffffu, x[i], 1);
        inv_row(x, x, y, a, b, (int32_t)de);
    }
    const int32_t neg = __shfl_sync(0xffffffffu, x[INV_LIMBS - 1], 0, 4) >> 31;
#pragma unroll
    for (int i = 0; i < INV_LIMBS; ++i) y[i] = __shfl_sync(0xffffffffu, x[i], 2, 4);
    inv_finish(out, y, neg);
}

// the lane's coordinate of point i (identity past n)
FT_DEV void quad_ld(fe &v, const uint4 *p, size_t s, size_t i, size_t n, int l)
{
    const int plane = l == 0 ? 6 : l == 3 ? 0 : 2 * l;
    if (i < n) {
        fe_from_u4(v, p[plane * s + i], p[(plane + 1) * s + i]);
    } else {
        fe_0(v);
        v.v[0] = l == 1 || l == 2;
    }
}

FT_DEV void quad_st(uint4 *p, size_t s, size_t i, const fe &v, int l)
{
    const int plane = l == 0 ? 6 : l == 3 ? 0 : 2 * l;
    p[plane * s + i] = u4_lo(v);
    p[(plane + 1) * s + i] = u4_hi(v);
}

} // namespace ft
