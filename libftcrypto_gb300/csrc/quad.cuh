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
// lanes of a warp run these together (full-mask shuffles).
#pragma once
#include "ge.cuh"
#include "u4.cuh"

namespace ft {

FT_DEV void quad_shfl(fe &o, const fe &v, int src)
{
#pragma unroll
    for (int k = 0; k < 8; ++k) o.v[k] = __shfl_sync(0xffffffffu, v.v[k], src, 4);
}

FT_DEV void fe_select(fe &h, bool c, const fe &a, const fe &b)
{
#pragma unroll
    for (int k = 0; k < 8; ++k) h.v[k] = c ? a.v[k] : b.v[k];
}

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
FT_DEV void quad_p3(fe &v, int l)
{
    fe o;
    quad_shfl(o, v, (l + 1) & 3);
    fe_mul(v, v, o);
}

// p3 (T unused) doubled, to p1p1 (ge_p2_dbl)
FT_DEV void quad_dbl(fe &v, int l)
{
    fe x, y, t, s;
    quad_shfl(x, v, 3);
    quad_shfl(y, v, 1);
    fe_add(t, x, y);
    fe_select(t, l == 0, t, v);
    fe_sq(s, t); // (X+Y)^2, Y^2, Z^2, X^2
    quad_shfl(y, s, 1);
    quad_shfl(x, s, 3);
    fe_add(t, s, s);
    quad_shfl(t, t, 2);                              // 2 Z^2
    fe_addsub(v, y, x, l < 2 ? 0u : ~0u);            // lanes 0, 1: H; lanes 2, 3: G
    fe_select(t, l == 0, s, t);
    fe_sub(t, t, v);                                 // lane 0: E, lane 3: F
    fe_select(v, l == 0 || l == 3, t, v);
}

// the point's Y in y and X in x, in lanes 1 and 3
FT_DEV void quad_yx(fe &y, fe &x, const fe &v, int l)
{
    fe o;
    quad_shfl(o, v, l ^ 2);
    fe_select(y, l == 1, v, o);
    fe_select(x, l == 1, o, v);
}

// p3 plus cached, to p1p1 (ge_add)
FT_DEV void quad_add(fe &v, const fe &q, int l)
{
    fe y, x, t, s, d;
    quad_yx(y, x, v, l);
    fe_addsub(t, y, x, l == 3 ? ~0u : 0u);
    fe_select(t, l & 1, t, v);
    fe_mul(s, t, q); // T T2d, (Y+X)(Y+X)', Z Z', (Y-X)(Y-X)'
    fe_add(d, s, s);
    fe_select(d, l == 2, d, s);
    quad_shfl(y, d, l < 2 ? 1 : 2);
    quad_shfl(x, s, l < 2 ? 3 : 0);
    fe_addsub(v, y, x, l == 0 || l == 3 ? ~0u : 0u);
}

// p3 to cached (ge_p3_to_cached)
FT_DEV void quad_cached(fe &c, const fe &v, int l)
{
    fe y, x, t;
    quad_yx(y, x, v, l);
    fe_addsub(t, y, x, l == 3 ? ~0u : 0u);
    fe_mul(c, v, fe_d2());
    fe_select(c, l == 0, c, v);
    fe_select(c, l & 1, t, c);
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
