// fe_inv.cuh — inversion mod p = 2^255 - 19 by division steps (Bernstein and
// Yang, "Fast constant-time gcd computation and modular inversion", 2019, in
// the variant that starts at delta = 1/2), constant time.
//
// z^(p-2) is a chain of 254 squarings that nothing in one thread overlaps:
// 75 us on a warp alone, whatever the number of points it serves.  A
// division step works on the low words of f and g only: 30 of them give a
// 2 x 2 matrix of 31-bit entries, which is then applied to f, g (exactly
// divisible by 2^30) and to d, e (divisible mod p), with d z = f and e z = g
// (mod p) throughout.  From f = p, g = z, 590 steps take every g below 2^256
// to 0 and f to +-1; 20 rounds of 30 are 600.
//
// f, g, d, e are nine limbs of 30 bits, two's complement: limbs 0-7 in
// [0, 2^30), limb 8 signed.  p is 2^15 in limb 8 and -19 in limb 0.
#pragma once
#include "fe.cuh"

static constexpr int INV_LIMBS = 9, INV_BITS = 30, INV_ROUNDS = 20;
static constexpr int32_t INV_MASK = (1 << INV_BITS) - 1;

// 30 division steps on the low words of f and g: (f, g) 2^30 becomes
// (u f + v g, q f + r g); eta = -(delta + 1/2)
FT_DEV void inv_steps(int32_t &eta, uint32_t f, uint32_t g, int32_t &mu, int32_t &mv, int32_t &mq, int32_t &mr)
{
    uint32_t u = 1, v = 0, q = 0, r = 1;
#pragma unroll 6
    for (int i = 0; i < INV_BITS; ++i) {
        const uint32_t odd = 0u - (g & 1u);
        const uint32_t swap = odd & (uint32_t)(eta >> 31); // g odd and delta > 0
        // g + f where g is odd, g - f with a swap; f becomes the old g
        const uint32_t g1 = g + ((f & odd) ^ swap) - swap;
        const uint32_t q1 = q + ((u & odd) ^ swap) - swap;
        const uint32_t r1 = r + ((v & odd) ^ swap) - swap;
        f = (g & swap) | (f & ~swap);
        u = ((q & swap) | (u & ~swap)) << 1;
        v = ((r & swap) | (v & ~swap)) << 1;
        eta = (int32_t)((uint32_t)eta ^ swap) - 1;
        g = g1 >> 1; // the top bits are never used: 30 steps read the low 30
        q = q1;
        r = r1;
    }
    mu = (int32_t)u;
    mv = (int32_t)v;
    mq = (int32_t)q;
    mr = (int32_t)r;
}

// (f, g) = (u f + v g, q f + r g) / 2^30, exact
FT_DEV void inv_apply(int32_t f[INV_LIMBS], int32_t g[INV_LIMBS], int32_t u, int32_t v, int32_t q, int32_t r)
{
    int64_t cf = (int64_t)u * f[0] + (int64_t)v * g[0];
    int64_t cg = (int64_t)q * f[0] + (int64_t)r * g[0];
    cf >>= INV_BITS;
    cg >>= INV_BITS;
#pragma unroll
    for (int i = 1; i < INV_LIMBS; ++i) {
        cf += (int64_t)u * f[i] + (int64_t)v * g[i];
        cg += (int64_t)q * f[i] + (int64_t)r * g[i];
        f[i - 1] = (int32_t)cf & INV_MASK;
        g[i - 1] = (int32_t)cg & INV_MASK;
        cf >>= INV_BITS;
        cg >>= INV_BITS;
    }
    f[INV_LIMBS - 1] = (int32_t)cf;
    g[INV_LIMBS - 1] = (int32_t)cg;
}

// x = (u d + v e + k p) / 2^30 for the k that makes it whole and keeps x in
// (-2p, p): a negative d or e (in (-2p, 0)) counts as itself plus p, then
// up to 2^30 - 1 times p are taken away
FT_DEV void inv_row_mod_p(int32_t x[INV_LIMBS], const int32_t d[INV_LIMBS], const int32_t e[INV_LIMBS], int32_t u,
                          int32_t v)
{
    constexpr uint32_t INV19 = 678152731u; // 19 * INV19 = 1 (mod 2^30)
    int32_t k = (u & (d[INV_LIMBS - 1] >> 31)) + (v & (e[INV_LIMBS - 1] >> 31));
    int64_t c = (int64_t)u * d[0] + (int64_t)v * e[0];
    // c + k p = c - 19 k (mod 2^30): take away m p, m = -(c - 19 k) / 19 mod 2^30
    const uint32_t m = (0u - ((uint32_t)c * INV19 - (uint32_t)k)) & (uint32_t)INV_MASK;
    k -= (int32_t)m;
    c -= (int64_t)19 * k;
    c >>= INV_BITS;
#pragma unroll
    for (int i = 1; i < INV_LIMBS; ++i) {
        c += (int64_t)u * d[i] + (int64_t)v * e[i];
        if (i == INV_LIMBS - 1) c += (int64_t)k * (1 << 15);
        x[i - 1] = (int32_t)c & INV_MASK;
        c >>= INV_BITS;
    }
    x[INV_LIMBS - 1] = (int32_t)c;
}

// x += p under the mask; limbs 0-7 back in [0, 2^30)
FT_DEV void inv_add_p(int32_t x[INV_LIMBS], int32_t mask)
{
    int32_t c = x[0] - (19 & mask);
#pragma unroll
    for (int i = 0; i < INV_LIMBS - 1; ++i) {
        x[i] = c & INV_MASK;
        c = x[i + 1] + (c >> INV_BITS);
    }
    x[INV_LIMBS - 1] = c + ((1 << 15) & mask);
}

// out = 1/z mod p, below p; 0 for z = 0
FT_DEV void fe_inv(fe &out, const fe &z)
{
    fe c;
    fe_canon(c, z);
    int32_t f[INV_LIMBS], g[INV_LIMBS], d[INV_LIMBS], e[INV_LIMBS];
#pragma unroll
    for (int i = 0; i < INV_LIMBS; ++i) {
        const int w = 30 * i / 32, b = 30 * i % 32;
        uint32_t x = c.v[w] >> b;
        if (b > 2 && w < 7) x |= c.v[w + 1] << (32 - b);
        g[i] = (int32_t)(x & (uint32_t)INV_MASK);
        f[i] = i == 0 ? INV_MASK - 18 : i == INV_LIMBS - 1 ? (1 << 15) - 1 : INV_MASK; // p
        d[i] = 0;
        e[i] = i == 0;
    }
    int32_t eta = -1;
#pragma unroll 1
    for (int round = 0; round < INV_ROUNDS; ++round) {
        int32_t u, v, q, r, x[INV_LIMBS];
        const uint32_t f0 = (uint32_t)f[0] | (uint32_t)f[1] << 30, g0 = (uint32_t)g[0] | (uint32_t)g[1] << 30;
        inv_steps(eta, f0, g0, u, v, q, r);
        inv_row_mod_p(x, d, e, u, v);
        inv_row_mod_p(e, d, e, q, r);
#pragma unroll
        for (int i = 0; i < INV_LIMBS; ++i) d[i] = x[i];
        inv_apply(f, g, u, v, q, r);
    }
    // f = +-1 (p itself where z = 0, with d = 0): 1/z = d f, d in (-2p, p)
    const int32_t neg = f[INV_LIMBS - 1] >> 31;
    inv_add_p(d, d[INV_LIMBS - 1] >> 31);
#pragma unroll
    for (int i = 0; i < INV_LIMBS; ++i) d[i] = (d[i] ^ neg) - neg;
    inv_add_p(d, 0); // carries of the negation
    inv_add_p(d, d[INV_LIMBS - 1] >> 31);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        const int i = 32 * w / 30, b = 32 * w % 30;
        uint32_t x = (uint32_t)d[i] >> b | (uint32_t)d[i + 1] << (30 - b);
        if (i + 2 < INV_LIMBS && 60 - b < 32) x |= (uint32_t)d[i + 2] << (60 - b);
        out.v[w] = x;
    }
}
