// fe_inv.cuh — inversion mod p = 2^255 - 19 by division steps, constant time.
//
// The division steps, the transition matrices of several of them and their
// use on d and e are Bernstein and Yang's ("Fast constant-time gcd computation
// and modular inversion", 2019).  The variant that starts at delta = 1/2 and
// its bound of 590 steps for 256 bits are P. Wuille's (safegcd-bounds, 2021).
// The layout, nine signed limbs of 30 bits, 20 rounds of 30 steps, d and e kept
// in (-2p, p) and brought into [0, p) in two additions at the end, is the one
// that P. Dettman and P. Wuille describe for libsecp256k1 ("The safegcd
// implementation in libsecp256k1 explained", 2021).  The steps by multiply-adds
// and the split over the four lanes of a quad (quad_inv) are this library's.
//
// z^(p-2) is a chain of 254 squarings that nothing in one thread overlaps:
// 75 us on a warp alone, whatever the number of points it serves; this takes
// 17, and 12 with a quad of lanes per inverse (quad_inv).  A
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
// (u f + v g, q f + r g); eta = -(delta + 1/2).  What a step adds to g, q and r
// is m = 0, 1 or -1 times f, u and v, by multiply-adds: the logic pipe, which
// the masks for it would go through, is what bounds a step.
FT_DEV void inv_steps(int32_t &eta, uint32_t f, uint32_t g, int32_t &mu, int32_t &mv, int32_t &mq, int32_t &mr)
{
    uint32_t u = 1, v = 0, q = 0, r = 1;
#pragma unroll 6
    for (int i = 0; i < INV_BITS; ++i) {
        const uint32_t odd = g & 1u;
        const uint32_t swap = (0u - odd) & (uint32_t)(eta >> 31); // g odd and delta > 0
        const uint32_t m = odd + 2u * swap;
        // g + f where g is odd, g - f with a swap; f becomes the old g
        const uint32_t g1 = g + m * f, q1 = q + m * u, r1 = r + m * v;
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

// x = (a d + b e + k p) / 2^30.  With the mask modp: k makes it whole and keeps
// x in (-2p, p): a negative d or e (in (-2p, 0)) counts as itself plus p, then
// up to 2^30 - 1 times p are taken away.  Without: k = 0, the sum is whole.
FT_DEV void inv_row(int32_t x[INV_LIMBS], const int32_t d[INV_LIMBS], const int32_t e[INV_LIMBS], int32_t a, int32_t b,
                    int32_t modp)
{
    constexpr uint32_t INV19 = 678152731u; // 19 * INV19 = 1 (mod 2^30)
    int32_t k = (a & (d[INV_LIMBS - 1] >> 31)) + (b & (e[INV_LIMBS - 1] >> 31));
    int64_t c = (int64_t)a * d[0] + (int64_t)b * e[0];
    // c + k p = c - 19 k (mod 2^30): take away m p, m = -(c - 19 k) / 19 mod 2^30
    const uint32_t m = (0u - ((uint32_t)c * INV19 - (uint32_t)k)) & (uint32_t)INV_MASK;
    k = (k - (int32_t)m) & modp;
    c -= (int64_t)19 * k;
    c >>= INV_BITS;
#pragma unroll
    for (int i = 1; i < INV_LIMBS; ++i) {
        c += (int64_t)a * d[i] + (int64_t)b * e[i];
        if (i == INV_LIMBS - 1) c += (int64_t)k * (1 << 15);
        x[i - 1] = (int32_t)c & INV_MASK; // (x may be d: limb i - 1 of it is done with)
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

// limb i of p
FT_DEV int32_t inv_p(int i) { return i == 0 ? INV_MASK - 18 : i == INV_LIMBS - 1 ? (1 << 15) - 1 : INV_MASK; }

// the limbs of a canonical value
FT_DEV void inv_limbs(int32_t g[INV_LIMBS], const fe &c)
{
#pragma unroll
    for (int i = 0; i < INV_LIMBS; ++i) {
        const int w = 30 * i / 32, b = 30 * i % 32;
        uint32_t x = c.v[w] >> b;
        if (b > 2 && w < 7) x |= c.v[w + 1] << (32 - b);
        g[i] = (int32_t)(x & (uint32_t)INV_MASK);
    }
}

// d, in (-2p, p), negated under the mask neg, as a field element below p
FT_DEV void inv_finish(fe &out, int32_t d[INV_LIMBS], int32_t neg)
{
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

// out = 1/z mod p, below p; 0 for z = 0
FT_DEV void fe_inv(fe &out, const fe &z)
{
    fe c;
    fe_canon(c, z);
    int32_t f[INV_LIMBS], g[INV_LIMBS], d[INV_LIMBS], e[INV_LIMBS], x[INV_LIMBS];
    inv_limbs(g, c);
#pragma unroll
    for (int i = 0; i < INV_LIMBS; ++i) {
        f[i] = inv_p(i);
        d[i] = 0;
        e[i] = i == 0;
    }
    int32_t eta = -1;
#pragma unroll 1
    for (int round = 0; round < INV_ROUNDS; ++round) {
        int32_t u, v, q, r;
        const uint32_t f0 = (uint32_t)f[0] | (uint32_t)f[1] << 30, g0 = (uint32_t)g[0] | (uint32_t)g[1] << 30;
        inv_steps(eta, f0, g0, u, v, q, r);
        inv_row(x, d, e, u, v, -1);
        inv_row(e, e, d, r, q, -1);
#pragma unroll
        for (int i = 0; i < INV_LIMBS; ++i) d[i] = x[i];
        inv_row(x, f, g, u, v, 0);
        inv_row(g, g, f, r, q, 0);
#pragma unroll
        for (int i = 0; i < INV_LIMBS; ++i) f[i] = x[i];
    }
    // f = +-1 (p itself where z = 0, with d = 0): 1/z = d f
    inv_finish(out, d, f[INV_LIMBS - 1] >> 31);
}
