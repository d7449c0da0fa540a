// comb256.cuh — the fixed-base comb in signed radix 256, its entries looked
// up by the tensor cores (k_comb256 in k_encrypt.cu).
//
// A scalar a (enc_ref_scalar's: below 0.53 * 2^256) is first made smaller than
// 8 L, a multiple of the order of every point of the curve, and written as 32
// digits: b = a + sum_{i<31} 128 * 256^i, digit i < 31 is byte i of b minus
// 128, in [-128, 127], digit 31 is byte 31 of b, at most 128.  Then
//   a*Q = sum_i d_i * (256^i * Q):
// 32 mixed additions instead of radix 32's 52.  Reading 128 entries under
// masks would cost far more than the additions that saves.  So the lookup is
// a matrix product: row m of A is the one-hot vector of |d| of unit m, B holds
// the row of the table, every entry split into 72 f16 integers (three of 11,
// 11 and 10 bits per 32-bit word), and the f32 products are 1 * value plus
// zeros: exact.  Constant time: every entry takes part in every product, no
// address depends on a digit.
//
// A table row is a K-major B operand of COMB_K = 128 entries x COMB_N = 80
// columns (72 used): element (column n, entry k) at (k / 8) * 16 COMB_N +
// n * 16 + (k % 8) * 2, entry k = (k + 1) * 256^row * Q.  Column 24 f + 8 c + w
// is part c of word w of coordinate f ((y+x)/2, (y-x)/2, dxy).
#pragma once
#include "ge.cuh"

static constexpr int COMB_ROWS = 32, COMB_K = 128, COMB_N = 80;
static constexpr int COMB_CHUNK = 16 * COMB_N;                   // bytes of 8 entries
static constexpr int COMB_ROW_BYTES = COMB_K / 8 * COMB_CHUNK;   // a table row

// rows of a value below 2^bits (bits <= 64): the top digit carries no bias
// and is at most 128
constexpr int comb_rows(unsigned bits) { return bits / 8 + 1; }

// a - 8 L where a >= 8 L (a < 16 L), in constant time
FT_DEV void comb_reduce(uint32_t a[8])
{
    constexpr uint32_t L8[8] = {0xe7ae9f68u, 0xc09318d2u, 0x17bce6b2u, 0xa6f7cef5u, 0u, 0u, 0u, 0x80000000u};
    uint32_t r[8];
    r[0] = sub_cc(a[0], L8[0]);
#pragma unroll
    for (int k = 1; k < 8; ++k) r[k] = subc_cc(a[k], L8[k]);
    const uint32_t keep = subc(0u, 0u); // all ones: a < 8 L
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = (a[k] & keep) | (r[k] & ~keep);
}

// b = a + sum_{i<31} 128 * 256^i
FT_DEV void comb_recode(uint32_t b[8], const uint32_t a[8])
{
    b[0] = add_cc(a[0], 0x80808080u);
#pragma unroll
    for (int k = 1; k < 7; ++k) b[k] = addc_cc(a[k], 0x80808080u);
    b[7] = addc(a[7], 0x00808080u);
}

// the same for a 64-bit value in `rows` digits (72 bits)
FT_DEV void comb_recode_small(uint32_t b[3], uint64_t m, int rows)
{
    const uint64_t bias = rows >= 9 ? 0x8080808080808080ull : 0x8080808080808080ull & ((1ull << (8 * (rows - 1))) - 1ull);
    b[0] = add_cc((uint32_t)m, (uint32_t)bias);
    b[1] = addc_cc((uint32_t)(m >> 32), (uint32_t)(bias >> 32));
    b[2] = addc(0u, 0u);
}

// the signed digit in byte `row & 3` of word `row >> 2`
FT_DEV int comb_digit(uint32_t word, int row, bool top) { return (int)(word >> (8 * (row & 3)) & 255u) - (top ? 0 : 128); }

FT_DEV int comb_offset(int n, int k) { return (k >> 3) * COMB_CHUNK + n * 16 + (k & 7) * 2; }

// part c of a table word
FT_DEV uint32_t comb_part(uint32_t w, int c) { return c == 0 ? w & 2047u : c == 1 ? w >> 11 & 2047u : w >> 22; }

// The product adds 2^23 to every column, so that its f32 is the integer with
// the exponent bits 0x4b000000, and 724 to the columns of part 2: 16 entries
// more, the same in all rows, of which every row of A selects the first 2048
// times and the second once (the f16 pair COMB_MAGIC_A).  The pair of column n:
static constexpr uint32_t COMB_MAGIC_A = 0x3c006800u;

FT_DEV uint32_t comb_magic(int n)
{
    return n >= 72 ? 0u : (n / 8 % 3 == 2 ? 0x61a80000u : 0u) | 0x6c00u; // 4096 and 724 or 0
}

// the table word of its three columns' bits: shifted by 11 and 22 the exponent
// bits are gone, and 724 << 22 (0x2d4 << 22) cancels those of the first
FT_DEV uint32_t comb_word(uint32_t p0, uint32_t p1, uint32_t p2) { return (p2 << 22) + (p1 << 11) + p0; }

// -f for the canonical f under the mask (a table word group: f < 2^255)
FT_DEV void comb_neg(fe &f, uint32_t m)
{
    uint32_t r[8]; // ~f = 2^256 - 1 - f, that is -f + 37 (mod p), at least 2^255
    r[0] = sub_cc(f.v[0] ^ m, 37u & m);
#pragma unroll
    for (int k = 1; k < 7; ++k) r[k] = subc_cc(f.v[k] ^ m, 0u);
    r[7] = subc(f.v[7] ^ m, 0u);
#pragma unroll
    for (int k = 0; k < 8; ++k) f.v[k] = r[k];
}

// the entry of |d| negated for d < 0
FT_DEV void comb_signed(ge_precomp &t, int d)
{
    const uint32_t neg = 0u - ((uint32_t)d >> 31);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t p = t.yplusx.v[k], q = t.yminusx.v[k];
        t.yplusx.v[k] = (p & ~neg) | (q & neg);
        t.yminusx.v[k] = (q & ~neg) | (p & neg);
    }
    comb_neg(t.xy2d, neg);
}

// ---- additions of halved entries, on tight coordinates (fe.cuh)
//
// With (y+x)/2, (y-x)/2 and dxy in an entry the four intermediate coordinates
// come out halved, the same point, and 2 Z is Z: one sum fewer, and the others
// tight (1,048,576 ciphertexts 5.45 -> 5.22 ms).

// h += the entry t (ge_madd and ge_p1p1_to_p3 on halves)
FT_DEV void comb_add(ge_p3 &h, const ge_precomp &t)
{
    fe e, f, g, k;
    add_tight(g, h.Y, h.X);
    sub_tight(f, h.Y, h.X);
    mul_tight_x2(g, g, t.yplusx, f, f, t.yminusx);
    sub_tight(e, g, f);
    add_tight(k, g, f);
    mul_tight(g, t.xy2d, h.T);
    sub_tight(f, h.Z, g);
    add_tight(g, h.Z, g);
    mul_tight_x2(h.X, e, f, h.Y, k, g);
    mul_tight_x2(h.Z, g, f, h.T, e, k);
}

// h = the entry itself: x = (y+x)/2 - (y-x)/2, y their sum (both below 2^255)
FT_DEV void comb_first(ge_p3 &h, const ge_precomp &t)
{
    fe one;
    fe_1(one);
    fe_sub(h.X, t.yplusx, t.yminusx);
    fe_add(h.Y, t.yplusx, t.yminusx);
    mul_tight(h.T, h.X, h.Y);
    mul_tight_x2(h.X, h.X, one, h.Y, h.Y, one);
    h.Z = one;
}

// 1/2 mod p = 2^254 - 9
FT_DEV fe fe_half() { return fe_const(0xfffffff7u, ~0u, ~0u, ~0u, ~0u, ~0u, ~0u, 0x3fffffffu); }

// word w of the identity's entry (1/2, 1/2, 0)
FT_DEV uint32_t comb_identity(int w) { return w >= 16 ? 0u : (w & 7) == 0 ? 0xfffffff7u : (w & 7) == 7 ? 0x3fffffffu : ~0u; }
