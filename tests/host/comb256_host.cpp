// comb256_host.cpp — host build of the radix-256 comb (comb256.cuh) over the C
// stand-ins of ptx_emul.h, with the matrix product of the lookup written out
// as the one product it keeps, for tests/test_comb256_host.py.  TEST HARNESS
// ONLY.
#include <string.h>
#include <vector>
#include "../../libftcrypto_gb300/csrc/u4.cuh"
#include "../../libftcrypto_gb300/csrc/enc_comb.cuh"
#include "../../libftcrypto_gb300/csrc/comb256.cuh"
#include "../../libftcrypto_gb300/csrc/fe_inv.cuh"

static std::vector<float> g_tab; // [row][offset / 2]
static bool g_tight = true;

// f < 2^255 + 1463
static bool tight(const fe &f)
{
    if (!(f.v[7] >> 31)) return true;
    for (int k = 1; k < 8; ++k)
        if (f.v[k] != (k == 7 ? 0x80000000u : 0u)) return false;
    return f.v[0] < 1463u;
}

static void put_row(int row, const ge_p3 &base)
{
    ge_p3 acc = base;
    ge_cached c;
    ge_p3_to_cached(c, base);
    float *o = &g_tab[(size_t)row * COMB_ROW_BYTES / 2];
    for (int k = 0; k < COMB_K; ++k) {
        fe zi, x, y, xy, e[3];
        fe_inv(zi, acc.Z);
        fe_mul(x, acc.X, zi);
        fe_mul(y, acc.Y, zi);
        fe_mul(xy, x, y);
        fe_mul(e[2], xy, fe_d());
        fe_mul(x, x, fe_half());
        fe_mul(y, y, fe_half());
        fe_add(e[0], y, x);
        fe_sub(e[1], y, x);
        for (int j = 0; j < 3; ++j) {
            fe_canon(e[j], e[j]);
            for (int w = 0; w < 8; ++w)
                for (int p = 0; p < 3; ++p) o[comb_offset(24 * j + 8 * p + w, k) / 2] = (float)comb_part(e[j].v[w], p);
        }
        ge_p1p1 r;
        ge_add(r, acc, c);
        ge_p1p1_to_p3(acc, r);
    }
}

// the value of a normal f16, 0 for 0
static float half(uint32_t bits)
{
    bits &= 0xffffu;
    return bits ? (float)((bits & 1023u) + 1024u) * (float)(1u << (bits >> 10)) / 33554432.0f : 0.0f;
}

static void add_row(ge_p3 &h, bool first, int row, int d)
{
    ge_precomp e;
    const int k = (d < 0 ? -d : d) - 1;
    fe *f[3] = {&e.yplusx, &e.yminusx, &e.xy2d};
    const float *o = &g_tab[(size_t)row * COMB_ROW_BYTES / 2];
    for (int w = 0; w < 24; ++w) {
        uint32_t p[3];
        for (int c = 0; c < 3; ++c) {
            const int n = 24 * (w / 8) + 8 * c + w % 8;
            const uint32_t m = comb_magic(n);
            const float x = half(COMB_MAGIC_A) * half(m) + half(COMB_MAGIC_A >> 16) * half(m >> 16) +
                            (k < 0 ? (float)comb_part(comb_identity(w), c) : o[comb_offset(n, k) / 2]);
            memcpy(&p[c], &x, 4);
        }
        f[w / 8]->v[w % 8] = comb_word(p[0], p[1], p[2]);
    }
    comb_signed(e, d);
    if (first) {
        comb_first(h, e);
    } else {
        comb_add(h, e);
        for (const fe *c : {&h.X, &h.Y, &h.Z, &h.T}) g_tight = g_tight && tight(*c);
    }
}

extern "C" {

// whether every coordinate so far was below 2^255 + 1463
int hc_comb256_tight(void) { return g_tight; }

// mul_tight's and fe_tighten's bounds on any operands; sums and differences of
// what they give
int hc_comb256_field(const uint8_t *a32, const uint8_t *b32, uint8_t *prod32, uint8_t *sum32, uint8_t *diff32)
{
    fe a, b, p, s;
    memcpy(a.v, a32, 32);
    memcpy(b.v, b32, 32);
    mul_tight(p, a, b);
    memcpy(prod32, p.v, 32);
    add_tight(s, p, p);
    memcpy(sum32, s.v, 32);
    fe_tighten(a);
    fe_tighten(b);
    sub_tight(s, a, b);
    memcpy(diff32, s.v, 32);
    return tight(p) && tight(a) && tight(b);
}


void hc_comb256_table(const uint8_t *q128)
{
    g_tab.assign((size_t)COMB_ROWS * COMB_ROW_BYTES / 2, 0.0f);
    ge_p3 Q;
    memcpy(Q.X.v, q128, 32);
    memcpy(Q.Y.v, q128 + 32, 32);
    memcpy(Q.Z.v, q128 + 64, 32);
    memcpy(Q.T.v, q128 + 96, 32);
    for (int row = 0; row < COMB_ROWS; ++row) {
        put_row(row, Q);
        for (int i = 0; i < 8; ++i) {
            ge_p1p1 r;
            ge_p3_dbl(r, Q);
            ge_p1p1_to_p3(Q, r);
        }
    }
}

// a_i * Q by the 32 rows, and the digits
void hc_comb256(uint8_t *pts, int32_t *digits, const uint8_t *scalars, size_t n)
{
    for (size_t i = 0; i < n; ++i) {
        uint32_t s[8], a[8], b[8];
        memcpy(s, scalars + 32 * i, 32);
        enc_ref_scalar(a, s);
        comb_reduce(a);
        comb_recode(b, a);
        ge_p3 h;
        for (int row = COMB_ROWS - 1; row >= 0; --row) {
            const int d = comb_digit(b[row >> 2], row, row == COMB_ROWS - 1);
            digits[32 * i + row] = d;
            add_row(h, row == COMB_ROWS - 1, row, d);
        }
        memcpy(pts + 128 * i, &h, 128);
    }
}

// m_i * Q for m_i < 2^bits
void hc_comb256_small(uint8_t *pts, const uint64_t *m, size_t n, unsigned bits)
{
    const int rows = comb_rows(bits);
    for (size_t i = 0; i < n; ++i) {
        uint32_t b[3];
        comb_recode_small(b, m[i], rows);
        ge_p3 h;
        for (int row = 0; row < rows; ++row) add_row(h, row == 0, row, comb_digit(b[row >> 2], row, row == rows - 1));
        memcpy(pts + 128 * i, &h, 128);
    }
}

} // extern "C"
