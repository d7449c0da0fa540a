// k_smul.cu — the constant-time variable-base ladder with four lanes per point
// (k_smul_quad), and the dispatch between it and the one-thread ladder
// (ladder.cuh, one instantiation per block size in k_ladder.cu) by length and
// by the run-time block size knob.  The fixed-base kernels are in
// k_encrypt.cu.
#include "internal.h"
#include "ladder.cuh"
#include "quad.cuh"

namespace ft {

// Latency-bound lengths: four lanes per point (quad.cuh), so that a window's
// 36 multiplications and squarings take 10 in sequence instead of 36 (one
// point: 244 us against 553 with one thread in the 128-thread kernel).  A
// block of 128 threads holds 32 points; a thread keeps its coordinate of the
// 8-entry table in shared memory, [entry][half][thread], and scans all of it
// under masks for each digit, as the one-thread ladder does.
static constexpr int QUAD_NT = 128;

__global__ void __launch_bounds__(QUAD_NT, 5) k_smul_quad(uint4 *p, size_t s, size_t n, const uint4 *sc, int sc_step)
{
    __shared__ uint4 smem[8 * 2 * QUAD_NT], trade[4 * QUAD_NT];
    QuadX x(trade, QUAD_NT);
    const uint32_t m013 = quad_mask(threadIdx.x & 3, 11);
    uint4 *tab = smem + threadIdx.x;
    const int l = threadIdx.x & 3;
    const size_t i = ((size_t)blockIdx.x * QUAD_NT + threadIdx.x) >> 2;
    fe P, v, c;
    uint32_t b[8], a[8];
    quad_ld(P, p, s, i, n, l);
    if (i < n) {
        load_scalar(a, sc, i * (size_t)sc_step);
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = 0u;
    }
    __syncwarp();
    recode_bias(b, a);
    // entries in the order 1P, 2P, 4P, 8P (doublings of the last), 5P, 3P
    // (P + 4P, P + 2P), 6P (a doubling), 7P (P + 6P): the reference's
    // formula for each, with P and the last point live
    v = P;
    quad_cached(c, v, x);
    tab[0] = u4_lo(c);
    tab[QUAD_NT] = u4_hi(c);
#pragma unroll 1
    for (int step = 0; step < 7; ++step) {
        if (0x58 >> step & 1) {
            const int e = 0x5013000 >> (4 * step) & 7;
            fe_from_u4(c, tab[2 * e * QUAD_NT], tab[(2 * e + 1) * QUAD_NT]);
            v = P;
            quad_add(v, c, x);
        } else {
            quad_dbl(v, x);
        }
        quad_p3(v, x);
        quad_cached(c, v, x);
        const int e = 0x6524731 >> (4 * step) & 7;
        tab[2 * e * QUAD_NT] = u4_lo(c);
        tab[(2 * e + 1) * QUAD_NT] = u4_hi(c);
    }
    // the ladder of smul_ladder
    fe_0(v);
    v.v[0] = l == 1 || l == 2;
    int d = pop_top_nibble(b); // digit 63 carries no bias
#pragma unroll 1
    for (int w = 63;; --w) {
        const uint32_t bneg = (uint32_t)d >> 31, nm = 0u - bneg;
        const uint32_t babs = (uint32_t)((d ^ -(int)bneg) + (int)bneg);
        fe t;
        fe_0(c);
        c.v[0] = l != 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            fe_from_u4(t, tab[2 * k * QUAD_NT], tab[(2 * k + 1) * QUAD_NT]);
            fe_cmov(c, t, ct_eq_mask(babs, (uint32_t)(k + 1)));
        }
        // -P: Y+X and Y-X trade lanes, T2d is negated
        fe o;
        x.put(c);
        x.get(o, l ^ 2);
        fe_neg(t, c);
        fe_pick(t, o, t, x.m0);
        fe_cmov(c, t, nm & m013);
        quad_add(v, c, x);
        quad_p3(v, x);
        if (w == 0) break;
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            quad_dbl(v, x);
            quad_p3(v, x);
        }
        d = pop_top_nibble(b) - 8;
    }
    if (i < n) quad_st(p, s, i, v, l);
}

// ------------------------------------------------------------ launchers

static int g_ladder_nt = 384; // tables half in TMEM: the fastest on GB300 in whole waves

int ladder_block() { return g_ladder_nt; }

int set_ladder_block(int nt)
{
    if (nt != 128 && nt != 192 && nt != 224 && nt != 384 && nt != 448) return -1;
    g_ladder_nt = nt;
    return 0;
}

size_t ladder_wave_points()
{
    switch (g_ladder_nt) {
    case 128: return ladder_wave_128();
    case 192: return ladder_wave_192();
    case 224: return ladder_wave_224();
    case 448: return ladder_wave_448();
    default: return ladder_wave_384();
    }
}

// up to three of the quad kernel's warps per scheduler
bool ladder_is_short(size_t n) { return g_ladder_nt == 384 && n <= 96 * (size_t)sm_count(); }

static cudaError_t smul_quad(View v, size_t n, const uint4 *sc, int sc_step, cudaStream_t st)
{
    k_smul_quad<<<(unsigned)((n + QUAD_NT / 4 - 1) / (QUAD_NT / 4)), QUAD_NT, 0, st>>>(v.p, v.s, n, sc, sc_step);
    return cudaGetLastError();
}

// Fewer points than a wave of the 384-thread ladder (384 per SM) cost a whole
// one: twelve warps on each SM share its pipe for 1,134 us, on one SM or on
// all.  Measured with 152 SMs, us per launch by points per SM:
//               <= 32   <= 64   <= 96  <= 128  <= 160  <= 224  <= 256  <= 384
//   quad           244     317     441     567     688     941    1070    1569
//   128 threads    553     553     553     554    1106    1106    1106    1657
//   224 threads    771     775     775     776     776     776    1538    1544
//   384 threads   1130    1133    1133    1134    1134    1134    1134    1135
// so the points go to four lanes each up to 160 per SM, then to the largest
// block with its tables in shared memory, and to four lanes again between the
// points that holds and 256 per SM.
static cudaError_t smul_part_wave(View v, size_t n, const uint4 *sc, int sc_step, cudaStream_t st)
{
    const size_t sm = (size_t)sm_count();
    if (n <= 160 * sm) return smul_quad(v, n, sc, sc_step, st);
    if (n <= 224 * sm) return ladder_launch_224(v.p, v.s, n, sc, sc_step, st);
    if (n <= 256 * sm) return smul_quad(v, n, sc, sc_step, st);
    return ladder_launch_384(v.p, v.s, n, sc, sc_step, st);
}

// With the block size knob at 384 (the default): whole waves of the
// 384-thread ladder, then the points left over by the rule above, in a
// second launch where they do not need the 384-thread kernel.  Any other
// setting of the knob is that kernel for every length.
cudaError_t smul_var(View v, size_t n, const uint8_t *sc, int sc_step, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    const uint4 *s4 = (const uint4 *)sc;
    switch (g_ladder_nt) {
    case 128: return ladder_launch_128(v.p, v.s, n, s4, sc_step, st);
    case 192: return ladder_launch_192(v.p, v.s, n, s4, sc_step, st);
    case 448: return ladder_launch_448(v.p, v.s, n, s4, sc_step, st);
    case 224: return ladder_launch_224(v.p, v.s, n, s4, sc_step, st);
    default: break;
    }
    const size_t sm = (size_t)sm_count(), wave = 384 * sm, rest = n % wave;
    if (n < wave) return smul_part_wave(v, n, s4, sc_step, st);
    const size_t bulk = rest > 256 * sm ? n : n - rest;
    cudaError_t e = ladder_launch_384(v.p, v.s, bulk, s4, sc_step, st);
    if (e != cudaSuccess || bulk == n) return e;
    return smul_part_wave(View{v.p + bulk, v.s}, rest, s4 + 2 * bulk * (size_t)sc_step, sc_step, st);
}

} // namespace ft
