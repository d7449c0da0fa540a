// k_encrypt.cu — the fixed-base kernels: encryption, re-randomisation and
// multiples of B, with the tables they read.
//
//   encryption   c1 = r*B, c2 = m*B + r*PK (ftx_encrypt; the reference
//                composes it from ft_array_from_scalars, ft_array_init_point +
//                ft_mul and ft_array_from_small_scalars + ft_add);
//                re-randomisation adds r*B and r*PK in place (ACC)
//   base         a_i * B for 32-byte scalars or uint64 values
//                (ft_array_from_scalars, ft_array_from_small_scalars,
//                ft_array_init_scalar; the reference uses its variable-base
//                ladder here, ftcrypto.cu:895-913)
//
// Both are lists of units, a unit being one output point: half 0 or 1 of a
// ciphertext, or a_i * B.  Two kernels compute them:
//   k_comb256    radix 256, one thread per unit, table rows looked up by the
//                tensor cores (comb256.cuh); for lengths that fill the GPU
//   k_comb_lanes radix 32 (enc_comb.cuh), 8 to 32 lanes per unit that share
//                its rows and add their sums in a tree; for short arrays
// and these make a point's tables:
//   k_comb_bases 32^i * Q and 256^i * Q by one chain of doublings, a quad of
//                lanes per doubling (quad.cuh)
//   k_comb_t32, k_comb_t256   the entries of the two combs
#include <algorithm>
#include <cuda_fp16.h>

#include "internal.h"
#include "points.cuh"
#include "enc_comb.cuh"
#include "comb256.cuh"
#include "fe_inv.cuh"
#include "quad.cuh"
#include "umma.cuh"

namespace ft {

// ------------------------------------------------------------ tables

// memory of a point's tables: 52 + 32 base points (8 uint4 each), the
// radix-32 table (word w of entry e of row r at (6 e + w) * 64 + r), the
// radix-256 table (COMB_ROW_BYTES a row)
static constexpr int T32_ROWS = 64, N_BASES = ENC_ROWS + COMB_ROWS;
static constexpr size_t BASES_U4 = (size_t)N_BASES * 8, T32_U4 = (size_t)ENC_ENTRIES * 6 * T32_ROWS;
static_assert(BASES_U4 * 16 + T32_U4 * 16 + (size_t)COMB_ROWS * COMB_ROW_BYTES == COMB_TABLE_BYTES, "table size");

static uint4 *bases_of(CombTable t) { return (uint4 *)t.mem; }
static uint4 *t32_of(CombTable t) { return (uint4 *)t.mem + BASES_U4; }
static uint8_t *t256_of(CombTable t) { return t.mem + (BASES_U4 + T32_U4) * 16; }

// One warp: Q doubled 255 times, kept every 5 and every 8 bits.  A chain of
// dependent doublings is all latency; with four lanes on each a doubling
// takes a squaring and a multiplication in sequence instead of seven.
__global__ void __launch_bounds__(32) k_comb_bases(uint4 *out, const uint4 *q, size_t qs)
{
    __shared__ uint4 trade[4 * 32];
    QuadX x(trade, 32);
    const int l = threadIdx.x & 3;
    const bool w = threadIdx.x < 4;
    fe v;
    quad_ld(v, q, qs, 0, 1, l);
    const int plane = l == 0 ? 6 : l == 3 ? 0 : 2 * l;
#pragma unroll 1
    for (int bit = 0;; ++bit) {
        if (w && bit % 5 == 0) {
            out[(bit / 5) * 8 + plane] = u4_lo(v);
            out[(bit / 5) * 8 + plane + 1] = u4_hi(v);
        }
        if (w && bit % 8 == 0) {
            out[(ENC_ROWS + bit / 8) * 8 + plane] = u4_lo(v);
            out[(ENC_ROWS + bit / 8) * 8 + plane + 1] = u4_hi(v);
        }
        if (bit == 5 * (ENC_ROWS - 1)) break;
        __syncwarp();
        quad_dbl(v, x);
        quad_p3(v, x);
    }
}

// k * P as an affine table entry, k < 2^bits public
FT_DEV void comb_entry(ge_precomp &t, const uint4 *base, int k, int bits)
{
    ge_p3 P, acc;
    sm_ld_p3(P, base, 0);
    ge_cached c;
    ge_p3_to_cached(c, P);
    ge_p3_0(acc);
#pragma unroll 1
    for (int b = bits - 1; b >= 0; --b) {
        ge_p1p1 r;
        ge_p3_dbl(r, acc);
        ge_p1p1_to_p3(acc, r);
        if (k >> b & 1) {
            ge_add(r, acc, c);
            ge_p1p1_to_p3(acc, r);
        }
    }
    fe zi, x, y;
    fe_inv(zi, acc.Z);
    fe_mul(x, acc.X, zi);
    fe_mul(y, acc.Y, zi);
    fe_add(t.yplusx, y, x);
    fe_sub(t.yminusx, y, x);
    fe_mul(x, x, y);
    fe_mul(t.xy2d, x, fe_d2());
    fe_canon(t.yplusx, t.yplusx);
    fe_canon(t.yminusx, t.yminusx);
    fe_canon(t.xy2d, t.xy2d);
}

__global__ void __launch_bounds__(64) k_comb_t32(uint4 *out, const uint4 *bases)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = t % T32_ROWS, e = t / T32_ROWS;
    if (row >= ENC_ROWS || e >= ENC_ENTRIES) return;
    ge_precomp p;
    comb_entry(p, bases + 8 * row, e + 1, 5);
    uint4 *o = out + (size_t)e * 6 * T32_ROWS + row;
    o[0 * T32_ROWS] = u4_lo(p.yplusx);
    o[1 * T32_ROWS] = u4_hi(p.yplusx);
    o[2 * T32_ROWS] = u4_lo(p.yminusx);
    o[3 * T32_ROWS] = u4_hi(p.yminusx);
    o[4 * T32_ROWS] = u4_lo(p.xy2d);
    o[5 * T32_ROWS] = u4_hi(p.xy2d);
}

__global__ void __launch_bounds__(64) k_comb_t256(uint8_t *out, const uint4 *bases)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = t / COMB_K, k = t % COMB_K;
    if (row >= COMB_ROWS) return;
    ge_precomp p;
    comb_entry(p, bases + 8 * (ENC_ROWS + row), k + 1, 8);
    uint8_t *o = out + (size_t)row * COMB_ROW_BYTES;
    auto put = [&](int f, const fe &x) {
#pragma unroll
        for (int w = 0; w < 8; ++w)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                *(__half *)(o + comb_offset(24 * f + 8 * c + w, k)) = __uint2half_rn(comb_part(x.v[w], c));
    };
    put(0, p.yplusx);
    put(1, p.yminusx);
    put(2, p.xy2d);
#pragma unroll
    for (int n = 72; n < COMB_N; ++n) *(__half *)(o + comb_offset(n, k)) = __uint2half_rn(0u);
}

cudaError_t comb_bases(CombTable t, View q, cudaStream_t st)
{
    k_comb_bases<<<1, 32, 0, st>>>(bases_of(t), q.p, q.s);
    return cudaGetLastError();
}

cudaError_t comb_t32(CombTable t, cudaStream_t st)
{
    k_comb_t32<<<T32_ROWS * ENC_ENTRIES / 64, 64, 0, st>>>(t32_of(t), bases_of(t));
    return cudaGetLastError();
}

cudaError_t comb_t256(CombTable t, cudaStream_t st)
{
    k_comb_t256<<<COMB_ROWS * COMB_K / 64, 64, 0, st>>>(t256_of(t), bases_of(t));
    return cudaGetLastError();
}

// ------------------------------------------------------------ units

// What a launch computes: for each half h in [h0, h1), dst[h][i] (+)= the sum
// of the rows of scalar i over table tr[h] (`scalar` set) and of mrows[h]
// rows of m[i] over tm.  Table pointers are those of the launch's radix.
struct CombJob {
    uint4 *dst[2]; // (the two-element arrays are read with pick: an index would copy them to local memory)
    size_t s[2];
    const void *tr[2];
    const void *tm;
    const uint4 *sc; // 32-byte scalars, sc_step apart (0: one for all); null: none
    int sc_step;
    const uint64_t *m;
    int mrows[2];
    size_t n;
    int h0, h1;
    template <class T>
    FT_DEV static T pick(const T (&a)[2], int h) { return h ? a[1] : a[0]; }
};

// dst[i] = h, or dst[i] += h with ACC
template <bool ACC>
FT_DEV void comb_put(uint4 *dst, size_t s, size_t i, const ge_p3 &h)
{
    if (ACC) {
        ge_p3 x;
        ld_p3(x, dst, s, i);
        ge_addto(x, h);
        st_p3(dst, s, i, x);
    } else {
        st_p3(dst, s, i, h);
    }
}

// the scalar of unit i as the reference effectively uses it
FT_DEV void comb_scalar(uint32_t a[8], const CombJob &j, size_t i)
{
    const uint4 s0 = j.sc[2 * i * j.sc_step], s1 = j.sc[2 * i * j.sc_step + 1];
    const uint32_t x[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    enc_ref_scalar(a, x);
}

// ------------------------------------------------------------ radix 256

// ns between the issuing warps' polls (50: 5.64 ms for 1,048,576 ciphertexts, 500: 5.53)
static constexpr int COMB_SLEEP = 400;
static constexpr uint32_t COMB_IDESC = umma_idesc_f16(128, COMB_N);

// A block of G warpgroups: three table rows and the recoded scalars in shared
// memory; in tensor memory, per warpgroup, its products (COMB_N columns) and
// its one-hot rows (COMB_K / 2 columns).  Shared memory is padded so that no
// block's tensor-memory allocation waits for another's: one block per SM, or
// two of G = 1, which take half the columns each.
template <int G>
struct CombSmem {
    static constexpr int NT = 128 * G;
    static constexpr uint32_t A = COMB_N, PER_WG = COMB_N + COMB_K / 2, COLS = G == 1 ? 256 : 512;
    static_assert(G * PER_WG <= COLS, "tensor memory");
    static constexpr size_t B = 0, DIG = 3 * (size_t)COMB_ROW_BYTES, USED = DIG + (size_t)8 * NT * 4;
    static constexpr size_t BYTES = std::max(USED, (size_t)(G == 1 ? 80 : 116) * 1024);
};

// The work list of a block: tiles of 128 G units, those of half h1 - 1 (the
// longer one) first.  Every row of a tile is a step.  The G warpgroups compute:
// a warp waits for its warpgroup's product of the step (`done`), reads the
// selected entries, writes the next step's one-hot rows (`ready`) and adds the
// entries.  A warpgroup more issues everything asynchronous, from one thread
// each of four warps (on the four schedulers): warp g warpgroup g's next
// product once its four warps are ready, which runs beside their additions;
// warp 3 the loads of table rows, into three buffers shared by the warpgroups,
// a buffer when every warpgroup's product of it is done (`empty`).
// Bound by the multiply-add pipe of the additions (2,430 cycles a row and
// warp alone).  1,048,576 ciphertexts: 6.72 ms with a barrier of the block per
// step and one of its threads issuing; 6.25 to 6.50 with the last warp of a
// warpgroup to be ready issuing (it takes that warp 1,100 cycles, in which its
// own row and so its warpgroup's next product wait); 5.55 with one warp
// issuing for all, on whose scheduler the computing warps fell behind.
template <int G, bool ACC>
__global__ void __launch_bounds__(128 * (G + 1), 1) k_comb256(CombJob j, int *fault)
{
    using S = CombSmem<G>;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ uint64_t full[3], empty[3], done[G], ready[G];
    __shared__ uint32_t s_taddr;
    const int tid = threadIdx.x, wg = tid >> 7, warp = tid >> 5;
    const int nr = j.sc ? COMB_ROWS : 0;
    const unsigned per_half = (unsigned)((j.n + S::NT - 1) / S::NT), tiles = per_half * (j.h1 - j.h0);
    if (warp == 0) tmem_alloc(&s_taddr, S::COLS);
    if (tid == 0) {
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&empty[b], G);
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            mbar_init(&done[g], 1);
            mbar_init(&ready[g], 4);
        }
        mbar_fence_init();
    }
    tmem_sync_threads();

    if (wg == G && warp - 4 * G == 3) { // the loads
        if ((tid & 31) == 0) {
            unsigned tile = blockIdx.x, loads = 0;
            int t = 0;
            bool bad = false;
#pragma unroll 1
            for (unsigned buf = 0, use = 0; tile < tiles && !bad; ++loads) {
                const int h = j.h1 - 1 - (int)(tile / per_half);
                const uint8_t *src = t < nr
                                         ? (const uint8_t *)CombJob::pick(j.tr, h) + (size_t)(nr - 1 - t) * COMB_ROW_BYTES
                                         : (const uint8_t *)j.tm + (size_t)(t - nr) * COMB_ROW_BYTES;
                // the buffer's use before this one
                if (use && !mbar_wait<COMB_SLEEP>(&empty[buf], (use - 1) & 1)) bad = true;
                if (!bad) {
                    mbar_expect(&full[buf], COMB_ROW_BYTES);
                    bulk_load(sm + S::B + buf * COMB_ROW_BYTES, src, COMB_ROW_BYTES, &full[buf]);
                }
                if (++t == nr + CombJob::pick(j.mrows, h)) {
                    t = 0;
                    tile += gridDim.x;
                }
                if (++buf == 3) {
                    buf = 0;
                    ++use;
                }
            }
            // the last copies have landed before the block ends
#pragma unroll 1
            for (unsigned k = loads < 3 ? 0 : loads - 3; k < loads; ++k)
                if (!mbar_wait<COMB_SLEEP>(&full[k % 3], (k / 3) & 1)) bad = true;
            if (bad) *(volatile int *)fault = 1;
        }
        __syncwarp();
    } else if (wg == G) { // the products of warpgroup g
        const int g = warp - 4 * G;
        if (g < G && (tid & 31) == 0) {
            unsigned steps = 0;
#pragma unroll 1
            for (unsigned k = blockIdx.x; k < tiles; k += gridDim.x)
                steps += nr + CombJob::pick(j.mrows, j.h1 - 1 - (int)(k / per_half));
            const uint32_t dt = s_taddr + S::PER_WG * g;
            unsigned buf = 0, use = 0; // the step's buffer, and that buffer's use
#pragma unroll 1
            for (unsigned q = 0; q < steps; ++q) {
                if (!mbar_wait<COMB_SLEEP>(&full[buf], use & 1) || !mbar_wait<COMB_SLEEP>(&ready[g], q & 1)) {
                    *(volatile int *)fault = 1;
                    break;
                }
                tmem_fence_after();
                const uint64_t bd = umma_desc(smem_addr(sm + S::B + buf * COMB_ROW_BYTES), COMB_CHUNK, 128);
#pragma unroll
                for (int k = 0; k < COMB_K / 16; ++k)
                    umma_f16_ta(dt, dt + S::A + 8u * k, bd + k * (2 * COMB_CHUNK >> 4), COMB_IDESC, k != 0);
                umma_commit(&done[g]);
                umma_commit(&empty[buf]);
                if (++buf == 3) {
                    buf = 0;
                    ++use;
                }
            }
        }
        __syncwarp();
    } else {
        uint32_t *dig = (uint32_t *)(sm + S::DIG) + tid;
        const uint32_t my_tmem = tmem_warp_addr(s_taddr + S::PER_WG * wg, warp, 0u);
        unsigned q = 0; // steps so far
        bool bad = false;
#pragma unroll 1
        for (unsigned tile = blockIdx.x; tile < tiles && !bad; tile += gridDim.x) {
            const int half = j.h1 - 1 - (int)(tile / per_half);
            const size_t i = (size_t)(tile % per_half) * S::NT + tid;
            const bool live = i < j.n;
            const int mr = CombJob::pick(j.mrows, half), rows = nr + mr;
            ge_p3 h;
            ge_precomp e;
            int d = 0;
            // step t adds row t; step -1 only looks up row 0
#pragma unroll 1
            for (int t = -1; t < rows; ++t) {
                if (t >= 0) {
                    bad = __any_sync(0xffffffffu, !mbar_wait(&done[wg], q & 1));
                    if (bad) break;
                    tmem_fence_after();
                    ++q;
                    fe *const f[3] = {&e.yplusx, &e.yminusx, &e.xy2d};
#pragma unroll
                    for (int g = 0; g < 3; ++g) {
                        float p[24];
                        tmem_ld24(my_tmem + 24 * g, p);
#pragma unroll
                        for (int k = 0; k < 8; ++k) f[g]->v[k] = comb_word(p[k], p[8 + k], p[16 + k]);
                    }
                    comb_signed(e, d);
                }
                const int nt = t + 1;
                if (nt < rows) { // digit nt and its one-hot row in A
                    if (nt == 0 && nr) {
                        uint32_t a[8], b[8];
                        if (live) {
                            comb_scalar(a, j, i);
                        } else {
#pragma unroll
                            for (int k = 0; k < 8; ++k) a[k] = 0u;
                        }
                        comb_reduce(a);
                        comb_recode(b, a);
#pragma unroll
                        for (int k = 0; k < 8; ++k) dig[k * S::NT] = b[k];
                    }
                    if (nt == nr) {
                        uint32_t b[3];
                        comb_recode_small(b, live && j.m ? j.m[i] : 0, mr);
#pragma unroll
                        for (int k = 0; k < 3; ++k) dig[k * S::NT] = b[k];
                    }
                    const int row = nt < nr ? nr - 1 - nt : nt - nr;
                    d = comb_digit(dig[(row >> 2) * S::NT], row, nt < nr ? nt == 0 : nt == rows - 1);
                    // half2 of 1024 + |d| - 1 twice, compared with 1024 + entry
                    const uint32_t babs = (uint32_t)(d < 0 ? -d : d);
                    const uint32_t xh = (0x6400u + babs - 1u) * 0x10001u;
                    const __half2 x = *(const __half2 *)&xh;
#pragma unroll
                    for (int c = 0; c < COMB_K / 2; c += 8) {
                        uint32_t w[8];
#pragma unroll
                        for (int p = 0; p < 8; ++p) {
                            const uint32_t ch = (0x6400u + 2u * (c + p)) * 0x10001u + 0x10000u;
                            const __half2 eq = __heq2(x, *(const __half2 *)&ch);
                            w[p] = *(const uint32_t *)&eq;
                        }
                        tmem_st8(my_tmem + S::A + c, w);
                    }
                    tmem_wait_st();
                    tmem_fence_before();
                    __syncwarp();
                    if ((tid & 31) == 0) mbar_arrive(&ready[wg]);
                }
                if (t == 0) {
                    comb_first(h, e);
                } else if (t > 0) {
                    ge_p1p1 r;
                    ge_madd(r, h, e);
                    ge_p1p1_to_p3(h, r);
                }
            }
            if (live && !bad) comb_put<ACC>(CombJob::pick(j.dst, half), CombJob::pick(j.s, half), i, h);
        }
        if (bad) *(volatile int *)fault = 1;
    }
    tmem_sync_threads();
    if (warp == 0) tmem_free(s_taddr, S::COLS);
}

// ------------------------------------------------------------ radix 32

// L lanes per unit: lane k of a unit sums its rows k, k + L, ..., then the
// lanes' sums are added in a tree.  The table is read from L1 / L2, a row to
// each lane (consecutive rows are consecutive words); the digits are
// recoded by each lane.
static constexpr int LANES_NT = 64;

template <int L, bool ACC>
__global__ void __launch_bounds__(LANES_NT) k_comb_lanes(CombJob j)
{
    __shared__ uint32_t s_dig[2][10][LANES_NT];
    const size_t u = ((size_t)blockIdx.x * LANES_NT + threadIdx.x) / L;
    const int lane = threadIdx.x % L;
    const size_t units = j.n * (j.h1 - j.h0);
    const bool live = u < units;
    const int half = live ? j.h1 - 1 - (int)(u / j.n) : j.h0;
    const size_t i = live ? u % j.n : 0;
    const int nr = j.sc ? ENC_ROWS : 0, mr = CombJob::pick(j.mrows, half), rows = nr + mr;
    uint32_t c[9];
    if (nr) {
        uint32_t a[8];
        comb_scalar(a, j, i);
        enc_recode(c, a, ENC_ROWS);
#pragma unroll
        for (int k = 0; k < 9; ++k) s_dig[0][k][threadIdx.x] = c[k];
        s_dig[0][9][threadIdx.x] = 0u;
    }
    if (mr) {
        const uint64_t m = j.m ? j.m[i] : 0;
        const uint32_t a[8] = {(uint32_t)m, (uint32_t)(m >> 32), 0u, 0u, 0u, 0u, 0u, 0u};
        enc_recode(c, a, mr);
#pragma unroll
        for (int k = 0; k < 9; ++k) s_dig[1][k][threadIdx.x] = c[k];
        s_dig[1][9][threadIdx.x] = 0u;
    }
    const uint4 *tr = (const uint4 *)CombJob::pick(j.tr, half), *tm = (const uint4 *)j.tm;
    ge_p3 h;
    ge_p3_0(h);
#pragma unroll 1
    for (int t = lane; t < rows; t += L) {
        const bool second = t >= nr;
        const int row = second ? t - nr : t, bit = 5 * row;
        const uint32_t lo = s_dig[second][bit >> 5][threadIdx.x], hi = s_dig[second][(bit >> 5) + 1][threadIdx.x];
        const int d = (int)(__funnelshift_r(lo, hi, bit & 31) & 31u) - 16;
        ge_precomp e;
        enc_select<T32_ROWS>(e, d, (second ? tm : tr) + row);
        if (t == lane) {
            comb_first(h, e);
        } else {
            ge_p1p1 r;
            ge_madd(r, h, e);
            ge_p1p1_to_p3(h, r);
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int o = L / 2; o > 0; o >>= 1) {
        ge_p3 x;
        shfl_down_p3(x, h, o);
        ge_addto(h, x);
    }
    if (live && lane == 0) comb_put<ACC>(CombJob::pick(j.dst, half), CombJob::pick(j.s, half), i, h);
}

// ------------------------------------------------------------ launchers

// Up to 12 units per warp scheduler the radix-32 kernel is faster: 1,824
// ciphertexts (6 units) 68 us, 3,648 (12) 77 us with eight lanes a unit, 108 us
// beyond with four, against 97 us in the radix-256 kernel for any number up to
// 128 units per SM.
bool comb_is_wide(size_t units) { return units > (size_t)sm_count() * 48; }

// Warpgroups per block: a round of 128 G units per SM takes about 90, 120 and
// 158 us for G = 1, 2 and 3, so G = 3 for many rounds, else the one whose
// rounds take the least (38,912 ciphertexts: 244 us with 2, 330 with 3).
static int comb_warpgroups(size_t units)
{
    const size_t per_sm = (units + sm_count() - 1) / sm_count();
    const size_t us[4] = {0, 90, 120, 158};
    int best = 3;
    for (int g = 2; g >= 1; --g)
        if ((per_sm + 128 * g - 1) / (128 * g) * us[g] < (per_sm + 128 * best - 1) / (128 * best) * us[best]) best = g;
    return best;
}

template <int G, bool ACC>
static cudaError_t launch_256(const CombJob &j, int *fault, cudaStream_t st)
{
    using S = CombSmem<G>;
    static SmemAttr attr;
    cudaError_t e = ensure_smem_attr(attr, (const void *)k_comb256<G, ACC>, S::BYTES);
    if (e != cudaSuccess) return e;
    const size_t tiles = (j.n + S::NT - 1) / S::NT * (j.h1 - j.h0), cap = (size_t)sm_count();
    k_comb256<G, ACC><<<(unsigned)std::min(tiles, cap), S::NT + 128, S::BYTES, st>>>(j, fault);
    return cudaGetLastError();
}

template <int L, bool ACC>
static cudaError_t launch_lanes(const CombJob &j, cudaStream_t st)
{
    const size_t threads = j.n * (j.h1 - j.h0) * L;
    k_comb_lanes<L, ACC><<<(unsigned)((threads + LANES_NT - 1) / LANES_NT), LANES_NT, 0, st>>>(j);
    return cudaGetLastError();
}

// a job whose tables are those of tr0, tr1 (halves 0 and 1) and tm, and whose
// m has mbits bits (0: none) in the halves of mask mhalf
template <bool ACC>
static cudaError_t comb_launch(CombJob j, const CombTable *tr0, const CombTable *tr1, const CombTable *tm,
                               unsigned mbits, unsigned mhalf, int *fault, cudaStream_t st)
{
    if (j.n == 0) return cudaSuccess;
    const size_t units = j.n * (j.h1 - j.h0);
    const bool wide = comb_is_wide(units);
    const CombTable *tr[2] = {tr0, tr1};
    for (int h = 0; h < 2; ++h) {
        j.tr[h] = tr[h] ? (wide ? (const void *)t256_of(*tr[h]) : (const void *)t32_of(*tr[h])) : nullptr;
        j.mrows[h] = mbits && (mhalf >> h & 1) ? (wide ? comb_rows(mbits) : enc_digits(mbits)) : 0;
    }
    j.tm = wide ? (const void *)t256_of(*tm) : (const void *)t32_of(*tm);
    if (wide) {
        switch (comb_warpgroups(units)) {
        case 1: return launch_256<1, ACC>(j, fault, st);
        case 2: return launch_256<2, ACC>(j, fault, st);
        default: return launch_256<3, ACC>(j, fault, st);
        }
    }
    const size_t warps = (size_t)sm_count() * 4;
    if (units <= 2 * warps) return launch_lanes<32, ACC>(j, st);
    if (units <= 4 * warps) return launch_lanes<16, ACC>(j, st);
    return launch_lanes<8, ACC>(j, st);
}

template <bool ACC>
static cudaError_t ciphertexts(View c1, View c2, size_t n, const uint8_t *r, const uint64_t *m, unsigned bits,
                               const CombTable &tb, const CombTable &tp, int *fault, cudaStream_t st)
{
    CombJob j{};
    j.dst[0] = c1.p;
    j.s[0] = c1.s;
    j.dst[1] = c2.p;
    j.s[1] = c2.s;
    j.sc = (const uint4 *)r;
    j.sc_step = 1;
    j.m = m;
    j.n = n;
    j.h1 = 2;
    if (c1.p != c2.p) return comb_launch<ACC>(j, &tb, &tp, &tb, bits, 2u, fault, st);
    // one array for both halves: the second after the first
    j.h1 = 1;
    cudaError_t e = comb_launch<ACC>(j, &tb, &tp, &tb, bits, 2u, fault, st);
    if (e != cudaSuccess) return e;
    j.h0 = 1;
    j.h1 = 2;
    return comb_launch<ACC>(j, &tb, &tp, &tb, bits, 2u, fault, st);
}

size_t encrypt_pass() { return (size_t)sm_count() * 384 / 2; }

cudaError_t encrypt(View c1, View c2, size_t n, const uint8_t *r, const uint64_t *m, unsigned bits,
                    const CombTable &tb, const CombTable &tp, int *fault, cudaStream_t st)
{
    return ciphertexts<false>(c1, c2, n, r, m, bits, tb, tp, fault, st);
}

cudaError_t rerandomise(View c1, View c2, size_t n, const uint8_t *r, const CombTable &tb, const CombTable &tp,
                        int *fault, cudaStream_t st)
{
    return ciphertexts<true>(c1, c2, n, r, nullptr, 0, tb, tp, fault, st);
}

cudaError_t smul_base(View v, size_t n, const uint8_t *sc, int sc_step, const CombTable &tb, int *fault, cudaStream_t st)
{
    CombJob j{};
    j.dst[0] = v.p;
    j.s[0] = v.s;
    j.sc = (const uint4 *)sc;
    j.sc_step = sc_step;
    j.n = n;
    j.h1 = 1;
    return comb_launch<false>(j, &tb, nullptr, &tb, 0, 0u, fault, st);
}

cudaError_t smul_base_small(View v, size_t n, const uint64_t *small, const CombTable &tb, int *fault, cudaStream_t st)
{
    CombJob j{};
    j.dst[0] = v.p;
    j.s[0] = v.s;
    j.m = small;
    j.n = n;
    j.h1 = 1;
    return comb_launch<false>(j, &tb, nullptr, &tb, 64, 1u, fault, st);
}

} // namespace ft
