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
// ciphertext, or a_i * B.  k_comb256 computes them, one thread per unit, in
// radix 256 with table rows looked up by the tensor cores (comb256.cuh); for
// short arrays the blocks of a cluster share a unit's rows.  A point's table
// is made by
//   k_comb_bases 256^i * Q by one chain of doublings, a quad of lanes per
//                doubling (quad.cuh)
//   k_comb_t256  the entries
#include <algorithm>
#include <cuda_fp16.h>

#include "internal.h"
#include "points.cuh"
#include "enc_comb.cuh"
#include "comb256.cuh"
#include "comb_roles.cuh"
#include "fe_inv.cuh"
#include "quad.cuh"
#include "umma.cuh"

namespace ft {

// ------------------------------------------------------------ tables

// memory of a point's table: the base points (8 uint4 each), the rows
static constexpr size_t BASES_U4 = (size_t)COMB_ROWS * 8;
static_assert(BASES_U4 * 16 + (size_t)COMB_ROWS * COMB_ROW_BYTES == COMB_TABLE_BYTES, "table size");

static uint4 *bases_of(CombTable t) { return (uint4 *)t.mem; }
static uint8_t *rows_of(CombTable t) { return t.mem + BASES_U4 * 16; }

// One warp: Q doubled 248 times, kept every 8 bits.  A chain of dependent
// doublings is all latency; with four lanes on each a doubling takes a
// squaring and a multiplication in sequence instead of seven.
__global__ void __launch_bounds__(32) k_comb_bases(uint4 *out, const uint4 *q, size_t qs)
{
    __shared__ uint4 trade[4 * 32];
    QuadX x(trade, 32);
    const int l = threadIdx.x & 3, plane = l == 0 ? 6 : l == 3 ? 0 : 2 * l;
    fe v;
    quad_ld(v, q, qs, 0, 1, l);
#pragma unroll 1
    for (int bit = 0;; ++bit) {
        if (threadIdx.x < 4 && bit % 8 == 0) {
            out[bit + plane] = u4_lo(v);
            out[bit + plane + 1] = u4_hi(v);
        }
        if (bit == 8 * (COMB_ROWS - 1)) break;
        __syncwarp();
        quad_dbl(v, x);
        quad_p3(v, x);
    }
}

// k * P as a halved affine entry (comb256.cuh), k < 2^bits public
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
    fe zi, x, y, xy;
    fe_inv(zi, acc.Z);
    fe_mul(x, acc.X, zi);
    fe_mul(y, acc.Y, zi);
    fe_mul(xy, x, y);
    fe_mul(t.xy2d, xy, fe_d());
    fe_mul(x, x, fe_half());
    fe_mul(y, y, fe_half());
    fe_add(t.yplusx, y, x);
    fe_sub(t.yminusx, y, x);
    fe_canon(t.yplusx, t.yplusx);
    fe_canon(t.yminusx, t.yminusx);
    fe_canon(t.xy2d, t.xy2d);
}

__global__ void __launch_bounds__(64) k_comb_t256(uint8_t *out, const uint4 *bases)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int row = t / COMB_K, k = t % COMB_K;
    if (row >= COMB_ROWS) return;
    ge_precomp p;
    comb_entry(p, bases + 8 * row, k + 1, 8);
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

cudaError_t comb_table(CombTable t, View q, cudaStream_t st)
{
    k_comb_bases<<<1, 32, 0, st>>>(bases_of(t), q.p, q.s);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_comb_t256<<<COMB_ROWS * COMB_K / 64, 64, 0, st>>>(rows_of(t), bases_of(t));
    return cudaGetLastError();
}

// ------------------------------------------------------------ units

// What a launch computes: for each half h in [h0, h1), dst[h][i] (+)= the sum
// of the rows of scalar i over table tr[h] (`scalar` set) and of mrows[h]
// rows of m[i] over tm.
struct CombJob {
    uint4 *dst[2]; // (the two-element arrays are read with pick: an index would copy them to local memory)
    size_t s[2];
    const uint8_t *tr[2]; // tables' rows
    const uint8_t *tm;
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
// its one-hot rows (COMB_K / 2 columns, then 8 for the 16 constant entries).
// Shared memory is padded so that no block's tensor-memory allocation waits for
// another's: one block per SM, or two of G = 1, which take half the columns
// each.
template <int G>
struct CombSmem {
    static constexpr int NT = 128 * G;
    static constexpr uint32_t A = COMB_N, PER_WG = COMB_N + COMB_K / 2 + 8, COLS = G == 1 ? 256 : 512;
    static_assert(G * PER_WG <= COLS, "tensor memory");
    static constexpr size_t B = 0, MAGIC = COMB_BUFS * (size_t)COMB_ROW_BYTES,
                            DIG = MAGIC + 2 * COMB_CHUNK, X = DIG + (size_t)8 * NT * 4;
    static constexpr size_t USED = X + (G == 1 ? 2 * (size_t)8 * NT * 16 : 0); // X: points from the cluster's others
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
// issuing for all, on whose scheduler the computing warps fell behind; 5.53
// with four; 5.45 with the 2^23 that makes integers of the f32 in the product;
// 5.22 with comb_add.  (What is added to the multiplications is not hidden by
// them: about a cycle an instruction.  The one-hot rows written by the issuing
// warps instead: 5.69 against 5.45.)
// SPLIT (G = 1): the blocks of a cluster (2, 4 or 8) take a part of a tile's
// rows each, then add their points up in pairs, through the shared memory of
// the lower block of each pair.
template <int G, bool ACC, bool SPLIT>
__global__ void __launch_bounds__(128 * (G + 1), SPLIT ? 2 : 1) k_comb256(CombJob j, int *fault)
{
    using S = CombSmem<G>;
    extern __shared__ __align__(128) uint8_t sm[];
    __shared__ uint64_t full[COMB_BUFS], empty[COMB_BUFS], done[G], ready[G];
    __shared__ uint32_t s_taddr;
    const int tid = threadIdx.x, wg = tid >> 7, warp = tid >> 5;
    const int nr = j.sc ? COMB_ROWS : 0;
    const unsigned per_half = (unsigned)((j.n + S::NT - 1) / S::NT), tiles = per_half * (j.h1 - j.h0);
    const unsigned parts = SPLIT ? cluster_size() : 1u, part = SPLIT ? cluster_rank() : 0u;
    const unsigned tile0 = blockIdx.x / parts, hop = gridDim.x / parts;
    // this block's rows [r0, r1) of a tile of half h
    auto span = [&](int h, int &r0, int &r1) {
        const unsigned rows = nr + CombJob::pick(j.mrows, h);
        r0 = (int)(rows * part / parts);
        r1 = (int)(rows * (part + 1) / parts);
    };
    if (warp == 0) tmem_alloc(&s_taddr, S::COLS);
    if (tid == 0) {
#pragma unroll
        for (int b = 0; b < (int)COMB_BUFS; ++b) {
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
    if (tid < COMB_N) { // the 16 entries after the row's, the same for every row
        uint4 *m = (uint4 *)(sm + S::MAGIC) + tid;
        const uint32_t id = tid < 72 ? comb_part(comb_identity(tid / 24 * 8 + (tid & 7)), tid / 8 % 3) : 0u;
        m[0] = make_uint4(comb_magic(tid), __half_as_ushort(__uint2half_rn(id)), 0u, 0u);
        m[COMB_N] = make_uint4(0u, 0u, 0u, 0u);
    }
    fence_async_smem();
    tmem_sync_threads();
    if (SPLIT) cluster_sync(); // every block of it runs

    ge_p3 h;
    if (wg == G) { // one thread each: warp 3 the loads, warp g the products of warpgroup g
        const int role = warp - 4 * G;
        if ((tid & 31) == 0 && (role < G || role == 3)) {
            unsigned steps = 0;
#pragma unroll 1
            for (unsigned tile = tile0; tile < tiles; tile += hop) {
                int r0, r1;
                span(j.h1 - 1 - (int)(tile / per_half), r0, r1);
                steps += r1 - r0;
            }
            auto wait_full = [&](unsigned b, unsigned parity) { return mbar_wait<COMB_SLEEP>(&full[b], parity); };
            bool ok;
            if (role == 3) {
                unsigned tile = tile0;
                int half = j.h1 - 1 - (int)(tile / per_half), t, end;
                span(half, t, end);
                ok = comb_load(
                    steps, wait_full,
                    [&](unsigned b, unsigned parity) { return mbar_wait<COMB_SLEEP>(&empty[b], parity); },
                    [&](unsigned b) {
                        if (t == end) {
                            tile += hop;
                            half = j.h1 - 1 - (int)(tile / per_half);
                            span(half, t, end);
                        }
                        const uint8_t *src = t < nr ? CombJob::pick(j.tr, half) + (size_t)(nr - 1 - t) * COMB_ROW_BYTES
                                                    : j.tm + (size_t)(t - nr) * COMB_ROW_BYTES;
                        ++t;
                        mbar_expect(&full[b], COMB_ROW_BYTES);
                        bulk_load(sm + S::B + b * COMB_ROW_BYTES, src, COMB_ROW_BYTES, &full[b]);
                    });
            } else {
                const uint32_t dt = s_taddr + S::PER_WG * role;
                ok = comb_issue(
                    steps, wait_full, [&](unsigned parity) { return mbar_wait<COMB_SLEEP>(&ready[role], parity); },
                    [&](unsigned parity) { return mbar_wait<COMB_SLEEP>(&done[role], parity); },
                    [&](unsigned b) {
                        tmem_fence_after();
                        const uint64_t bd = umma_desc(smem_addr(sm + S::B + b * COMB_ROW_BYTES), COMB_CHUNK, 128);
                        umma_f16_ta(dt, dt + S::A + COMB_K / 2, umma_desc(smem_addr(sm + S::MAGIC), COMB_CHUNK, 128),
                                    COMB_IDESC, false);
#pragma unroll
                        for (int k = 0; k < COMB_K / 16; ++k)
                            umma_f16_ta(dt, dt + S::A + 8u * k, bd + k * (2 * COMB_CHUNK >> 4), COMB_IDESC, true);
                        umma_commit(&done[role]);
                        umma_commit(&empty[b]);
                    });
            }
            if (!ok) *(volatile int *)fault = 1;
        }
        __syncwarp();
    } else {
        uint32_t *dig = (uint32_t *)(sm + S::DIG) + tid;
        const uint32_t my_tmem = tmem_warp_addr(s_taddr + S::PER_WG * wg, warp, 0u);
        {
            const uint32_t w[8] = {COMB_MAGIC_A, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
            tmem_st8(my_tmem + S::A + COMB_K / 2, w); // what the rows multiply those entries by
        }
        unsigned q = 0; // steps so far
        bool bad = false;
#pragma unroll 1
        for (unsigned tile = tile0; tile < tiles && !bad; tile += hop) {
            const int half = j.h1 - 1 - (int)(tile / per_half);
            const size_t i = (size_t)(tile % per_half) * S::NT + tid;
            const bool live = i < j.n;
            const int mr = CombJob::pick(j.mrows, half), rows = nr + mr;
            int r0, r1;
            span(half, r0, r1);
            ge_precomp e;
            int d = 0;
            // step t adds row t; the step before r0 only looks up row r0
#pragma unroll 1
            for (int t = r0 - 1; t < r1; ++t) {
                if (t >= r0) {
                    bad = __any_sync(0xffffffffu, !mbar_wait(&done[wg], q & 1));
                    if (bad) break;
                    tmem_fence_after();
                    ++q;
                    fe *const f[3] = {&e.yplusx, &e.yminusx, &e.xy2d};
#pragma unroll
                    for (int g = 0; g < 3; ++g) {
                        uint32_t p[24];
                        tmem_ld24(my_tmem + 24 * g, p);
#pragma unroll
                        for (int k = 0; k < 8; ++k) f[g]->v[k] = comb_word(p[k], p[8 + k], p[16 + k]);
                    }
                    comb_signed(e, d);
                }
                const int nt = t + 1;
                if (nt < r1) { // digit nt and its one-hot row in A
                    if (nt == r0 && nt < nr) {
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
                    if (nt == nr || (nt == r0 && nt > nr)) {
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
                    const uint32_t zh = 0x63ffu; // 1023.5, x for the digit 0; 0 in the high half, which x is not
                    const __half2 zero = __heq2(x, *(const __half2 *)&zh);
                    tmem_st1(my_tmem + S::A + COMB_K / 2 + 1, *(const uint32_t *)&zero);
                    tmem_wait_st();
                    tmem_fence_before();
                    __syncwarp();
                    if ((tid & 31) == 0) mbar_arrive(&ready[wg]);
                }
                if (t == r0) {
                    comb_first(h, e);
                } else if (t > r0) {
                    comb_add(h, e);
                }
            }
            if (!SPLIT && live && !bad) comb_put<ACC>(CombJob::pick(j.dst, half), CombJob::pick(j.s, half), i, h);
        }
        if (bad) *(volatile int *)fault = 1;
    }
    if (SPLIT) {
        __syncwarp();
        uint4 *x = (uint4 *)(sm + S::X) + tid; // two buffers in turn of [word][thread]
#pragma unroll 1
        for (unsigned to = parts / 2; to > 0; to >>= 1, x += x < (uint4 *)(sm + S::X) + 8 * S::NT ? 8 * S::NT : -8 * S::NT) {
            if (wg < G && part >= to && part < 2 * to) {
                const fe *const c[4] = {&h.X, &h.Y, &h.Z, &h.T};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    cluster_store(x + 2 * k * S::NT, part - to, u4_lo(*c[k]));
                    cluster_store(x + (2 * k + 1) * S::NT, part - to, u4_hi(*c[k]));
                }
            }
            cluster_sync();
            if (wg < G && part < to) {
                ge_p3 y;
                ld_p3(y, x, S::NT, 0);
                ge_addto(h, y);
            }
        }
        const int half = j.h1 - 1 - (int)(tile0 / per_half);
        const size_t i = (size_t)(tile0 % per_half) * S::NT + tid;
        if (wg < G && part == 0 && i < j.n) comb_put<ACC>(CombJob::pick(j.dst, half), CombJob::pick(j.s, half), i, h);
    }
    tmem_sync_threads();
    if (warp == 0) tmem_free(s_taddr, S::COLS);
}

// ------------------------------------------------------------ launchers

template <int G, bool ACC, bool SPLIT>
static cudaError_t launch_256(const CombJob &j, size_t tiles, unsigned parts, int *fault, cudaStream_t st)
{
    using S = CombSmem<G>;
    static SmemAttr attr;
    cudaError_t e = ensure_smem_attr(attr, (const void *)k_comb256<G, ACC, SPLIT>, S::BYTES);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = parts;
    cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)(SPLIT ? tiles * parts : std::min<size_t>(tiles, sm_count())));
    c.blockDim = dim3(S::NT + 128);
    c.dynamicSmemBytes = S::BYTES;
    c.stream = st;
    c.attrs = &cluster;
    c.numAttrs = SPLIT ? 1 : 0;
    return cudaLaunchKernelEx(&c, k_comb256<G, ACC, SPLIT>, j, fault);
}

// a job whose scalars' tables are tr0 and tr1 (halves 0 and 1), m's is tm, and
// whose m has mbits bits (0: none) in the halves of mask mhalf
template <bool ACC>
static cudaError_t comb_launch(CombJob j, const CombTable *tr0, const CombTable *tr1, const CombTable *tm,
                               unsigned mbits, unsigned mhalf, int *fault, cudaStream_t st)
{
    if (j.n == 0) return cudaSuccess;
    const CombTable *tr[2] = {tr0, tr1};
    for (int h = 0; h < 2; ++h) {
        j.tr[h] = tr[h] ? rows_of(*tr[h]) : nullptr;
        j.mrows[h] = mbits && (mhalf >> h & 1) ? comb_rows(mbits) : 0;
    }
    j.tm = rows_of(*tm);
    const size_t halves = j.h1 - j.h0, sm = sm_count();
    auto tiles = [&](int g) { return (j.n + 128 * g - 1) / (128 * g) * halves; };
    // Up to a tile per SM, a tile's rows are split over as many blocks as give
    // two per SM at most.
    const size_t t = tiles(1);
    if (t <= sm) {
        const unsigned parts = 8 * t <= 2 * sm ? 8 : 4 * t <= 2 * sm ? 4 : 2;
        return launch_256<1, ACC, true>(j, t, parts, fault, st);
    }
    // Beyond, a round of a tile of 256 units per SM takes about 103 us, of 384
    // about 146: 384 for many rounds, else what takes the least (38,912
    // ciphertexts: 229 us in two of 256, 306 in two of 384; 1,048,576: 5.21 ms
    // in 36 of 384, 54 of 256 would take 5.56).
    const size_t r2 = (tiles(2) + sm - 1) / sm, r3 = (tiles(3) + sm - 1) / sm;
    if (r2 * 103 < r3 * 146) return launch_256<2, ACC, false>(j, tiles(2), 1, fault, st);
    return launch_256<3, ACC, false>(j, tiles(3), 1, fault, st);
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
