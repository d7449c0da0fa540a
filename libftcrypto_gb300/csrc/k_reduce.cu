// k_reduce.cu — reductions whose combine operator is point addition.
//
//   reduce   sum of n points (ft_array_reduce; k_ft_array_reduce,
//            ftcrypto.cu:1414-1471).  Many points: every thread accumulates a
//            grid-strided subset with one addition (9 multiplications) per
//            point; then, or for few points at once, four lanes per point
//            (quad.cuh), a block per SM, and one block.  ~1 addition per
//            input point (the reference's tree does the same count but with
//            most threads idle at the upper levels and 160-byte AoS loads).
//   scan     inclusive / exclusive prefix (ft_array_scan / ft_array_prescan;
//            ftcrypto.cu:1474-1586): per-thread sums of K consecutive points,
//            block-wide scans of those sums, a scan of the blocks' totals that
//            shifts them, then each thread rescans its K points from its
//            prefix.  ~2 + 10/K additions per point, no waits between blocks.
//            Short arrays are scanned by blocks directly.  Correct
//            for every length (the reference's kernel indexes its tile sums
//            wrongly above 256 x grid points, ftcrypto.cu:1512).
//   segsum   out[s] = sum of src[e] (or src[perm[e]]) for e in
//            [off[s], off[s+1]): each thread sums SEG_K = 32 consecutive points
//            segment by segment, writes the segments that begin and end inside
//            it and records the parts of the segments crossing its edges; a
//            second kernel joins those parts (k_seg_walk / k_seg_join).
//            ~1 + 1/32 additions per point.  It serves ft_reduce_isum
//            (ftcrypto.cu:1113-1217, accumulating into res) and the CSR
//            segmented-sum extension.
//   keys_to_csr  counting sort of ft_reduce_isum's keys on the device
//            (replaces the reference's host std::sort, ftcrypto.cu:1170).
#include <algorithm>

#include <cmath>
#include <mutex>

#include "internal.h"
#include "points.cuh"
#include "quad.cuh"

namespace ft {

// ------------------------------------------------------------ sums

// acc += v, a quad of lanes per point (quad.cuh)
FT_DEV void quad_addto(fe &acc, const fe &v, QuadX &x)
{
    fe c;
    quad_cached(c, v, x);
    quad_add(acc, c, x);
    quad_p3(acc, x);
}

// Sums of few points, each block's in out[block]: what a launch costs is its
// chain of additions, and with four lanes on each an addition takes 3
// multiplications in sequence instead of 9.
template <int NT>
__global__ void __launch_bounds__(NT) k_reduce_quad(const uint4 *p, size_t s, size_t n, uint4 *out, size_t os)
{
    static_assert(NT % 32 == 0 && NT <= 256, "a warp of quads holds the warps' sums");
    __shared__ uint4 trade[4 * NT], part[NT / 32 * 8];
    QuadX x(trade, NT);
    const int l = threadIdx.x & 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t q = threadIdx.x >> 2, stride = (size_t)gridDim.x * (NT / 4);
    fe acc, v;
    size_t base = (size_t)blockIdx.x * (NT / 4);
    quad_ld(acc, p, s, base + q, n, l);
#pragma unroll 1
    for (base += stride; base < n; base += stride) {
        quad_ld(v, p, s, base + q, n, l);
        quad_addto(acc, v, x);
    }
    auto tree = [&](int o) {
#pragma unroll 1
        for (; o >= 4; o >>= 1) {
#pragma unroll
            for (int k = 0; k < 8; ++k) v.v[k] = __shfl_down_sync(0xffffffffu, acc.v[k], o);
            quad_addto(acc, v, x);
        }
    };
    tree(16);
    if (NT > 32) {
        if (lane < 4) {
            part[8 * warp + l] = u4_lo(acc);
            part[8 * warp + 4 + l] = u4_hi(acc);
        }
        __syncthreads();
        if (warp > 0) return;
        if (lane < NT / 8) {
            fe_from_u4(acc, part[8 * (lane >> 2) + l], part[8 * (lane >> 2) + 4 + l]);
        } else {
            fe_0(acc);
            acc.v[0] = l == 1 || l == 2;
        }
        tree(NT / 16);
    }
    if (threadIdx.x < 4) quad_st(out, os, blockIdx.x, acc, l);
}

// Sums of many points, 32 per block.  A minimum of one block per SM in the
// launch bounds lets ptxas take 124 registers instead of 106 (still four
// blocks of 128 threads per SM): the sum of 16,777,216 points 1.539 -> 1.483
// ms.  Two points per step (158 registers, three blocks per SM) measured 1.546
// ms, with 128 registers forced (spills) 1.559 ms.  The next point arrives in
// shared memory while this one is added (8,388,608 points 749 -> 725 us).  A block leaves its last
// 32 sums to k_reduce_quad: summing them here took 16 warps of an SM five
// more additions each, 29 us of a launch of 8,388,608 points.
static constexpr int RED_NT = 128, RED_OUT = 32;

__global__ void __launch_bounds__(RED_NT, 1) k_reduce(const uint4 *p, size_t s, size_t n, uint4 *out, size_t os)
{
    __shared__ uint4 sm[2 * 8 * RED_NT]; // the next point and this one
    ge_p3 acc, x;
    const size_t stride = (size_t)gridDim.x * RED_NT;
    size_t i = (size_t)blockIdx.x * RED_NT + threadIdx.x;
    uint4 *slot = sm + threadIdx.x, *next = slot + 8 * RED_NT;
    if (i < n) ld_p3(acc, p, s, i);
    else ge_p3_0(acc);
    ge_tighten(acc);
    size_t base = (size_t)blockIdx.x * RED_NT + stride;
    i += stride;
    if (i < n) point_fetch(slot, RED_NT, p, s, i);
    points_sent();
    // block-uniform steps with a barrier each: the warps stay on the same
    // stretch of the addition's code and share the instruction caches
    // (instruction-fetch stalls were 0.75 per issue): 2.09 -> 2.01 ms for
    // 16,777,216 points
#pragma unroll 1
    for (; base < n; base += stride) {
        __syncthreads();
        const bool here = i < n;
        i += stride;
        if (i < n) point_fetch(next, RED_NT, p, s, i);
        points_sent();
        points_wait<1>();
        if (here) {
            ld_p3(x, slot, RED_NT, 0);
            ge_accumulate(acc, x);
        }
        uint4 *const t = slot;
        slot = next;
        next = t;
    }
    points_wait<0>();
    // 128 sums to 64 to 32; the adding warps are on other schedulers in
    // other blocks
    const unsigned w = ((threadIdx.x >> 5) + blockIdx.x) & 3u, t = 32 * w + (threadIdx.x & 31);
#pragma unroll 1
    for (unsigned half = 64; half >= RED_OUT; half >>= 1) {
        __syncthreads();
        if (t >= half && t < 2 * half) st_p3(sm, 64, t - half, acc);
        __syncthreads();
        if (t < half) {
            ld_p3(x, sm, 64, t);
            ge_accumulate(acc, x);
        }
    }
    if (t < RED_OUT) st_p3(out, os, (size_t)blockIdx.x * RED_OUT + t, acc);
}

// ------------------------------------------------------------ scan

// inclusive scan over the first `width` lanes of the warp (a power of two);
// returns the lane's inclusive sum in acc
FT_DEV void warp_scan_incl(ge_p3 &acc, int width = 32)
{
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int o = 1; o < width; o <<= 1) {
        ge_p3 up, sum;
        shfl_up_p3(up, acc, o);
        sum = up;
        ge_addto(sum, acc);
        if (lane >= o) acc = sum;
    }
}

// The scan kernels take up to two arrays of one length (the two halves of a
// ciphertext array, ftx_ct_scan): blockIdx.y selects the array, so both are
// scanned by the same launches and share the latency-bound lower levels.
struct ScanSet {
    uint4 *p[2];
    size_t s[2];
    // array blockIdx.y, chosen by selects (indexing the parameter array with
    // blockIdx.y would copy it to local memory)
    FT_DEV uint4 *ptr() const { return blockIdx.y ? p[1] : p[0]; }
    FT_DEV size_t stride() const { return blockIdx.y ? s[1] : s[0]; }
};

// Blocks of 128 threads per SM that the scan's passes and the segmented sum's
// walk are compiled for (__launch_bounds__ minimum): three for the scan (168
// registers; four, 128 registers, spill: 2.68 against 1.95 ms for 2 x 4,194,304
// points), four for the walk (128 registers: 1.73 against 1.81 ms at three).
static constexpr int SCAN_BLOCKS = 3;
#ifndef FT_SEG_WALK_MINB
#define FT_SEG_WALK_MINB 4
#endif


#ifndef FT_WAVE_FIT
#define FT_WAVE_FIT 1
#endif

// Blocks of `fn` (block size `nt`, no dynamic shared memory) resident on the
// whole GPU at once, from the occupancy calculator; cached by the caller.
static int resident_blocks(const void *fn, int nt)
{
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, nt, 0) != cudaSuccess || per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    return per_sm * sm_count();
}

// Of the points-per-thread candidates ks[0..nk) (ascending), the one whose
// launch of ceil(ceil(n / k) / 128) * m blocks of 128 threads fills its last
// wave of `resident` blocks best (waves / ceil(waves) highest; ties go to
// the smaller k).  One walk per thread, so a last wave at 74% leaves a
// quarter of the GPU idle for 1/7 of the launch (16,777,216 points at 32 per
// thread in four 128-thread blocks per SM: 6.74 waves; at 36: 5.99).
static int wave_fit_k(size_t n, int m, const int *ks, int nk, const int *resident)
{
    int best = ks[0];
    double best_eff = -1.0;
    for (int i = 0; i < nk; ++i) {
        const size_t blocks = ((n + ks[i] - 1) / ks[i] + 127) / 128 * (size_t)m;
        const double waves = (double)blocks / resident[i];
        const double eff = waves / std::ceil(waves);
        if (eff > best_eff + 1e-9) {
            best_eff = eff;
            best = ks[i];
        }
    }
    return best;
}

// (An L1 prefetch of the thread's next pair of points before each step
// measured slower: the two-half scan of 4,194,304 points 1.93 -> 1.96 ms,
// the segmented sum of 16,777,216 points 1.66 -> 1.77 ms.  Copying the
// rescan's next pair into shared memory with cp.async while the current
// pair is added — no registers held for it, 64 KB per block, still three
// blocks per SM — measured the same for both halves, 1.046 -> 1.062 ms for
// one array and 1.014 -> 1.064 ms for the prescan.)
// per-thread sums of K consecutive points: ts[t] = sum of p[tK .. tK+K).  The
// thread loads its points two at a time: the two 16-byte words of a pair fill
// one 32-byte sector of each plane, which is then read from DRAM once (one
// point at a time, the sector's second half can be evicted before the next
// step and read again: 1.29x the algorithmic bytes in the sums, 1.39x in the
// rescan, measured), and memory is waited for once per two points.  A step is
// one addition, with a barrier, so that the block's warps share the
// instruction caches: 2 x 4,194,304 points 1.80 -> 1.71 ms against two
// additions a step without.  (Fetching the next pair into shared memory
// meanwhile measured 1.85 ms, a warp fetching its threads' next four points
// together, coalesced, 1.79: the additions bound the passes, not the loads.)
__global__ void __launch_bounds__(128, SCAN_BLOCKS) k_scan_sums(ScanSet in, size_t n, int K, ScanSet ts)
{
    const uint4 *p = in.ptr();
    const size_t s = in.stride();
    const size_t t = (size_t)blockIdx.x * 128 + threadIdx.x, e0 = t * K;
    ge_p3 acc, x, y;
    if (e0 < n) ld_p3(acc, p, s, e0);
    if (e0 + 1 < n) ld_p3(y, p, s, e0 + 1);
    ge_tighten(acc);
#pragma unroll 1
    for (int k = 1; k < K; ++k) {
        __syncthreads();
        const size_t e = e0 + k;
        if (e >= n) continue;
        if (k & 1) {
            x = y;
        } else {
            ld_p3(x, p, s, e);
            if (e + 1 < n) ld_p3(y, p, s, e + 1);
        }
        ge_accumulate(acc, x);
    }
    if (e0 < n) st_p3(ts.ptr(), ts.stride(), t, acc);
}

// rescan each thread's K points starting from its exclusive prefix ts[t];
// `exclusive` a template parameter: as a run-time flag the inclusive form
// needed 210 registers (two blocks per SM) instead of 168 (three)
template <int exclusive>
__global__ void __launch_bounds__(128, SCAN_BLOCKS) k_scan_apply(ScanSet io, size_t n, int K, ScanSet ts)
{
    uint4 *p = io.ptr();
    const size_t s = io.stride();
    const size_t t = (size_t)blockIdx.x * 128 + threadIdx.x, e0 = t * K;
    ge_p3 pre, x, y;
    if (e0 < n) ld_p3(pre, ts.ptr(), ts.stride(), t);
    ge_tighten(pre);
#pragma unroll 1
    for (int k = 0; k < K; ++k) {
        __syncthreads();
        const size_t e = e0 + k;
        if (e >= n) continue;
        if (k & 1) {
            x = y;
        } else {
            ld_p3(x, p, s, e);
            if (e + 1 < n) ld_p3(y, p, s, e + 1);
        }
        if (exclusive) st_p3(p, s, e, pre);
        ge_accumulate(pre, x);
        if (!exclusive) st_p3(p, s, e, pre);
    }
}

// each block scans its 128 P points in place (P consecutive points per
// thread; the inclusive form only for P = 1) and writes their total
__global__ void __launch_bounds__(128, SCAN_BLOCKS) k_scan_block(ScanSet io, size_t n, int P, int inclusive, ScanSet tot)
{
    __shared__ uint4 sm[4 * 8];
    uint4 *p = io.ptr();
    const size_t s = io.stride();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t e0 = ((size_t)blockIdx.x * 128 + threadIdx.x) * P;
    ge_p3 incl, v;
    ge_p3_0(incl);
    if (e0 < n) ld_p3(incl, p, s, e0);
#pragma unroll 1
    for (int k = 1; k < P && e0 + k < n; ++k) {
        ld_p3(v, p, s, e0 + k);
        ge_addto(incl, v);
    }
    __syncwarp();
    warp_scan_incl(incl);
    if (lane == 31) sm_st_p3(sm, warp, incl);
    __syncthreads();
    if (warp == 0) {
        if (lane < 4) sm_ld_p3(v, sm, lane);
        else ge_p3_0(v);
        warp_scan_incl(v, 4);
        if (lane == 3) st_p3(tot.ptr(), tot.stride(), blockIdx.x, v);
        ge_p3 ex;
        shfl_up_p3(ex, v, 1);
        if (lane == 0) ge_p3_0(ex);
        if (lane < 4) sm_st_p3(sm, lane, ex);
    }
    if (!inclusive) {
        shfl_up_p3(v, incl, 1);
        if (lane == 0) ge_p3_0(v);
        incl = v;
    }
    __syncthreads();
    sm_ld_p3(v, sm, warp);
    ge_addto(incl, v); // the block's points before this thread's (and its own)
#pragma unroll 1
    for (int k = 0; k < P; ++k) {
        const size_t e = e0 + k;
        if (e >= n) break;
        if (k + 1 < P) ld_p3(v, p, s, e);
        st_p3(p, s, e, incl);
        if (k + 1 < P) ge_addto(incl, v);
    }
}

// p[e] += the exclusive prefix of e's block of `per` points (a multiple of
// 128); the first block's is the identity
__global__ void __launch_bounds__(128) k_scan_shift(ScanSet io, size_t n, int per, ScanSet tot)
{
    uint4 *p = io.ptr();
    const size_t s = io.stride();
    const size_t e = (size_t)per + (size_t)blockIdx.x * 128 + threadIdx.x;
    if (e >= n) return;
    ge_p3 x, y;
    ld_p3(y, tot.ptr(), tot.stride(), e / per);
    ld_p3(x, p, s, e);
    ge_addto(x, y);
    st_p3(p, s, e, x);
}

// One block per array scans n <= NT / 4 * kpt points in place, a quad of lanes
// per addition (quad.cuh): sums of kpt consecutive points per quad, a scan of
// those over the block, then the rescan.  One block is all latency: 218 points
// took 52 us with a thread per addition.
template <int NT>
__global__ void __launch_bounds__(NT) k_scan_small(ScanSet io, size_t n, int kpt, int exclusive)
{
    __shared__ uint4 trade[4 * NT], vals[4 * NT];
    QuadX x(trade, NT);
    uint4 *p = io.ptr();
    const size_t s = io.stride();
    const int l = threadIdx.x & 3, q = threadIdx.x >> 2;
    const size_t e0 = (size_t)q * kpt;
    fe acc, v;
    quad_ld(acc, p, s, e0, n, l);
#pragma unroll 1
    for (int k = 1; k < kpt; ++k) {
        quad_ld(v, p, s, e0 + k, n, l);
        quad_addto(acc, v, x);
    }
    // inclusive scan over the quads, then the one before; two buffers in turn
    int flip = 0;
#pragma unroll 1
    for (int o = 1;; o <<= 1) {
        const int back = o < NT / 4 ? o : 1;
        uint4 *w = vals + flip + threadIdx.x;
        w[0] = u4_lo(acc);
        w[NT] = u4_hi(acc);
        __syncthreads();
        if (q >= back) {
            fe_from_u4(v, w[-4 * back], w[NT - 4 * back]);
        } else {
            fe_0(v);
            v.v[0] = l == 1 || l == 2;
        }
        __syncwarp();
        if (o >= NT / 4) break;
        quad_addto(acc, v, x);
        flip ^= 2 * NT;
    }
    acc = v;
#pragma unroll 1
    for (int k = 0; k < kpt; ++k) {
        const size_t e = e0 + k;
        quad_ld(v, p, s, e, n, l);
        if (exclusive && e < n) quad_st(p, s, e, acc, l);
        __syncwarp();
        quad_addto(acc, v, x);
        if (!exclusive && e < n) quad_st(p, s, e, acc, l);
    }
}

static const int SMALL_NT = 256;

size_t scan_scratch_bytes(size_t n, int m) { return (size_t)m * scan_scratch_points(n) * 128 + 256; }

// Points per thread of the sums and the rescan; 1: the block scans take the
// points themselves.  Two warps per scheduler hold m * n = 256 points per SM;
// beyond, K is the least that makes the launches whole waves of SCAN_BLOCKS
// blocks per SM, up to 40 points a thread (2 x 4,194,304 points: 1.82 ms at 16,
// 1.71 at 36, 1.79 at 72; 2 x 1,000,000: 0.53, 0.50, 0.67).
static int scan_points(size_t n, int m)
{
    const size_t sm = (size_t)sm_count(), wave = 128 * SCAN_BLOCKS * sm;
    if (n * m <= 256 * sm) return 1;
    size_t waves = (n * m + 40 * wave - 1) / (40 * wave);
    size_t k = (n * m + waves * wave - 1) / (waves * wave);
    k = (std::max(k, scan_level_k(n)) + 1) / 2 * 2;
    return (int)k;
}

// Sums of K points per thread, block-wide scans of those sums, a scan of the
// blocks' totals (one block up to SCAN_SMALL_MAX, else this routine), which
// shifts the sums' scans, then the rescan from each thread's prefix: about
// 2 + 10 / K additions per point, no waits between blocks.  The chain of
// additions between the sums and the rescan, which no launch fills the GPU
// with, is 11 + 13 of a quad + 1 (1,000,000 ciphertexts: 70 us; 156 us as three
// levels of 4 points per thread and a last block).  m arrays (1 or 2) of n points each go
// through the same launches; scratch holds m x scan_scratch_points(n) points.
cudaError_t scan_set(const View *v, int m, size_t n, int exclusive, void *scratch, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (m < 1 || m > 2) return cudaErrorInvalidValue;
    ScanSet io{};
    for (int i = 0; i < m; ++i) {
        io.p[i] = v[i].p;
        io.s[i] = v[i].s;
    }
    if (n <= SCAN_SMALL_MAX) {
        const int kpt = (int)((n + SMALL_NT / 4 - 1) / (SMALL_NT / 4));
        k_scan_small<SMALL_NT><<<dim3(1, m), SMALL_NT, 0, st>>>(io, n, kpt, exclusive);
        return cudaGetLastError();
    }
    uint4 *next = (uint4 *)scratch;
    auto take = [&](ScanSet &set, View *views, size_t count) {
        for (int i = 0; i < m; ++i) {
            views[i] = View{next, count};
            set.p[i] = next;
            set.s[i] = count;
            next += FT_PLANES * count;
        }
    };
    const int K = scan_points(n, m);
    const size_t nt = (n + K - 1) / K;
    ScanSet sums = io, totals{};
    View vs[2], vt[2];
    const dim3 grid((unsigned)((nt + 127) / 128), m);
    cudaError_t e;
    if (K > 1) {
        take(sums, vs, nt);
        k_scan_sums<<<grid, 128, 0, st>>>(io, n, K, sums);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    // points per thread of the block scans: P (2 + 7 / P additions a point, in
    // a chain of 2 P + 7): more of them where the chain is not what counts
    const size_t warps = 128 * (size_t)sm_count(); // threads, one warp per scheduler
    const int P = K == 1 || nt * m <= warps ? 1 : nt * m <= 4 * warps ? 2 : 4, per = 128 * P;
    const size_t nb = (nt + per - 1) / per;
    take(totals, vt, nb);
    k_scan_block<<<dim3((unsigned)nb, m), 128, 0, st>>>(sums, nt, P, K == 1 && !exclusive, totals);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (nb > 1) {
        if ((e = scan_set(vt, m, nb, 1, next, st)) != cudaSuccess) return e;
        k_scan_shift<<<dim3((unsigned)((nt - per + 127) / 128), m), 128, 0, st>>>(sums, nt, per, totals);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (K == 1) return cudaSuccess;
    if (exclusive) k_scan_apply<1><<<grid, 128, 0, st>>>(io, n, K, sums);
    else k_scan_apply<0><<<grid, 128, 0, st>>>(io, n, K, sums);
    return cudaGetLastError();
}

cudaError_t scan(View v, size_t n, int exclusive, void *scratch, cudaStream_t st)
{
    return scan_set(&v, 1, n, exclusive, scratch, st);
}

// ------------------------------------------------------------ reduce launcher

// blocks of the first pass over many points: one wave, every block resident
static size_t reduce_blocks()
{
    static std::once_flag once;
    static size_t resident;
    std::call_once(once, [] { resident = (size_t)resident_blocks((const void *)k_reduce, RED_NT); });
    return resident;
}

// Blocks of a quad pass: 32 quads each, up to one per SM.  One block alone
// (of 64 quads) takes up to 5 points a quad, which saves a launch: a sum of 33
// to 128 points 17.3 to 18.7 us against 25.4 with two (25.5 before there were
// quads), of 257 23.1, of 384 25.0 against 25.4, of 512 28.0 against 25.6.
static size_t quad_blocks(size_t n)
{
    return n <= 5 * 64 ? 1 : std::min<size_t>((n + 31) / 32, (size_t)sm_count());
}

size_t reduce_scratch_bytes(size_t n)
{
    (void)n;
    return (reduce_blocks() * RED_OUT + (size_t)sm_count()) * 128 + 256;
}

// A point per thread of the first pass and more: that pass, whose sums
// (19,456 with 152 SMs) are then the points; the sums of a block per SM by
// quads; one block's.  8,388,608 points 781 -> 749 us, 1,000 points 37 -> 18.
cudaError_t reduce(View out, View src, size_t n, void *scratch, cudaStream_t st)
{
    if (n == 0) return set_zero(out, 1, st);
    cudaError_t e;
    const size_t g = reduce_blocks();
    uint4 *next = (uint4 *)scratch;
    if (n > g * RED_NT) {
        const View part{next, g * RED_OUT};
        next += FT_PLANES * g * RED_OUT;
        k_reduce<<<(unsigned)g, RED_NT, 0, st>>>(src.p, src.s, n, part.p, part.s);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        src = part;
        n = g * RED_OUT;
    }
    const size_t q = quad_blocks(n);
    if (q > 1) {
        const View part{next, q};
        k_reduce_quad<128><<<(unsigned)q, 128, 0, st>>>(src.p, src.s, n, part.p, part.s);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        src = part;
        n = q;
    }
    k_reduce_quad<256><<<1, 256, 0, st>>>(src.p, src.s, n, out.p, out.s);
    return cudaGetLastError();
}

// ------------------------------------------------------------ segmented sum

FT_DEV int upper_bound_i32(const int32_t *a, int lo, int hi, long long x) // first i in [lo,hi) with a[i] > x
{
    while (lo < hi) {
        int mid = lo + ((hi - lo) >> 1);
        if ((long long)a[mid] <= x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

FT_DEV void seg_write(uint4 *op, size_t os, int sg, const ge_p3 &v, int accumulate)
{
    if (accumulate) {
        ge_p3 r;
        ld_p3(r, op, os, sg);
        ge_addto(r, v);
        st_p3(op, os, sg, r);
    } else {
        st_p3(op, os, sg, v);
    }
}

// record flags of a thread in the segmented sum
#define SEG_HEAD 1u   // H[t] holds the part of a segment that began before the thread
#define SEG_CLOSE 2u  // ... and that segment ends inside the thread (or at its last point)
#define SEG_TAIL 4u   // L[t] holds the start of segment lseg[t], which continues past the thread

// The arrays of one or two segmented sums over the same offsets (the two
// halves of a ciphertext array): output, source and scratch of sum y in
// slot y, chosen by blockIdx.y (a select, not an index, so the struct stays
// in parameter space).
struct SegSet {
    uint4 *op[2];
    size_t os[2];
    const uint4 *sp[2];
    size_t ss[2];
    uint4 *H[2];
    uint4 *Lp[2];
    uint32_t *flags[2];
    int32_t *lseg[2];
    template <class T>
    FT_DEV static T pick(const T (&a)[2]) { return blockIdx.y ? a[1] : a[0]; }
};

// Pass 1: thread t sums its K consecutive points segment by segment.  A
// segment that begins and ends inside the thread is written at once; the
// parts of segments crossing the thread's edges go to H / L.
// four blocks per SM (128 registers, a few spills to L1) rather than two at
// 202 registers: 2.58 against 2.68 ms for 16,777,216 points (measured)
template <int K>
__global__ void __launch_bounds__(128, FT_SEG_WALK_MINB) k_seg_walk(SegSet set, const int32_t *off, int nseg,
                                                                    long long nsrc, const int32_t *perm, int accumulate,
                                                                    size_t hs)
{
    uint4 *op = SegSet::pick(set.op);
    const size_t os = SegSet::pick(set.os);
    const uint4 *sp = SegSet::pick(set.sp);
    const size_t ss = SegSet::pick(set.ss);
    uint4 *H = SegSet::pick(set.H);
    uint4 *Lp = SegSet::pick(set.Lp);
    uint32_t *flags = SegSet::pick(set.flags);
    int32_t *lseg = SegSet::pick(set.lseg);
    const long long nt = (nsrc + K - 1) / K;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; // the launch covers nt
    const bool live = t < nt;
    {
        const long long e0 = live ? t * K : 0;
        const long long e1 = live ? min(e0 + K, nsrc) : 0;
        int sg = live ? upper_bound_i32(off, 0, nseg + 1, e0) - 1 : 0; // segment holding e0 (skips empty ones)
        bool open_before = live && (long long)off[sg] < e0;
        uint32_t fl = 0;
        ge_p3 acc;
        ge_p3_0(acc);
        // every thread of the block takes the K steps, with a barrier each:
        // the warps stay on the same stretch of code and share the
        // instruction caches (instruction-fetch stalls were 1.45 per issue):
        // 2.32 -> 2.21 ms for 16,777,216 points in 1,048,576 segments
#pragma unroll 1
        for (int k = 0; k < K; ++k) {
            __syncthreads();
            const long long e = e0 + k;
            if (e >= e1) continue;
            while ((long long)off[sg + 1] <= e) ++sg;
            ge_p3 x;
            ld_p3(x, sp, ss, perm ? (size_t)perm[e] : (size_t)e);
            if ((long long)off[sg] == e || e == e0) acc = x;
            else ge_addto(acc, x);
            if ((long long)off[sg + 1] == e + 1) { // last point of segment sg
                if (open_before) {
                    st_p3(H, hs, t, acc);
                    fl |= SEG_HEAD | SEG_CLOSE;
                    open_before = false;
                } else {
                    seg_write(op, os, sg, acc, accumulate);
                }
            }
        }
        if (live && (long long)off[sg + 1] > e1) { // the last segment continues past the thread
            if (open_before) {
                st_p3(H, hs, t, acc);
                fl |= SEG_HEAD;
            } else {
                st_p3(Lp, hs, t, acc);
                fl |= SEG_TAIL;
                lseg[t] = sg;
            }
        }
        if (live) flags[t] = fl;
    }
}

// Pass 2: a segment started in thread t and continuing past it totals
// L[t] + H[t+1] + ... + H[u], u the first later thread whose head closes it.
__global__ void __launch_bounds__(128) k_seg_join(SegSet set, size_t hs, size_t nt, int accumulate)
{
    uint4 *op = SegSet::pick(set.op);
    const size_t os = SegSet::pick(set.os);
    const uint4 *H = SegSet::pick(set.H);
    const uint4 *Lp = SegSet::pick(set.Lp);
    const uint32_t *flags = SegSet::pick(set.flags);
    const int32_t *lseg = SegSet::pick(set.lseg);
    FT_GRID_LOOP(t, nt)
    {
        if (!(flags[t] & SEG_TAIL)) continue;
        ge_p3 sum;
        ld_p3(sum, Lp, hs, t);
#pragma unroll 1
        for (size_t u = t + 1; u < nt; ++u) {
            ge_p3 h;
            ld_p3(h, H, hs, u);
            ge_addto(sum, h);
            if (flags[u] & SEG_CLOSE) break;
        }
        seg_write(op, os, lseg[t], sum, accumulate);
    }
}

__global__ void __launch_bounds__(256) k_seg_empty(SegSet set, const int32_t *off, size_t nseg)
{
    uint4 *op = SegSet::pick(set.op);
    const size_t os = SegSet::pick(set.os);
    FT_GRID_LOOP(sg, nseg)
    {
        if (off[sg] == off[sg + 1]) {
            ge_p3 z;
            ge_p3_0(z);
            st_p3(op, os, sg, z);
        }
    }
}

// points per thread of the walk: 32 rather than 16 halves the threads' fixed
// costs (the binary search for the first segment, the edge partials, the
// join): 2.59 -> 2.32 ms for 16,777,216 points in 1,048,576 segments (64 and
// 128 measure the same as 32; 8 is 3.84 ms)
static const int SEG_K = 32;

size_t segsum_scratch_bytes(size_t nsrc, int m)
{
    size_t nt = (nsrc + SEG_K - 1) / SEG_K;
    const size_t one = ((2 * nt * 128 + 2 * nt * 4 + 1024) + 255) / 256 * 256; // each sum's part 256-byte aligned
    return (size_t)m * one;
}

// out[s] (+)= sum of src[perm ? perm[e] : e], e in [off[s], off[s+1]):
// ~1 + 1/SEG_K additions per point, two kernels, no waits between blocks.
// A segment spanning m threads costs m sequential additions in pass 2
// (m ~ length / 32; 1-2 for the benchmark's mean lengths 8-32).  m (1 or
// 2) sums over the same offsets and source length go through the same
// launches (grid dimension y); scratch holds m x segsum_scratch_bytes(nsrc).
cudaError_t segsum_set(const View *out, const View *src, int m, const int32_t *off, size_t nseg, size_t nsrc,
                       const int32_t *perm, int accumulate, void *scratch, cudaStream_t st)
{
    if (nseg == 0) return cudaSuccess;
    if (m < 1 || m > 2) return cudaErrorInvalidValue;
    SegSet set{};
    for (int i = 0; i < m; ++i) {
        set.op[i] = out[i].p;
        set.os[i] = out[i].s;
        set.sp[i] = src[i].p;
        set.ss[i] = src[i].s;
    }
    cudaError_t e;
    if (!accumulate) {
        const dim3 g((unsigned)std::min<size_t>((nseg + 255) / 256, 65535), m);
        k_seg_empty<<<g, 256, 0, st>>>(set, off, nseg);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (nsrc == 0) return cudaSuccess;
    // points per thread: 32, 36 or 40, whichever fills the walk's last wave
    // best (at least 32, so the scratch sized for SEG_K suffices)
    static const int ks[3] = {32, 36, 40};
    static int res[3];
    static std::once_flag once;
    std::call_once(once, [] {
        res[0] = resident_blocks((const void *)k_seg_walk<32>, 128);
        res[1] = resident_blocks((const void *)k_seg_walk<36>, 128);
        res[2] = resident_blocks((const void *)k_seg_walk<40>, 128);
    });
    const int K = FT_WAVE_FIT ? wave_fit_k(nsrc, m, ks, 3, res) : SEG_K;
    const size_t nt = (nsrc + K - 1) / K;
    for (int i = 0; i < m; ++i) {
        uint8_t *base = (uint8_t *)scratch + (size_t)i * segsum_scratch_bytes(nsrc, 1);
        set.H[i] = (uint4 *)base;
        set.Lp[i] = set.H[i] + FT_PLANES * nt;
        set.flags[i] = (uint32_t *)(set.Lp[i] + FT_PLANES * nt);
        set.lseg[i] = (int32_t *)(set.flags[i] + nt);
    }
    const dim3 grid((unsigned)((nt + 127) / 128), m);
    switch (K) {
    case 36: k_seg_walk<36><<<grid, 128, 0, st>>>(set, off, (int)nseg, (long long)nsrc, perm, accumulate, nt); break;
    case 40: k_seg_walk<40><<<grid, 128, 0, st>>>(set, off, (int)nseg, (long long)nsrc, perm, accumulate, nt); break;
    default: k_seg_walk<SEG_K><<<grid, 128, 0, st>>>(set, off, (int)nseg, (long long)nsrc, perm, accumulate, nt); break;
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_seg_join<<<grid, 128, 0, st>>>(set, nt, nt, accumulate);
    return cudaGetLastError();
}

cudaError_t segsum(View out, const int32_t *off, size_t nseg, View src, size_t nsrc, const int32_t *perm,
                   int accumulate, void *scratch, cudaStream_t st)
{
    return segsum_set(&out, &src, 1, off, nseg, nsrc, perm, accumulate, scratch, st);
}

// ------------------------------------------------------------ long segments

// dst[e] = src[perm[e]]
__global__ void __launch_bounds__(256) k_gather_i32(uint4 *d, size_t ds, const uint4 *s, size_t ss,
                                                    const int32_t *perm, size_t n)
{
    FT_GRID_LOOP(e, n)
    {
        const size_t j = (size_t)perm[e];
#pragma unroll
        for (int k = 0; k < FT_PLANES; ++k) d[k * ds + e] = s[k * ss + j];
    }
}

// out[s] (+)= P[off[s+1] - 1] - P[off[s] - 1], P the inclusive prefix sums
// (P[-1] the identity): each segment as a difference of two prefixes
__global__ void __launch_bounds__(128) k_seg_diff(uint4 *op, size_t os, const int32_t *off, size_t nseg,
                                                  const uint4 *P, size_t ps, int accumulate)
{
    FT_GRID_LOOP(sg, nseg)
    {
        const int32_t a = off[sg], b = off[sg + 1];
        ge_p3 v;
        if (a == b) {
            if (accumulate) continue;
            ge_p3_0(v);
        } else {
            ld_p3(v, P, ps, (size_t)b - 1);
            if (a > 0) {
                ge_p3 q;
                ld_p3(q, P, ps, (size_t)a - 1);
                ge_subfrom(v, q);
            }
        }
        seg_write(op, os, (int)sg, v, accumulate);
    }
}

// the largest off[s+1] - off[s] into *d_max (which the caller zeroes)
__global__ void __launch_bounds__(256) k_seg_maxlen(const int32_t *off, size_t nseg, int32_t *d_max)
{
    int32_t m = 0;
    FT_GRID_LOOP(sg, nseg) m = max(m, off[sg + 1] - off[sg]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(d_max, m);
}

cudaError_t segment_maxlen(const int32_t *d_off, size_t nseg, int32_t *d_max, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(d_max, 0, sizeof(int32_t), st);
    if (e != cudaSuccess || nseg == 0) return e;
    k_seg_maxlen<<<(unsigned)std::min<size_t>((nseg + 255) / 256, 1024), 256, 0, st>>>(d_off, nseg, d_max);
    return cudaGetLastError();
}

bool segsum_prefers_prefix(size_t nsrc, size_t max_len)
{
    // the walk's join adds the parts of a segment spanning m threads one
    // after another (m = length / 32, ~7 us each); the prefix path costs
    // about one scan more than the walk, whatever the lengths
    return max_len > std::max<size_t>(2048, nsrc / 1024);
}

size_t segsum_prefix_scratch_bytes(size_t nsrc)
{
    return ((nsrc * 128 + 255) / 256) * 256 + scan_scratch_bytes(nsrc);
}

// the same sums through one inclusive scan of the (gathered) points and a
// difference of two prefixes per segment: ~2 additions per point, and no
// chain of additions longer than the scan's whatever the segment lengths
cudaError_t segsum_prefix(View out, const int32_t *off, size_t nseg, View src, size_t nsrc, const int32_t *perm,
                          int accumulate, void *scratch, cudaStream_t st)
{
    if (nseg == 0) return cudaSuccess;
    View P{(uint4 *)scratch, nsrc};
    void *scan_tmp = (uint8_t *)scratch + ((nsrc * 128 + 255) / 256) * 256;
    cudaError_t e = cudaSuccess;
    if (nsrc) {
        if (perm) {
            k_gather_i32<<<(unsigned)std::min<size_t>((nsrc + 255) / 256, (size_t)sm_count() * 16), 256, 0, st>>>(
                P.p, P.s, src.p, src.s, perm, nsrc);
            e = cudaGetLastError();
        } else {
            e = copy_points(P, src, nsrc, st);
        }
        if (e == cudaSuccess) e = scan(P, nsrc, 0, scan_tmp, st);
        if (e != cudaSuccess) return e;
    }
    k_seg_diff<<<(unsigned)std::min<size_t>((nseg + 127) / 128, (size_t)sm_count() * 32), 128, 0, st>>>(
        out.p, out.s, off, nseg, P.p, P.s, accumulate);
    return cudaGetLastError();
}

// ------------------------------------------------------------ counting sort

// Lanes of a warp holding the same key add their count with one atomic (the
// lowest of them): repeated keys, up to all keys equal, do not serialise on
// one counter.
__global__ void k_key_hist(const uint64_t *keys, size_t n, size_t nkeys, int32_t *cnt, long long *bad)
{
    FT_GRID_LOOP(i, n)
    {
        const uint64_t k = keys[i];
        const unsigned peers = __match_any_sync(__activemask(), k);
        if (k >= nkeys) atomicMax(bad, (long long)i);
        else if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&cnt[k], __popc(peers));
    }
}

// places index i of key k at cur[k] + its rank among the warp's lanes of key k
__global__ void k_key_place(const uint64_t *keys, size_t n, size_t nkeys, int32_t *cur, int32_t *perm)
{
    FT_GRID_LOOP(i, n)
    {
        const uint64_t k = keys[i];
        const unsigned peers = __match_any_sync(__activemask(), k);
        const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
        int32_t base = 0;
        if (k < nkeys && lane == leader) base = atomicAdd(&cur[k], __popc(peers));
        base = __shfl_sync(peers, base, leader);
        if (k < nkeys) perm[base + __popc(peers & ((1u << lane) - 1u))] = (int32_t)i;
    }
}

// exclusive scan of int32 in blocks of 1024 x 4; block totals scanned recursively
__global__ void __launch_bounds__(1024) k_iscan_block(int32_t *a, size_t n, int32_t *bsum)
{
    __shared__ int32_t ws[32];
    const size_t base = (size_t)blockIdx.x * 4096 + threadIdx.x * 4;
    int32_t v[4], t = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = base + k < n ? a[base + k] : 0;
        t += v[k];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t incl = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) ws[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int32_t w = ws[lane];
        int32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int32_t u = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += u;
        }
        ws[lane] = wi - w;
        if (lane == 31 && bsum) bsum[blockIdx.x] = wi;
    }
    __syncthreads();
    int32_t run = ws[warp] + incl - t;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (base + k < n) a[base + k] = run;
        run += v[k];
    }
}

__global__ void k_iscan_add(int32_t *a, size_t n, const int32_t *bsum)
{
    FT_GRID_LOOP(i, n) a[i] += bsum[i / 4096];
}

static cudaError_t iscan_excl(int32_t *a, size_t n, int32_t *tmp, cudaStream_t st)
{
    size_t nb = (n + 4095) / 4096;
    k_iscan_block<<<(unsigned)nb, 1024, 0, st>>>(a, n, nb > 1 ? tmp : nullptr);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || nb == 1) return e;
    e = iscan_excl(tmp, nb, tmp + nb, st);
    if (e != cudaSuccess) return e;
    k_iscan_add<<<(unsigned)((n + 255) / 256 < 65535 ? (n + 255) / 256 : 65535), 256, 0, st>>>(a, n, tmp);
    return cudaGetLastError();
}

size_t isum_scratch_bytes(size_t n, size_t nkeys)
{
    (void)n;
    size_t t = 0, m = nkeys + 1;
    while (m > 1) {
        m = (m + 4095) / 4096;
        t += m;
    }
    return (nkeys + 1 + t + 64) * sizeof(int32_t);
}

cudaError_t keys_to_csr(int32_t *off, int32_t *perm, const uint64_t *keys, size_t n, size_t nkeys,
                        long long *bad, void *scratch, cudaStream_t st)
{
    int32_t *cur = (int32_t *)scratch;
    int32_t *tmp = cur + nkeys + 1;
    cudaError_t e = cudaMemsetAsync(off, 0, (nkeys + 1) * sizeof(int32_t), st);
    if (e != cudaSuccess) return e;
    unsigned g = (unsigned)((n + 255) / 256 < 65535 ? ((n + 255) / 256 ? (n + 255) / 256 : 1) : 65535);
    k_key_hist<<<g, 256, 0, st>>>(keys, n, nkeys, off, bad);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = iscan_excl(off, nkeys + 1, tmp, st)) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(cur, off, (nkeys + 1) * sizeof(int32_t), cudaMemcpyDeviceToDevice, st)) != cudaSuccess)
        return e;
    k_key_place<<<g, 256, 0, st>>>(keys, n, nkeys, cur, perm);
    return cudaGetLastError();
}

} // namespace ft
