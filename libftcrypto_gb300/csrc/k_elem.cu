// k_elem.cu — element-wise kernels: group ops, comparisons, gather/scatter and
// the wire formats (folded 32 B, affine 64 B, reference-limb 160 B, packed 128 B).
//
// Kernel <-> reference kernel (ftcrypto.cu):
//   k_set_zero        k_ft_array_set_zero (252)       k_broadcast   k_ft_array_set_point (275)
//   k_add (sub=0/1)   k_ft_add (1089) / k_ft_sub (1220) k_neg        k_ft_neg (1244)
//   k_index           k_ft_index (1262)                k_equal       k_ft_equal (1281)
//   k_mux             k_ft_array_mux (1014)
//   k_gather/k_scatter/k_scatter_zero/k_gather_range/k_scatter_range
//                     k_ft_array_{get_subset,assign_to_subset,assign_zero_to_subset,get_range,assign_to_range} (390-515)
//   k_zinv            k_ft_array_to_bytes_folded (629) / k_ft_array_to_bytes_affine (659), batched inversion
//   k_decode          k_ft_array_from_bytes_folded (735)
//   k_from_affine     k_ft_array_from_bytes_affine (793)
//   k_validate        k_ft_array_validate (859)
#include "internal.h"
#include "points.cuh"
#include "quad.cuh"

#define FT_TABLE_QUAL static __constant__
#define FT_WANT_L_SLIDE
#include "base_table.inc"

namespace ft {

static int g_sm_count = 0;
int sm_count()
{
    if (!g_sm_count) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (g_sm_count <= 0) g_sm_count = 1;
    }
    return g_sm_count;
}

static inline unsigned grid_for(size_t n, int block, int per_sm = 8)
{
    size_t need = (n + block - 1) / block;
    size_t cap = (size_t)sm_count() * per_sm;
    if (need > cap) need = cap;
    if (need == 0) need = 1;
    return (unsigned)need;
}

// ------------------------------------------------------------ group ops

__global__ void __launch_bounds__(256) k_set_zero(uint4 *p, size_t s, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        ge_p3 z;
        ge_zero(z);
        st_p3(p, s, i, z);
    }
}

__global__ void __launch_bounds__(256) k_broadcast(uint4 *p, size_t s, size_t n, const uint4 *q, size_t qs)
{
    FT_GRID_LOOP(i, n)
    {
#pragma unroll
        for (int k = 0; k < FT_PLANES; ++k) p[k * s + i] = q[k * qs];
    }
}

__global__ void __launch_bounds__(128, 4) k_add(uint4 *r, size_t rs, const uint4 *a, size_t as, size_t n, int sub)
{
    after_previous();
    FT_GRID_LOOP(i, n)
    {
        ge_p3 x, y;
        ld_p3(x, r, rs, i);
        ld_p3(y, a, as, i);
        if (sub) ge_subfrom(x, y);
        else ge_addto(x, y);
        st_p3(r, rs, i, x);
    }
}

// ciphertext add: (r1, r2) += (a1, a2) over one index space of 2n points,
// so both halves of a ciphertext array share one launch
__global__ void __launch_bounds__(128, 4) k_add_ct(uint4 *r1, size_t r1s, const uint4 *a1, size_t a1s, uint4 *r2,
                                                   size_t r2s, const uint4 *a2, size_t a2s, size_t n, int sub)
{
    after_previous();
    FT_GRID_LOOP(j, 2 * n)
    {
        const bool hi = j >= n;
        const size_t i = hi ? j - n : j;
        uint4 *r = hi ? r2 : r1;
        const uint4 *a = hi ? a2 : a1;
        const size_t rs = hi ? r2s : r1s, as = hi ? a2s : a1s;
        ge_p3 x, y;
        ld_p3(x, r, rs, i);
        ld_p3(y, a, as, i);
        if (sub) ge_subfrom(x, y);
        else ge_addto(x, y);
        st_p3(r, rs, i, x);
    }
}

// negates Y and T, as ge25519_neg of ftcrypto.cu:163-167 does
__global__ void __launch_bounds__(256) k_neg(uint4 *p, size_t s, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        ge_p3 x;
        ld_p3(x, p, s, i);
        fe_neg(x.Y, x.Y);
        fe_neg(x.T, x.T);
        st_p3(p, s, i, x);
    }
}

__global__ void __launch_bounds__(256) k_index(int64_t *out, const uint4 *p, size_t s, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        ge_p3 x;
        ld_p3(x, p, s, i);
        out[i] = !ge_iszero(x);
    }
}

__global__ void __launch_bounds__(128, 4) k_equal(int64_t *out, const uint4 *a, size_t as, const uint4 *b, size_t bs,
                                                  size_t n, int invert)
{
    FT_GRID_LOOP(i, n)
    {
        ge_p3 x, y;
        ld_p3(x, a, as, i);
        ld_p3(y, b, bs, i);
        out[i] = ge_equal(x, y) ^ invert;
    }
}

__global__ void __launch_bounds__(256) k_mux(uint4 *t, size_t ts, const int64_t *cond, const uint4 *f, size_t fs, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        if (cond[i] == 0) {
#pragma unroll
            for (int k = 0; k < FT_PLANES; ++k) t[k * ts + i] = f[k * fs + i];
        }
    }
}

__global__ void __launch_bounds__(256) k_gather(uint4 *d, size_t ds, const uint4 *s, size_t ss, const uint64_t *idx, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        size_t j = idx[i];
#pragma unroll
        for (int k = 0; k < FT_PLANES; ++k) d[k * ds + i] = s[k * ss + j];
    }
}

__global__ void __launch_bounds__(256) k_scatter(uint4 *d, size_t ds, const uint4 *s, size_t ss, const uint64_t *idx, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        size_t j = idx[i];
#pragma unroll
        for (int k = 0; k < FT_PLANES; ++k) d[k * ds + j] = s[k * ss + i];
    }
}

__global__ void __launch_bounds__(256) k_scatter_zero(uint4 *d, size_t ds, const uint64_t *idx, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        ge_p3 z;
        ge_zero(z);
        st_p3(d, ds, idx[i], z);
    }
}

__global__ void __launch_bounds__(256) k_gather_range(uint4 *d, size_t ds, const uint4 *s, size_t ss, size_t start,
                                                      size_t step, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        size_t j = start + i * step;
#pragma unroll
        for (int k = 0; k < FT_PLANES; ++k) d[k * ds + i] = s[k * ss + j];
    }
}

__global__ void __launch_bounds__(256) k_scatter_range(uint4 *d, size_t ds, const uint4 *s, size_t ss, size_t start,
                                                       size_t step, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        size_t j = start + i * step;
#pragma unroll
        for (int k = 0; k < FT_PLANES; ++k) d[k * ds + j] = s[k * ss + i];
    }
}

// ------------------------------------------------------------ wire formats

// Canonical outputs that divide by Z (folded and affine encodings): K points
// per thread, four threads, share one division-step inversion (quad_inv) by
// Montgomery's trick, 3 multiplications per point more.  A zero Z counts as 1 inside the
// product and its inverse as 0, which is what fe25519_invert(0) = 0 gives
// the reference.  Thread t of a warp takes the points 32 k + t of the warp's
// 32 K, so its loads and stores are those of whole warps; the products of
// the earlier points wait in shared memory (32 bytes per point).
static constexpr int ZINV_NT = 128;

// the Z of point i (1 past n), as loaded
FT_DEV void load_z(uint4 z[2], const uint4 *p, size_t s, size_t n, size_t i)
{
    z[0] = i < n ? p[4 * s + i] : make_uint4(1u, 0u, 0u, 0u);
    z[1] = i < n ? p[5 * s + i] : make_uint4(0u, 0u, 0u, 0u);
}

// 1 in the place of a zero Z, which the mask then tells
FT_DEV void use_z(fe &z, uint32_t &zero_mask, const uint4 w[2])
{
    fe_from_u4(z, w[0], w[1]);
    zero_mask = 0u - (uint32_t)fe_iszero(z);
    fe one;
    fe_1(one);
    fe_cmov(z, one, zero_mask);
}

// The lanes of a warp, converged, emit its points i, lane l the point l past a
// multiple of 32, below n.
struct EmitFolded {
    // Lanes 16 apart trade half of their 32 bytes, so that a store instruction
    // of the warp writes 512 contiguous bytes: the output may be host memory.
    FT_DEV static void emit(uint4 *o, size_t i, size_t n, const fe &x, const fe &y)
    {
        fe yc;
        fe_canon(yc, y);
        yc.v[7] ^= fe_isnegative(x) << 31;
        const uint4 a = u4_lo(yc), b = u4_hi(yc);
        const unsigned up = threadIdx.x >> 4 & 1u;
        uint4 t = up ? a : b;
        t.x = __shfl_xor_sync(0xffffffffu, t.x, 16);
        t.y = __shfl_xor_sync(0xffffffffu, t.y, 16);
        t.z = __shfl_xor_sync(0xffffffffu, t.z, 16);
        t.w = __shfl_xor_sync(0xffffffffu, t.w, 16);
        const size_t e = i - 16 * up; // lane l < 16 and l + 16: the points e and e + 16
        if (e < n) o[2 * e + up] = up ? t : a;
        if (e + 16 < n) o[2 * (e + 16) + up] = up ? b : t;
    }
};

struct EmitAffine {
    FT_DEV static void emit(uint4 *o, size_t i, size_t n, const fe &x, const fe &y)
    {
        fe xc, yc;
        fe_canon(xc, x);
        fe_canon(yc, y);
        if (i >= n) return;
        o += 4 * i;
        o[0] = u4_lo(xc);
        o[1] = u4_hi(xc);
        o[2] = u4_lo(yc);
        o[3] = u4_hi(yc);
    }
};

template <class Emit>
__global__ void __launch_bounds__(ZINV_NT) k_zinv(uint4 *out, const uint4 *p, size_t s, size_t n, int K)
{
    extern __shared__ uint4 pre[]; // [k][2][ZINV_NT]: product of the thread's first k points, k > 0
    uint4 *my = pre + threadIdx.x - 2 * ZINV_NT;
    const size_t base = ((size_t)blockIdx.x * (ZINV_NT / 32) + (threadIdx.x >> 5)) * 32 * K + (threadIdx.x & 31);
    // each point's words are loaded a step ahead of their use
    fe acc, z;
    uint32_t zm;
    uint4 w[2], nx[6];
    load_z(w, p, s, n, base);
    use_z(acc, zm, w);
    if (K > 1) load_z(nx, p, s, n, base + 32);
#pragma unroll 1
    for (int k = 1; k < K; ++k) {
        my[(2 * k) * ZINV_NT] = u4_lo(acc);
        my[(2 * k + 1) * ZINV_NT] = u4_hi(acc);
        use_z(z, zm, nx);
        if (k + 1 < K) load_z(nx, p, s, n, base + 32 * (size_t)(k + 1));
        fe_mul(acc, acc, z);
    }
    auto load = [&](int k) {
        const size_t i = base + 32 * (size_t)k;
        load_z(nx, p, s, n, i);
        if (i < n) {
#pragma unroll
            for (int c = 0; c < 4; ++c) nx[2 + c] = p[c * s + i];
        }
    };
    load(K - 1);
    // the quad's four products as one inverse: of this lane's and its
    // neighbour's, of both pairs', and back
    fe inv, other;
#pragma unroll
    for (int k = 0; k < 8; ++k) other.v[k] = __shfl_xor_sync(0xffffffffu, acc.v[k], 1);
    fe_mul(inv, acc, other);
#pragma unroll
    for (int k = 0; k < 8; ++k) z.v[k] = __shfl_xor_sync(0xffffffffu, inv.v[k], 2);
    fe_mul(inv, inv, z);
    fe_mul(other, other, z);
    quad_inv(inv, inv);
    fe_mul(inv, inv, other);
#pragma unroll 1
    for (int k = K - 1; k >= 0; --k) {
        const size_t i = base + 32 * (size_t)k;
        use_z(z, zm, nx);
        fe zinv = inv, x, y;
        fe_from_u4(x, nx[2], nx[3]);
        fe_from_u4(y, nx[4], nx[5]);
        if (k) {
            load(k - 1);
            fe q;
            fe_from_u4(q, my[(2 * k) * ZINV_NT], my[(2 * k + 1) * ZINV_NT]);
            fe_mul_x2(zinv, inv, q, inv, inv, z);
        }
        fe zero;
        fe_0(zero);
        fe_cmov(zinv, zero, zm);
        fe_mul_x2(x, x, zinv, y, y, zinv);
        Emit::emit(out, i, n, x, y);
    }
}

// Bound by the chain of 254 squarings per point.  `in` may be the caller's
// pinned memory: 32 bytes of a point across the host link wait behind the other
// warps' squarings, where a copy before the launch and the wait for it cost the
// call 28 us for 200,003 points (417 -> 389 us; 1,048,576: 1,969 -> 1,808; 16: 74
// -> 65).  (The next point's 32 bytes loaded a point ahead: 396 us, spills.)
__global__ void __launch_bounds__(128) k_decode(uint4 *p, size_t s, const uint4 *in, size_t n, long long *bad)
{
    FT_GRID_LOOP(i, n)
    {
        uint4 a = in[2 * i], b = in[2 * i + 1];
        uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        ge_p3 h;
        int r = ge_frombytes(h, w);
        st_p3(p, s, i, h);
        if (r) atomicMax(bad, (long long)i);
    }
}

// X, Y from bytes (top bit ignored), Z = 1, T = XY; no validation
__global__ void __launch_bounds__(256) k_from_affine(uint4 *p, size_t s, const uint4 *in, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
        uint4 w[4] = {in[4 * i], in[4 * i + 1], in[4 * i + 2], in[4 * i + 3]};
        uint32_t xw[8] = {w[0].x, w[0].y, w[0].z, w[0].w, w[1].x, w[1].y, w[1].z, w[1].w};
        uint32_t yw[8] = {w[2].x, w[2].y, w[2].z, w[2].w, w[3].x, w[3].y, w[3].z, w[3].w};
        ge_p3 h;
        fe_from_words(h.X, xw);
        fe_from_words(h.Y, yw);
        fe_1(h.Z);
        fe_mul(h.T, h.X, h.Y);
        st_p3(p, s, i, h);
    }
}

// bits [lo, lo + nb) of a 256-bit little-endian value, nb <= 32, lo constant
FT_DEV int64_t bits_at(const fe &c, int lo, int nb)
{
    int w = lo >> 5, b = lo & 31;
    uint64_t x = c.v[w];
    if (w + 1 < 8) x |= (uint64_t)c.v[w + 1] << 32;
    x >>= b;
    return (int64_t)(x & ((1ull << nb) - 1));
}

// canonical value -> the 10 signed limbs fe25519_frombytes (sodium_fe.cu:74-141)
// produces from the canonical bytes: same loads, same carry order
FT_DEV void fe_to_ref10(int32_t out[10], const fe &f)
{
    fe c;
    fe_canon(c, f);
    int64_t h[10];
    h[0] = bits_at(c, 0, 32);
    h[1] = bits_at(c, 32, 24) << 6;
    h[2] = bits_at(c, 56, 24) << 5;
    h[3] = bits_at(c, 80, 24) << 3;
    h[4] = bits_at(c, 104, 24) << 2;
    h[5] = bits_at(c, 128, 32);
    h[6] = bits_at(c, 160, 24) << 7;
    h[7] = bits_at(c, 184, 24) << 5;
    h[8] = bits_at(c, 208, 24) << 4;
    h[9] = (bits_at(c, 232, 24) & 8388607) << 2;
    int64_t carry;
    carry = (h[9] + (1LL << 24)) >> 25;
    h[0] += carry * 19;
    h[9] -= carry * (1LL << 25);
#pragma unroll
    for (int i = 1; i < 9; i += 2) {
        carry = (h[i] + (1LL << 24)) >> 25;
        h[i + 1] += carry;
        h[i] -= carry * (1LL << 25);
    }
#pragma unroll
    for (int i = 0; i < 10; i += 2) {
        carry = (h[i] + (1LL << 25)) >> 26;
        h[i + 1] += carry;
        h[i] -= carry * (1LL << 26);
    }
#pragma unroll
    for (int i = 0; i < 10; ++i) out[i] = (int32_t)h[i];
}

// sum of limb_i * 2^off_i (limbs signed, any magnitude below 2^31) mod p:
// positive and negative limbs go to two 288-bit accumulators, each folded
// with 2^256 = 38, and the results are subtracted
FT_DEV void fe_from_ref10(fe &f, const int32_t l[10])
{
    const int off[10] = {0, 26, 51, 77, 102, 128, 153, 179, 204, 230};
    uint32_t pos[16], neg[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) pos[k] = neg[k] = 0;
#pragma unroll
    for (int i = 0; i < 10; ++i) {
        int32_t v = l[i];
        uint32_t m = 0u - (uint32_t)(v < 0);
        uint32_t mag = ((uint32_t)v ^ m) - m;
        int w = off[i] >> 5, b = off[i] & 31;
        uint64_t sh = (uint64_t)mag << b;
        uint32_t lo = (uint32_t)sh, hi = (uint32_t)(sh >> 32);
        uint32_t cp = 0, cn = 0;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            uint64_t add = (k == w) ? lo : (k == w + 1 ? hi : 0u);
            uint64_t tp = (uint64_t)pos[k] + (add & ~(uint64_t)m) + cp;
            uint64_t tn = (uint64_t)neg[k] + (add & (uint64_t)m) + cn;
            pos[k] = (uint32_t)tp;
            cp = (uint32_t)(tp >> 32);
            neg[k] = (uint32_t)tn;
            cn = (uint32_t)(tn >> 32);
        }
    }
    fe a, b;
    fe_fold512(a, pos);
    fe_fold512(b, neg);
    fe_sub(f, a, b);
}

// Each warp converts 32 consecutive points into shared memory (rows of 41
// words: conflict-free) and writes their 5,120 contiguous bytes with
// coalesced stores; one thread writing its 160-byte struct directly made
// every store instruction of a warp touch 32 sectors.
__global__ void __launch_bounds__(128) k_to_ref160(int32_t *out, const uint4 *p, size_t s, size_t n)
{
    __shared__ int32_t stage[4][32 * 41];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int32_t *row = stage[warp] + 41 * lane;
#pragma unroll 1
    for (size_t base = (size_t)blockIdx.x * 128 + 32 * warp; base < n; base += (size_t)gridDim.x * 128) {
        const size_t i = base + lane;
        if (i < n) {
            ge_p3 h;
            ld_p3(h, p, s, i);
            fe_to_ref10(row, h.X);
            fe_to_ref10(row + 10, h.Y);
            fe_to_ref10(row + 20, h.Z);
            fe_to_ref10(row + 30, h.T);
        }
        __syncwarp();
        const int words = 40 * (int)(n - base < 32 ? n - base : 32);
        int32_t *o = out + 40 * base;
#pragma unroll 1
        for (int k = lane; k < words; k += 32) o[k] = stage[warp][41 * (k / 40) + k % 40];
        __syncwarp();
    }
}

// the mirror of k_to_ref160: each warp reads its 32 structs with coalesced
// loads into shared memory, then each thread converts its own
__global__ void __launch_bounds__(128) k_from_ref160(uint4 *p, size_t s, const int32_t *in, size_t n)
{
    __shared__ int32_t stage[4][32 * 41];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int32_t *row = stage[warp] + 41 * lane;
#pragma unroll 1
    for (size_t base = (size_t)blockIdx.x * 128 + 32 * warp; base < n; base += (size_t)gridDim.x * 128) {
        const int words = 40 * (int)(n - base < 32 ? n - base : 32);
        const int32_t *q = in + 40 * base;
#pragma unroll 1
        for (int k = lane; k < words; k += 32) stage[warp][41 * (k / 40) + k % 40] = q[k];
        __syncwarp();
        const size_t i = base + lane;
        if (i < n) {
            ge_p3 h;
            int32_t l[10];
#pragma unroll
            for (int j = 0; j < 10; ++j) l[j] = row[j];
            fe_from_ref10(h.X, l);
#pragma unroll
            for (int j = 0; j < 10; ++j) l[j] = row[10 + j];
            fe_from_ref10(h.Y, l);
#pragma unroll
            for (int j = 0; j < 10; ++j) l[j] = row[20 + j];
            fe_from_ref10(h.Z, l);
#pragma unroll
            for (int j = 0; j < 10; ++j) l[j] = row[30 + j];
            fe_from_ref10(h.T, l);
            st_p3(p, s, i, h);
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(256) k_to_packed(uint4 *out, const uint4 *p, size_t s, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
#pragma unroll
        for (int k = 0; k < FT_PLANES; ++k) out[8 * i + k] = p[k * s + i];
    }
}

__global__ void __launch_bounds__(256) k_from_packed(uint4 *p, size_t s, const uint4 *in, size_t n)
{
    FT_GRID_LOOP(i, n)
    {
#pragma unroll
        for (int k = 0; k < FT_PLANES; ++k) p[k * s + i] = in[8 * i + k];
    }
}

// ------------------------------------------------------------ validation

// L * A in the sliding-window sequence of ge25519_mul_l (sodium_ge.cu:795-847);
// variable time in the public group order only.
FT_DEV void ge_mul_l(ge_p3 &r, const ge_p3 &A)
{
    ge_cached Ai[8];
    ge_p1p1 t;
    ge_p3 u, A2;
    ge_p3_to_cached(Ai[0], A);
    ge_p3_dbl(t, A);
    ge_p1p1_to_p3(A2, t);
#pragma unroll 1
    for (int k = 1; k < 8; ++k) {
        ge_add(t, A2, Ai[k - 1]);
        ge_p1p1_to_p3(u, t);
        ge_p3_to_cached(Ai[k], u);
    }
    ge_p3_0(r);
#pragma unroll 1
    for (int i = 252; i >= 0; --i) {
        ge_p3_dbl(t, r);
        int d = FT_L_SLIDE_INIT[i];
        if (d > 0) {
            ge_p1p1_to_p3(u, t);
            ge_add(t, u, Ai[d / 2]);
        } else if (d < 0) {
            ge_p1p1_to_p3(u, t);
            ge_sub(t, u, Ai[(-d) / 2]);
        }
        ge_p1p1_to_p3(r, t);
    }
}

__global__ void __launch_bounds__(128) k_validate(const uint4 *p, size_t s, size_t n, long long *bad)
{
    FT_GRID_LOOP(i, n)
    {
        ge_p3 h;
        ld_p3(h, p, s, i);
        int ok = ge_is_on_curve(h);
        if (ok) {
            ge_p3 pl;
            ge_mul_l(pl, h);
            ok = fe_iszero(pl.X);
        }
        if (!ok) atomicMax(bad, (long long)i);
    }
}

// ------------------------------------------------------------ launchers

// *acc |= OR of v[0 .. n): one 64-bit atomic per warp
__global__ void __launch_bounds__(256) k_or_words(unsigned long long *acc, const uint64_t *v, size_t n)
{
    uint64_t x = 0;
    FT_GRID_LOOP(i, n) x |= v[i];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) x |= __shfl_xor_sync(0xffffffffu, x, d);
    if ((threadIdx.x & 31) == 0 && x) atomicOr(acc, (unsigned long long)x);
}

#define FT_LAUNCH(kern, n, block, ...)                                  \
    do {                                                                 \
        if ((n) == 0) return cudaSuccess;                                \
        kern<<<grid_for((n), (block)), (block), 0, st>>>(__VA_ARGS__);   \
        return cudaGetLastError();                                       \
    } while (0)

cudaError_t set_zero(View v, size_t n, cudaStream_t st) { FT_LAUNCH(k_set_zero, n, 256, v.p, v.s, n); }

cudaError_t or_words(uint64_t *acc, const uint64_t *v, size_t n, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(acc, 0, sizeof(uint64_t), st);
    if (e != cudaSuccess) return e;
    FT_LAUNCH(k_or_words, n, 256, (unsigned long long *)acc, v, n);
}
cudaError_t broadcast(View d, size_t n, View q, cudaStream_t st) { FT_LAUNCH(k_broadcast, n, 256, d.p, d.s, n, q.p, q.s); }
// (a block for every 128 points: 1,048,576 ciphertexts in 165 us, 178 with the
// 1,216 blocks of the other kernels)
static unsigned blocks_for(size_t n) { return (unsigned)((n + 127) / 128 < 0x7fffffff ? (n + 127) / 128 : 0x7fffffff); }

cudaError_t add(View r, View a, size_t n, int sub, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    return launch_next(k_add, blocks_for(n), 128, 0, st, r.p, r.s, a.p, a.s, n, sub);
}
cudaError_t add_ct(View r1, View r2, View a1, View a2, size_t n, int sub, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    return launch_next(k_add_ct, blocks_for(2 * n), 128, 0, st, r1.p, r1.s, a1.p, a1.s, r2.p, r2.s, a2.p, a2.s, n, sub);
}
cudaError_t neg(View v, size_t n, cudaStream_t st) { FT_LAUNCH(k_neg, n, 256, v.p, v.s, n); }
cudaError_t index_nonzero(int64_t *o, View v, size_t n, cudaStream_t st) { FT_LAUNCH(k_index, n, 256, o, v.p, v.s, n); }
cudaError_t equal(int64_t *o, View a, View b, size_t n, int inv, cudaStream_t st) { FT_LAUNCH(k_equal, n, 128, o, a.p, a.s, b.p, b.s, n, inv); }
cudaError_t mux(View t, const int64_t *c, View f, size_t n, cudaStream_t st) { FT_LAUNCH(k_mux, n, 256, t.p, t.s, c, f.p, f.s, n); }
cudaError_t gather(View d, View s, const uint64_t *ix, size_t n, cudaStream_t st) { FT_LAUNCH(k_gather, n, 256, d.p, d.s, s.p, s.s, ix, n); }
cudaError_t scatter(View d, View s, const uint64_t *ix, size_t n, cudaStream_t st) { FT_LAUNCH(k_scatter, n, 256, d.p, d.s, s.p, s.s, ix, n); }
cudaError_t scatter_zero(View d, const uint64_t *ix, size_t n, cudaStream_t st) { FT_LAUNCH(k_scatter_zero, n, 256, d.p, d.s, ix, n); }
cudaError_t gather_range(View d, View s, size_t a, size_t b, size_t n, cudaStream_t st) { FT_LAUNCH(k_gather_range, n, 256, d.p, d.s, s.p, s.s, a, b, n); }
cudaError_t scatter_range(View d, View s, size_t a, size_t b, size_t n, cudaStream_t st) { FT_LAUNCH(k_scatter_range, n, 256, d.p, d.s, s.p, s.s, a, b, n); }
cudaError_t decode(View v, const uint8_t *in, size_t n, long long *bad, cudaStream_t st) { FT_LAUNCH(k_decode, n, 128, v.p, v.s, (const uint4 *)in, n, bad); }
cudaError_t from_affine(View v, const uint8_t *in, size_t n, cudaStream_t st) { FT_LAUNCH(k_from_affine, n, 256, v.p, v.s, (const uint4 *)in, n); }
cudaError_t to_ref160(uint8_t *o, View v, size_t n, cudaStream_t st) { FT_LAUNCH(k_to_ref160, n, 128, (int32_t *)o, v.p, v.s, n); }
cudaError_t from_ref160(View v, const uint8_t *in, size_t n, cudaStream_t st) { FT_LAUNCH(k_from_ref160, n, 128, v.p, v.s, (const int32_t *)in, n); }
cudaError_t to_packed(uint8_t *o, View v, size_t n, cudaStream_t st) { FT_LAUNCH(k_to_packed, n, 256, (uint4 *)o, v.p, v.s, n); }
cudaError_t from_packed(View v, const uint8_t *in, size_t n, cudaStream_t st) { FT_LAUNCH(k_from_packed, n, 256, v.p, v.s, (const uint4 *)in, n); }
cudaError_t validate(View v, size_t n, long long *bad, cudaStream_t st) { FT_LAUNCH(k_validate, n, 128, v.p, v.s, n, bad); }

// Points per inversion: a warp's inversions cost its scheduler 24,000 cycles
// (12 us alone) and a point in the loops 1.5 us, so the points go one to a
// thread until every scheduler has a warp (sm_count x 128 threads), and then
// into longer threads: one block per SM up to 18 points a thread, two, three
// (72 KB of shared memory each), each launch one wave.  Measured (n: this K; one
// point a thread; 8; the earlier kernel's 8 points per chain of 254 squarings),
// us a launch into device memory: 16: 15 (K = 1); 15; 26; 90.  65,536: 23 (4);
// 44; 31; 87.  200,003: 38 (11); 112; 44; 88.  400,000: 51 (11); 209; 59.
// 1,048,576: 96 (18); 529; 122; 314.  (No K from 1 to 18 was better than the
// rule's by 1 us at eight lengths.)
// Into host memory a launch takes at least what the host link does, and blocks
// that start one after another keep it busy: threads of 6 points at most
// (1,048,576 folded points, the call: 253 us at 18, 219 at 6, 217 at 4;
// 4,194,304: 852, 755, 762).
static constexpr int ZINV_MAX_K = 18, ZINV_HOST_K = 6;
static int zinv_points(size_t n, int max_k)
{
    const size_t per_sm = (size_t)sm_count() * ZINV_NT;
    for (size_t blocks = 1; blocks <= 3; ++blocks) {
        const size_t k = (n + blocks * per_sm - 1) / (blocks * per_sm);
        if (k <= (size_t)max_k) return (int)k;
    }
    return max_k;
}

template <class Emit>
static cudaError_t zinv_launch(uint8_t *o, View v, size_t n, cudaStream_t st, int max_k = ZINV_MAX_K)
{
    if (n == 0) return cudaSuccess;
    const int K = zinv_points(n, max_k);
    const size_t smem = (size_t)(K - 1) * 2 * ZINV_NT * sizeof(uint4);
    const unsigned grid = (unsigned)((n + (size_t)ZINV_NT * K - 1) / ((size_t)ZINV_NT * K));
    static SmemAttr attr;
    cudaError_t e = ensure_smem_attr(attr, (const void *)k_zinv<Emit>, (size_t)ZINV_MAX_K * 2 * ZINV_NT * sizeof(uint4));
    if (e != cudaSuccess) return e;
    k_zinv<Emit><<<grid, ZINV_NT, smem, st>>>((uint4 *)o, v.p, v.s, n, K);
    return cudaGetLastError();
}

cudaError_t encode(uint8_t *o, View v, size_t n, cudaStream_t st) { return zinv_launch<EmitFolded>(o, v, n, st); }
cudaError_t encode_to_host(uint8_t *o, View v, size_t n, cudaStream_t st)
{
    return zinv_launch<EmitFolded>(o, v, n, st, ZINV_HOST_K);
}
cudaError_t to_affine(uint8_t *o, View v, size_t n, cudaStream_t st) { return zinv_launch<EmitAffine>(o, v, n, st); }

cudaError_t copy_points(View d, View s, size_t n, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    return cudaMemcpy2DAsync(d.p, d.s * sizeof(uint4), s.p, s.s * sizeof(uint4), n * sizeof(uint4), FT_PLANES,
                             cudaMemcpyDeviceToDevice, st);
}

} // namespace ft
