// umma.cuh — tcgen05.mma, mbarriers and bulk copies for the kernels that use
// the tensor cores as an exact table lookup (k_comb256 in k_encrypt.cu).
//
// The A operand is in tensor memory, written by the threads that own its rows;
// B sits in shared memory in the K-major layout without swizzle: core matrices
// of 8 rows x 16 bytes (128 contiguous bytes); here all rows of one 16-byte
// column chunk are contiguous, so element (row, k) of an f16 matrix of R rows
// is at (k / 8) * 16 R + row * 16 + (k % 8) * 2.
//
// Every wait is bounded: mbar_wait gives up after a fixed number of polls and
// says so, and the kernel then leaves its loops, waits (bounded again) for
// the copies and the products that it has started and frees its tensor memory
// (comb_roles.cuh).
#pragma once
#include "tmem.cuh"

namespace ft {

FT_DEV_TM uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

FT_DEV_TM void mbar_init(uint64_t *b, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}

FT_DEV_TM void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// polls until the phase of the given parity has completed; false after
// MBAR_POLLS polls (each of which the hardware may hold for a while)
static constexpr int MBAR_POLLS = 1 << 20;

// SLEEP_NS > 0: sleeps in between, for a warp whose polls would take issue
// slots from warps that compute
template <int SLEEP_NS = 0>
FT_DEV_TM bool mbar_wait(uint64_t *b, uint32_t parity)
{
    const uint32_t a = smem_addr(b);
    uint32_t done = 0;
#pragma unroll 1
    for (int i = 0; i < MBAR_POLLS && !done; ++i) {
        if (SLEEP_NS && i) __nanosleep(SLEEP_NS);
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(a), "r"(parity)
                     : "memory");
    }
    return done != 0;
}

FT_DEV_TM void mbar_arrive(uint64_t *b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}

// one arrival on b, and `bytes` of bulk copies to come before its phase ends
FT_DEV_TM void mbar_expect(uint64_t *b, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}

// `bytes` (a multiple of 16, both addresses 16-byte aligned) from global to
// shared memory, counted on b
FT_DEV_TM void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *b)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(b))
                 : "memory");
}

// generic-proxy writes of shared memory made visible to the tensor core
FT_DEV_TM void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// shared-memory matrix descriptor: K-major, no swizzle; `lbo` bytes between
// core matrices along K, `sbo` along the rows
FT_DEV_TM uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3fffu) | (uint64_t)((lbo >> 4) & 0x3fffu) << 16 |
           (uint64_t)((sbo >> 4) & 0x3fffu) << 32 | (uint64_t)1 << 46;
}

// kind::f16 with f16 operands, both K-major, f32 accumulators: D type at bit
// 4, N / 8 at 17, M / 16 at 24
constexpr uint32_t umma_idesc_f16(int m, int n)
{
    return 1u << 4 | (uint32_t)(n >> 3) << 17 | (uint32_t)(m >> 4) << 24;
}

// D (+)= A B, one K = 16 step, A in tensor memory (row m in lane m, two
// consecutive f16 a column: 8 columns); issued by one thread
FT_DEV_TM void umma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc, bool accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "r"(a_tmem), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
                 : "memory");
}

// arrives on b when the issuing thread's earlier tcgen05.mma are done
FT_DEV_TM void umma_commit(uint64_t *b)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(b))
                 : "memory");
}

// thread-block clusters: this block's rank and their number, a barrier of all
// threads of the cluster, and a store into the same place of another block's
// shared memory
FT_DEV_TM unsigned cluster_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

FT_DEV_TM unsigned cluster_size()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

FT_DEV_TM void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

FT_DEV_TM void cluster_store(uint4 *local, unsigned rank, uint4 v)
{
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(local)), "r"(rank));
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

FT_DEV_TM void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

FT_DEV_TM void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

FT_DEV_TM void tmem_st1(uint32_t ta, uint32_t v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(ta), "r"(v) : "memory");
}

// 24 consecutive columns of the thread's lane
FT_DEV_TM void tmem_ld24(uint32_t ta, uint32_t r[24])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%24];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23}, "
                 "[%25];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]),
                   "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]),
                   "=&r"(r[14]), "=&r"(r[15]), "=&r"(r[16]), "=&r"(r[17]), "=&r"(r[18]), "=&r"(r[19]), "=&r"(r[20]),
                   "=&r"(r[21]), "=&r"(r[22]), "=&r"(r[23])
                 : "r"(ta), "r"(ta + 8u)
                 : "memory");
}

} // namespace ft
