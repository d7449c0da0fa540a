// points.cuh — structure-of-arrays point storage in HBM.
//
// An array of n points is 8 planes of 16-byte words (uint4), plane stride
// `s` elements (s >= n):
//   plane 0,1: X words 0-3, 4-7     plane 4,5: Z words 0-3, 4-7
//   plane 2,3: Y words 0-3, 4-7     plane 6,7: T words 0-3, 4-7
// Thread i reads point i with eight 16-byte loads; a warp's load of one plane
// is 512 contiguous bytes.  128 bytes per point, the algorithmic minimum for
// an extended point (the reference stores 160-byte AoS ge25519_p3 structs).
#pragma once
#include "ge.cuh"
#include "u4.cuh"

#define FT_PLANES 8


FT_DEV void ld_p3(ge_p3 &r, const uint4 *__restrict__ p, size_t s, size_t i)
{
    uint4 w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) w[k] = p[k * s + i];
    fe_from_u4(r.X, w[0], w[1]);
    fe_from_u4(r.Y, w[2], w[3]);
    fe_from_u4(r.Z, w[4], w[5]);
    fe_from_u4(r.T, w[6], w[7]);
}

FT_DEV void st_p3(uint4 *__restrict__ p, size_t s, size_t i, const ge_p3 &r)
{
    p[0 * s + i] = u4_lo(r.X);
    p[1 * s + i] = u4_hi(r.X);
    p[2 * s + i] = u4_lo(r.Y);
    p[3 * s + i] = u4_hi(r.Y);
    p[4 * s + i] = u4_lo(r.Z);
    p[5 * s + i] = u4_hi(r.Z);
    p[6 * s + i] = u4_lo(r.T);
    p[7 * s + i] = u4_hi(r.T);
}

// warp shuffle of a whole point
FT_DEV void shfl_up_p3(ge_p3 &o, const ge_p3 &v, int delta)
{
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        o.X.v[k] = __shfl_up_sync(0xffffffffu, v.X.v[k], delta);
        o.Y.v[k] = __shfl_up_sync(0xffffffffu, v.Y.v[k], delta);
        o.Z.v[k] = __shfl_up_sync(0xffffffffu, v.Z.v[k], delta);
        o.T.v[k] = __shfl_up_sync(0xffffffffu, v.T.v[k], delta);
    }
}

// shared-memory staging of one point per slot, stored as 8 uint4
FT_DEV void sm_st_p3(uint4 *sm, int slot, const ge_p3 &r)
{
    uint4 *q = sm + 8 * slot;
    q[0] = u4_lo(r.X); q[1] = u4_hi(r.X); q[2] = u4_lo(r.Y); q[3] = u4_hi(r.Y);
    q[4] = u4_lo(r.Z); q[5] = u4_hi(r.Z); q[6] = u4_lo(r.T); q[7] = u4_hi(r.T);
}

FT_DEV void sm_ld_p3(ge_p3 &r, const uint4 *sm, int slot)
{
    const uint4 *q = sm + 8 * slot;
    fe_from_u4(r.X, q[0], q[1]);
    fe_from_u4(r.Y, q[2], q[3]);
    fe_from_u4(r.Z, q[4], q[5]);
    fe_from_u4(r.T, q[6], q[7]);
}

// Points on their way from global memory to shared memory without registers:
// a thread's slot of point j is 8 uint4, `threads` apart, and is the thread's
// alone, so points_wait by that thread is all that orders it.
FT_DEV void point_fetch(uint4 *slot, int threads, const uint4 *p, size_t s, size_t i)
{
#pragma unroll
    for (int k = 0; k < 8; ++k)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(slot + k * threads)),
                     "l"(p + k * s + i)
                     : "memory");
}

FT_DEV void points_sent() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// all but the last N groups of this thread's fetches have arrived
template <int N>
FT_DEV void points_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// First statement of a kernel launched by launch_next (internal.h): nothing of
// the launches before is read or overwritten before they are done, and the next
// such launch of the stream may place its blocks when all of this one's are past
// that.  (Allowed to from the start, those of several launches to come fill SMs
// while they wait, and the blocks that run are unevenly placed: rows of additions
// of 80 to 150 blocks 6.9 to 7.7 us each, 3.7 this way, 6.2 as plain launches; of
// 153 to 180 7.4 to 7.9, 4.7 to 4.9, 6.2; more than 1,000 the same.)
FT_DEV void after_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// grid-stride loop bounds in size_t
#define FT_GRID_LOOP(i, n) \
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += (size_t)blockDim.x * gridDim.x)
