// grid_barrier.cuh -- grid-wide barrier of a cooperative (co-resident) launch
// with a bounded wait.
#pragma once

#include "common.cuh"

namespace aot
{
// Barrier words (zeroed before the first launch; each barrier leaves them as it
// found them, but for the generation).
constexpr unsigned kBarrierGroups = 8, kBarrierFlat = 192;
struct GridBarrier
{
    u32 generation;  // barriers passed
    int error;       // a wait gave up
    u32 arrived;     // CTAs (or groups) at the current barrier
    u32 pad[13];
    u32 group[kBarrierGroups][16];  // CTAs of each group, a word per 64 bytes
};

constexpr u32 kBarrierSpins = 1u << 22;  // polls of about 128 ns: well over 0.5 s
constexpr u32 kBarrierHot = 64;          // polls without a pause: most barriers open within a microsecond

// Every CTA of the grid arrives; the last one opens the next generation.  CTAs
// of a large grid arrive in groups, the last of a group for the group: the
// atomics on one word pass one by one, 592 of them in about 3 us.  A CTA that polls more than
// kBarrierSpins times (or sees another CTA's error) records the error and
// leaves; the result is false for it and for every CTA that reads the error
// after the barrier, and the kernel returns.
__device__ __forceinline__ bool gridBarrier(GridBarrier *b)
{
    __shared__ int sOk;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        volatile u32 *gen = &b->generation;
        volatile int *err = &b->error;
        const u32 g = *gen;
        __threadfence();
        bool last;
        if (gridDim.x <= kBarrierFlat)
        {
            last = atomicAdd(&b->arrived, 1u) == gridDim.x - 1;
        }
        else
        {
            const u32 mine = blockIdx.x % kBarrierGroups;
            const u32 members = (gridDim.x - mine + kBarrierGroups - 1) / kBarrierGroups;
            last = atomicAdd(&b->group[mine][0], 1u) == members - 1;
            if (last)
            {
                atomicExch(&b->group[mine][0], 0u);
                __threadfence();
                last = atomicAdd(&b->arrived, 1u) == kBarrierGroups - 1;
            }
        }
        if (last)
        {
            atomicExch(&b->arrived, 0u);
            __threadfence();
            atomicAdd(&b->generation, 1u);
        }
        else
        {
            u32 spins = 0;
            while (*gen == g)
            {
                if (++spins <= kBarrierHot) continue;
                if (*err || spins > kBarrierSpins)
                {
                    atomicExch(&b->error, 1);
                    break;
                }
                __nanosleep(128);
            }
        }
        __threadfence();
        sOk = *err == 0;
    }
    __syncthreads();
    return sOk != 0;
}

template <class T>
__device__ __forceinline__ T vload(const T &x)
{
    return *static_cast<const volatile T *>(&x);
}
}  // namespace aot
