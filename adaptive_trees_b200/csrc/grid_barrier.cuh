// grid_barrier.cuh -- grid-wide barrier with a bounded wait, among the CTAs of
// a launch that run at the same time.
//
// A barrier ends only if every CTA that has to arrive is resident.  A
// cooperative launch makes sure of that by waiting until the whole grid fits
// beside what else runs on the GPU: 8 of 148 SMs held by another stream for
// 1.2 s held up a 1M particle build (0.2 ms) for as long.  A launch by team
// starts like any other.  Its CTAs enter a roll as they start; the roll closes
// when all have come, or when no more come for a while (kRollStill), and the
// CTAs on it -- all resident -- do the whole work, by their rank on the roll
// and the number on it.  A CTA that starts later returns at once.
#pragma once

#include "common.cuh"

namespace aot
{
// Barrier words (zero before every launch that uses them).
constexpr unsigned kBarrierGroups = 8, kBarrierFlat = 192;
struct GridBarrier
{
    u32 generation;  // barriers passed
    int error;       // a wait gave up
    u32 arrived;     // CTAs (or groups) at the current barrier
    u32 roll;        // CTAs that have started | kRollClosed
    u32 size;        // CTAs on the closed roll (0 before)
    u32 pad[11];
    u32 group[kBarrierGroups][16];  // CTAs of each group, a word per 64 bytes
};

constexpr u32 kBarrierSpins = 1u << 22;  // polls of about 128 ns: well over 0.5 s
constexpr u32 kBarrierHot = 64;          // polls without a pause: most barriers open within a microsecond
constexpr u32 kRollClosed = 0x80000000u;
constexpr u32 kRollStill = 64;           // polls of about 1 us without a new CTA that close the roll
constexpr u32 kLeftOut = 0xffffffffu;    // rank of a CTA that came after the roll was closed

// The CTAs that share a launch's work, and this one's place among them.
struct Team
{
    u32 rank, size;
};
// A whole grid (ordinary kernels and cooperative launches).
__device__ __forceinline__ Team wholeGrid() { return {blockIdx.x, gridDim.x}; }

template <class T>
__device__ __forceinline__ T vload(const T &x)
{
    return *static_cast<const volatile T *>(&x);
}

// Enters this CTA in the roll: its rank, or kLeftOut (it then returns).  The
// first of the team has rank 0.
__device__ __forceinline__ u32 enterRoll(GridBarrier *b)
{
    __shared__ u32 sRank;
    if (threadIdx.x == 0)
    {
        const u32 r = atomicAdd(&b->roll, 1u);
        sRank = r & kRollClosed ? kLeftOut : r;
        // the last one of the grid: nobody is left to wait for
        if (r == gridDim.x - 1) *static_cast<volatile u32 *>(&b->size) = gridDim.x;
    }
    __syncthreads();
    return sRank;
}

// Closes the roll (all threads of every CTA on it); the CTAs on it, or 0 where
// the wait gave up.
__device__ __forceinline__ u32 closeRoll(GridBarrier *b, u32 spinLimit = kBarrierSpins, u32 still = kRollStill)
{
    __shared__ u32 sSize;
    if (threadIdx.x == 0)
    {
        u32 seen = 0, same = 0, size = 0;
        for (u32 spins = 0; (size = vload(b->size)) == 0; ++spins)
        {
            const u32 roll = vload(b->roll);
            if (roll != seen)
            {
                seen = roll;
                same = 0;
            }
            else if (++same > still && !(roll & kRollClosed))
            {
                const u32 before = atomicOr(&b->roll, kRollClosed);
                if (!(before & kRollClosed)) *static_cast<volatile u32 *>(&b->size) = before;
                continue;
            }
            if (spins > spinLimit)
            {
                atomicExch(&b->error, 1);
                break;
            }
            if (spins > kBarrierHot / 4) __nanosleep(256);
        }
        sSize = size;
    }
    __syncthreads();
    return sSize;
}

// Every CTA of the team arrives; the last one opens the next generation.  CTAs
// of a large team arrive in groups, the last of a group for the group: the
// atomics on one word pass one by one, 592 of them in about 3 us.  A CTA that polls more than
// spinLimit times (or sees another CTA's error) records the error and
// leaves; the result is false for it and for every CTA that reads the error
// after the barrier, and the kernel returns.
__device__ __forceinline__ bool gridBarrier(GridBarrier *b, const Team &team, u32 spinLimit = kBarrierSpins)
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
        if (team.size <= kBarrierFlat)
        {
            last = atomicAdd(&b->arrived, 1u) == team.size - 1;
        }
        else
        {
            const u32 mine = team.rank % kBarrierGroups;
            const u32 members = (team.size - mine + kBarrierGroups - 1) / kBarrierGroups;
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
                if (*err || spins > spinLimit)
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
}  // namespace aot
