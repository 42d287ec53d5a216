// sort_fused.cuh -- the passes and the repair of a contiguous sort in one
// launch by team (grid_barrier.cuh).
//
// Small sorts are bound by launches: 10k keys in 3 passes spend 5 us in each
// pass, 1 us and a launch in each of the 5 passes the plan leaves out, and two
// launches in the repair.  Here the CTAs go through the same tiles phase by
// phase, with a grid barrier between:
//   counts     (optional) digit counts of the passes that run, and their bins;
//   passes     the onesweep passes; in each, CTAs take tiles from the pass's
//              counter until it runs out.  A tile's look-back waits only for
//              tiles taken before it, by CTAs that are resident and do not
//              wait for later tiles, so every wait ends.  (Without counts the
//              roll of the team closes behind the first pass: whoever takes a
//              tile is on it);
//   repair     the runs of equal high digits (sort_repair.cuh), tile by tile,
//              then the long ones.
#pragma once

#include "sort_repair.cuh"

namespace aot
{
namespace sort
{
struct FusedArgs
{
    PassArgs p;
    RepairArgs r;
    u32 tiles;
    u32 *hist;    // digit counts to be made (zero on entry), or nullptr: bins are in place
    u32 *binsOut; // (with hist) p.bins
    bool repair;  // the plan may leave digits out (else all passes run)
    bool whole;   // all 64 bits are sorted
};

template <int Items>
struct FusedShared
{
    union
    {
        SharedPass<kRadixBits, Items> pass;
        RepairShared<kThreads * Items> repair;
        LongShared<kThreads> longRun;
        u32 hist[kPassSlots * kRadix];
    };
};

// Three CTAs per SM, as the forest's sort.
template <int Items>
static __global__ void __launch_bounds__(kThreads, 3) fusedSortKernel(FusedArgs a)
{
    constexpr int kTile = kThreads * Items;
    static_assert(kThreads == kRepairThreads, "one CTA shape");
    extern __shared__ __align__(16) unsigned char smemRaw[];
    FusedShared<Items> &sm = *reinterpret_cast<FusedShared<Items> *>(smemRaw);
    const PassArgs &p = a.p;
    GridBarrier *bar = &p.ctl->sortBar;
    const int first = int(p.ctl->first);
    if (a.hist)
        for (int i = threadIdx.x; i < kPassSlots * kRadix; i += kThreads) sm.hist[i] = 0;
    Team team{enterRoll(bar), 0};
    if (team.rank == kLeftOut) return;
    const auto fail = [&] {
        if (threadIdx.x == 0) atomicExch(p.error, kErrLookback);
    };
    const auto barrier = [&] {
        if (!team.size) team.size = closeRoll(bar);
        return team.size && gridBarrier(bar, team);
    };
    if (a.hist)
    {
        team.size = closeRoll(bar);
        if (!team.size) return fail();
        for (size_t g = size_t(team.rank) * kThreads + threadIdx.x; g < p.n; g += size_t(team.size) * kThreads)
        {
            const u64 k = p.keysIn[g];
            for (int q = first; q < p.passes; ++q)
            {
                const int shift = p.beginBit + q * kRadixBits;
                const int bits = min(kRadixBits, p.endBit - shift);
                atomicAdd(&sm.hist[q * kRadix + int((k >> shift) & ((1u << bits) - 1))], 1u);
            }
        }
        __syncthreads();
        for (int i = first * kRadix + threadIdx.x; i < p.passes * kRadix; i += kThreads)
            if (sm.hist[i]) atomicAdd(a.hist + i, sm.hist[i]);
        if (!barrier()) return fail();
        if (team.rank == 0) scanBins(a.hist, a.binsOut, first, p.passes);
        if (!barrier()) return fail();
    }
    for (int pass = first; pass < p.passes; ++pass)
    {
        const int slot = pass - first;
        const int out = (p.endsIn0 ? p.passes - 1 - pass : slot + 1) & 1;
        const int shift = p.beginBit + pass * kRadixBits;
        const u64 *keysIn = slot ? (out ? p.k[0] : p.k[1]) : p.keysIn;
        const u32 *valsIn = slot ? (out ? p.v[0] : p.v[1]) : p.valsIn;
        while (onesweepTile<kRadixBits, Items>(ContiguousTiles<kTile>{p.n, p.bins + pass * kRadix}, keysIn, valsIn,
                                               out ? p.k[1] : p.k[0], out ? p.v[1] : p.v[0], shift,
                                               p.ctl->tileCounters + slot, p.status, passTag(p.ctl->epoch + u32(slot)),
                                               p.error, min(kRadixBits, p.endBit - shift), kLookbackSpins, a.tiles))
            __syncthreads();
        if (!barrier()) return fail();
    }
    if (!a.repair) return;
    const RepairArgs &r = a.r;
    if (first == 0)
    {
        // every pass has run; only the sample is left
        if (r.sample)
            for (size_t j = size_t(team.rank) * kThreads + threadIdx.x; (j << kSampleShift) < r.n;
                 j += size_t(team.size) * kThreads)
                r.sample[j] = r.k[0][j << kSampleShift];
        return;
    }
    if (vload(*p.error)) return;
    const bool inPlace = r.endsIn0 || ((u32(r.passes) - u32(first)) & 1u) == 0;
    for (u32 t = team.rank; t < a.tiles; t += team.size)
    {
        __syncthreads();
        const size_t begin = size_t(t) * kTile;
        if (a.whole && first == 4) repairTile<4>(r, sm.repair, u32(first), inPlace, begin, 0, r.n);
        else if (a.whole && first < 4) repairTile<3>(r, sm.repair, u32(first), inPlace, begin, 0, r.n);
        else repairTile<0>(r, sm.repair, u32(first), inPlace, begin, 0, r.n);
    }
    if (!barrier()) return fail();
    const u32 runs = vload(p.ctl->longRuns);
    if (runs) sortLongRuns(r, sm.longRun, first, runs, team);
}

// The kernel of a configuration (nullptr: none) and its shared memory.
static inline const void *fusedSort(int config, size_t &smem)
{
    if (kSortConfigs[config].bits != kRadixBits) return nullptr;
    switch (kSortConfigs[config].items)
    {
    case 8: smem = sizeof(FusedShared<8>); return reinterpret_cast<const void *>(&fusedSortKernel<8>);
    case 10: smem = sizeof(FusedShared<10>); return reinterpret_cast<const void *>(&fusedSortKernel<10>);
    case 16: smem = sizeof(FusedShared<16>); return reinterpret_cast<const void *>(&fusedSortKernel<16>);
    default: return nullptr;
    }
}
}  // namespace sort
}  // namespace aot
