// forest_sort.cuh -- the segmented sort of every system of a forest in one
// persistent (cooperative) launch.
//
// After the keys and the counts of their high digits (keygenKernel, a launch
// of its own at full occupancy), the phases of the launch-per-stage path,
// separated by grid barriers instead of launch boundaries:
//   plan       keys sampled at random positions tell how many high digits the
//              passes have to cover (sort_plan.cuh); every CTA draws the same
//              conclusion from the counts;
//   bins       per system (one CTA each) and pass, the global start of each
//              digit; a plan of more digits than key generation counted
//              counts the others first;
//   passes     the plan's onesweep passes; in each, CTAs take tiles from the pass's
//              counter until it runs out.  A tile's look-back waits only for
//              tiles taken before it, by CTAs that are resident and do not
//              wait for later tiles, so every wait ends;
//   repair     the runs of equal high digits (sort_repair.cuh), tile by tile,
//              then the long ones;
//   active     each system's active count (escaped keys sort last) and the
//              key sample of a build by levels.
// Only the 8-bit configurations (key generation counts their digits) run here.
#pragma once

#include "forest.cuh"
#include "grid_barrier.cuh"

namespace aot
{
namespace forest
{
// First pass whose digits key generation counts before a persistent sort
// (which plans after it): most plans pass over four digits or fewer.
constexpr int kCountedFrom = 4;

struct SortArgs
{
    Bufs f;                   // systems, per-system state, sorted keys (f.P = keys[0])
    sort::SegmentTiles tiles; // the tile table (bins: [pass][system][digit])
    u32 numTiles;
    sort::RepairArgs r;       // buffers, list of long runs, control block (zero on entry but for its epoch)
    sort::PlanArgs plan;      // (counters zero on entry)
    u32 *hist;                // [system][pass slot][digit]: counts of the passes from kCountedFrom on, else zero
    u32 *bins;
    u64 *status;              // [tile][digit]
    int *error;               // bounded look-back gave up
    u64 *sample;              // every 32nd sorted key (nullptr: none)
    size_t ns;
    GridBarrier *bar;
};

// A barrier gave up: the forest's error word tells the host (the keys are
// not sorted, and what follows on the stream leaves them alone).
__device__ __forceinline__ void fail(const SortArgs &p)
{
    if (threadIdx.x == 0) atomicExch(p.error, kErrLookback);
}

template <int Items>
struct SortShared
{
    union
    {
        sort::SharedPass<sort::kRadixBits, Items> pass;
        sort::RepairShared<sort::kThreads * Items> repair;
        sort::LongShared<sort::kThreads> longRun;
        sort::PlanShared plan;
        u32 hist[sort::kMaxPasses * sort::kRadix];
    };
};

// Digit counts of the passes [first, kCountedFrom) (a CTA per tile in turn).
__device__ __forceinline__ void countLowDigits(const SortArgs &p, int first, u32 *sh)
{
    for (int i = threadIdx.x; i < kCountedFrom * sort::kRadix; i += blockDim.x) sh[i] = 0;
    for (u32 t = blockIdx.x; t < p.numTiles; t += gridDim.x)
    {
        __syncthreads();
        for (u32 g = p.tiles.tileBegin[t] + threadIdx.x; g < p.tiles.tileEnd[t]; g += blockDim.x)
        {
            const u64 k = p.r.k[0][g];
            for (int q = first; q < kCountedFrom; ++q)
                atomicAdd(&sh[q * sort::kRadix + int((k >> (q * sort::kRadixBits)) & (sort::kRadix - 1))], 1u);
        }
        __syncthreads();
        u32 *h = p.hist + size_t(p.tiles.tileSeg[t]) * sort::kPassSlots * sort::kRadix;
        for (int i = first * sort::kRadix + threadIdx.x; i < kCountedFrom * sort::kRadix; i += blockDim.x)
        {
            if (sh[i]) atomicAdd(h + i, sh[i]);
            sh[i] = 0;
        }
    }
}

// Three CTAs per SM: the registers of the pass loop fit without spills.
template <int Items>
static __global__ void __launch_bounds__(sort::kThreads, 3) sortKernel(SortArgs p)
{
    constexpr int kTile = sort::kThreads * Items;
    static_assert(sort::kThreads == sort::kPlanThreads && sort::kThreads == sort::kRepairThreads, "one CTA shape");
    extern __shared__ __align__(16) unsigned char smemRaw[];
    SortShared<Items> &sm = *reinterpret_cast<SortShared<Items> *>(smemRaw);
    const u32 epoch = vload(p.r.ctl->epoch) + sort::kEpochStep;
    if (blockIdx.x * blockDim.x < p.plan.samples)
    {
        const auto keyAt = [&](size_t g, u32 &group) {
            group = systemOf(p.tiles.segBase, p.f.numSystems, u32(g));
            return p.r.k[0][g];
        };
        sort::planSample(keyAt, p.r.n, p.plan, epoch, sm.plan);
    }
    for (int sys = blockIdx.x; sys < p.f.numSystems; sys += gridDim.x)
        systemBins(p.f.systems, p.f.numSystems, sys, p.hist, p.bins, kCountedFrom, sort::kMaxPasses);
    if (!gridBarrier(p.bar, wholeGrid())) return fail(p);
    // every CTA has read it; stored before the first word that carries a tag of
    // it, so that the next sort has other tags however this one ends (with the
    // tags of a sort that gave up, its words would be taken for published
    // counts, and the places made of them can lie outside the buffers)
    if (blockIdx.x == 0 && threadIdx.x == 0) p.r.ctl->epoch = epoch;
    u32 repeats[sort::kPlanSets], more[sort::kPlanSets];
#pragma unroll
    for (int k = 0; k < sort::kPlanSets; ++k)
    {
        repeats[k] = vload(p.plan.counters->repeats[k]);
        more[k] = vload(p.plan.counters->more[k]);
    }
    const int first = p.plan.force >= 0 ? p.plan.force : int(sort::planFirst(repeats, more, p.plan.samples, p.r.n));
    if (blockIdx.x == 0 && threadIdx.x == 0) p.r.ctl->first = u32(first);  // (for who asks)
    if (first < kCountedFrom)
    {
        countLowDigits(p, first, sm.hist);
        if (!gridBarrier(p.bar, wholeGrid())) return fail(p);
        for (int sys = blockIdx.x; sys < p.f.numSystems; sys += gridDim.x)
            systemBins(p.f.systems, p.f.numSystems, sys, p.hist, p.bins, first, kCountedFrom);
        if (!gridBarrier(p.bar, wholeGrid())) return fail(p);
    }
    for (int pass = first; pass < sort::kMaxPasses; ++pass)
    {
        const int slot = pass - first;
        sort::SegmentTiles tiles = p.tiles;
        tiles.bins = p.bins + size_t(pass) * p.f.numSystems * sort::kRadix;
        const bool odd = slot & 1;
        while (sort::onesweepTile<sort::kRadixBits, Items>(
            tiles, odd ? p.r.k[1] : p.r.k[0], slot == 0 ? nullptr : odd ? p.r.v[1] : p.r.v[0],
            odd ? p.r.k[0] : p.r.k[1], odd ? p.r.v[0] : p.r.v[1], pass * sort::kRadixBits,
            p.r.ctl->tileCounters + slot, p.status, sort::passTag(epoch + u32(slot)), p.error, sort::kRadixBits,
            sort::kLookbackSpins, p.numTiles))
            __syncthreads();
        if (!gridBarrier(p.bar, wholeGrid())) return fail(p);
    }
    if (first > 0)
    {
        if (vload(*p.error)) return;
        for (u32 t = blockIdx.x; t < p.numTiles; t += gridDim.x)
        {
            __syncthreads();
            repairSystemTile<kTile>(p.r, sm.repair, u32(first), p.tiles, p.f.systems, t);
        }
        if (!gridBarrier(p.bar, wholeGrid())) return fail(p);
        const u32 runs = vload(p.r.ctl->longRuns);
        if (runs)
        {
            sort::sortLongRuns(p.r, sm.longRun, first, runs, wholeGrid());
            if (!gridBarrier(p.bar, wholeGrid())) return fail(p);
        }
    }
    activeAndSample<true>(p.f, p.sample, p.ns, size_t(blockIdx.x) * blockDim.x + threadIdx.x,
                          size_t(gridDim.x) * blockDim.x);
}

}  // namespace forest
}  // namespace aot
