// levelbuild.cuh -- device kernels of the converged octree build.
//
// The reference builds an octree from the root by rounds of split/merge
// decisions until a round changes nothing (rebalanceBuild, octree.cu:159-180;
// calculateNodeOp, octree_rebalance.cuh:174-249).  The decision value of a
// cell -- its particle count (LeafCount) or its near-field count NF = count x
// population of the 27 periodic same-level cells around it (NFCount,
// octree_rebalance.cuh:579-634) -- depends only on the particles, and it
// never grows from a cell to its children.  So the tree the rounds converge
// to is unique: a cell is an internal node exactly when its value exceeds the
// bucket and its level is below 21.  This file builds that tree one level at
// a time, without the rounds:
//   expand    the internal cells ("units") of level l get the begin indices
//             of their 8 children in the sorted keys (and, for NFCount, the
//             8 child counts as bytes);
//   nearField NFCount: the 27 cells around each level-l unit, from those
//             around its parent, and from their child counts the near-field
//             counts of the unit's children;
//   classify  the children whose value exceeds the bucket become the units of
//             level l + 1 (slots taken by warp-aggregated atomics); the
//             others are leaves of the tree (with the near field, or with
//             expand where the value is the count);
//   subtree, place: subtree leaf counts bottom-up, then every leaf's
//             position in the cornerstone array top-down.
// A LeafCount build is one launch by team (leafBuildKernel, grid_barrier.cuh):
// a unit's counts are differences of its begins, so expand and classify are
// one step (growUnits) with a grid barrier per level.  An NFCount build has two launches
// per level, and one each for the subtree counts and the placement.
//
// The capacity the reference ends with depends on how many leaves each round
// proposed (resizeWithHeadroom history, octree.cu:159-180 and 453-457).  That
// history follows from the same cells: the rounds start at the root; a leaf
// whose value exceeds the bucket splits in the next round by 1-4 levels at
// once (the level jump of calculateNodeOp), and a group of 8 leaves whose
// parent does not exceed it merges.  Call a cell reached by a split "landed"
// and the levels a split spans its "region".  A landed cell arrives at round
// a; if it is an internal node it splits at once, and its region's 8^k cells
// arrive at round a + 1; every leaf f of the final tree in that region, at
// relative depth j <= k, is then represented by its 8^(k-j) descendants at
// the landing level, which merge up one level per round, so f stands for
// 8^max(0, k - (t - a - 1) - j) leaves at round t >= a + 1.  Classify
// counts the final leaves per (a, k, j) and the landed internal nodes
// per round; the host sums the leaf counts of every round from them.
#pragma once

#include "grid_barrier.cuh"
#include "radix_sort.cuh"
#include "rebalance.cuh"

namespace aot
{
namespace lb
{
constexpr int kThreads = 256;
constexpr u32 kLeaf = 0xffffffffu;     // child slot: the child is a leaf
constexpr int kArrivals = 32;          // arrival rounds tracked (>= kOctLevels + 2)
constexpr int kJumps = 5;              // split depth k = 1..4
constexpr int kContribBins = kArrivals * kJumps * kJumps;
constexpr int kRow = rb::kGroupRow;    // unit row: key (2 words), 9 child begins, region word

// Device control block of one build.
struct Control
{
    u32 levelStart[kOctLevels + 2];
    u32 levelCount[kOctLevels + 2];
    int overflow;       // the unit arena is too small
    int late;           // an arrival round beyond the tracked ones
    int error;          // a bounded wait gave up
    int placeOverflow;  // the tree has more leaves than the cornerstone buffers hold
    GridBarrier bar;    // of the one-launch build, or of the placement
    u32 leaves;         // leaves of the tree
    u32 active;         // active particles
    int stateError;     // DeviceState::error
};

// The unit arena: units of all levels, level l at
// [levelStart[l], levelStart[l] + levelCount[l]).
struct Arena
{
    u32 *rows;       // [cap][kRow]
    u32 *val;        // [cap][8] value of each child (NF or count)
    u32 *child;      // [cap][8] unit index of an internal child, or kLeaf; units of a standing tree: a leaf's
                     // index | kLeafRef (LeafCount: by digit, NFCount: by octant)
    u64 *sub;        // [cap] leaves counted below the unit | children to come << 56
    u32 *offset;     // [cap] cornerstone index of the unit's first leaf (kPending before it is known)
    u32 *nbr;        // NFCount: [cap][27] the cells around each unit (nbrRef)
    u32 *parent;     // [cap] parent unit * 8 + the unit's place in its child slots (batch of trees: kLeaf for a root)
    u64 *rec;        // NFCount: [cap] child counts of a unit, a byte per octant (kBigRec: one does not fit)
    u32 *usys;       // batch of trees: [cap] the tree (system) of each unit
    u32 *sysRoot;    // batch of trees: [systems] each system's root unit, or kLeaf
    Control *ctl;
    unsigned long long *contrib;  // [kArrivals][kJumps][kJumps] final leaves per (a, k, j)
    unsigned long long *landed;   // [kArrivals] internal nodes landing in round t
    u32 cap;
};

// Region word of a unit, describing the region its children belong to:
// arrival round of the region's landed cell (8 bits), that cell's level
// (5 bits) and the region's depth k (3 bits).
__host__ __device__ __forceinline__ u32 regionWord(u32 a, u32 level, u32 k) { return a | (level << 8) | (k << 16); }
__device__ __forceinline__ u32 regionArrival(u32 w) { return w & 0xffu; }
__device__ __forceinline__ u32 regionLevel(u32 w) { return (w >> 8) & 0x1fu; }
__device__ __forceinline__ u32 regionDepth(u32 w) { return (w >> 16) & 7u; }
// The same word also holds the unit's own level (bits 19-23) and the curve
// state that orders its children (bits 24-29, Hilbert).
__host__ __device__ __forceinline__ u32 withUnit(u32 region, u32 level, u32 state)
{
    return (region & 0x7ffffu) | (level << 19) | (state << 24);
}
__device__ __forceinline__ u32 unitLevelOf(u32 w) { return (w >> 19) & 0x1fu; }
__device__ __forceinline__ u32 unitStateOf(u32 w) { return (w >> 24) & 0x3fu; }

// A cell around a unit, at the unit's level: a unit index when the cell is an
// internal node, else kLeafRef | (parent unit * 8 + octant) naming the leaf
// of the tree that holds the cell (the cell itself or a coarser leaf).
constexpr u32 kLeafRef = 0x80000000u;
// Child counts of which one is 255 or more.
constexpr u64 kBigRec = ~u64(0);
// A unit's first leaf is not known yet.
constexpr u32 kPending = 0xffffffffu;
constexpr int kSubShift = 56;
constexpr unsigned kPlaceSpins = 1u << 22;  // polls of a parent's placement

// Levels a leaf of value x at level m splits by (calculateNodeOp,
// octree_rebalance.cuh:188-249: 8, 64, 512 or 4096 children), given that it
// splits (x > bucket, m < 21).  LeafCount compares with 32-bit products of
// the bucket, NFCount with 64-bit ones.
__host__ __device__ __forceinline__ u32 splitDepth(bool nf, u32 x, u32 bucket, unsigned m)
{
    if (nf)
    {
        const u64 c = x, b = bucket;
        if (c > b * 262144 && m + 3 < kOctLevels) return 4;
        if (c > b * 4096 && m + 2 < kOctLevels) return 3;
        if (c > b * 64 && m + 1 < kOctLevels) return 2;
        return 1;
    }
    if (x > bucket * 512u && m + 3 < kOctLevels) return 4;
    if (x > bucket * 64u && m + 2 < kOctLevels) return 3;
    if (x > bucket * 8u && m + 1 < kOctLevels) return 2;
    return 1;
}

__device__ __forceinline__ u64 rowKey(const u32 *row) { return (u64(row[1]) << 32) | row[0]; }

// The root: a unit at level 0 when its value exceeds the bucket (NF of the
// root: 27 x count^2, clamped, octree.cu:23-38), else the whole tree is the
// root leaf, written straight to the cornerstone buffers.
// One warp: the active count by a warp-wide search, then lane 0.
__device__ __forceinline__ void rootUnit(const Arena &a, const rb::TreeBufs &tb, const u64 *P, size_t n, unsigned bucket,
                                         bool nf)
{
    DeviceState *st = tb.st;
    const unsigned active = n ? warpLowerBound(P, 0, u32(n), kMaxKey, int(threadIdx.x & 31)) : 0u;
    if (threadIdx.x != 0) return;
    const u64 sq = u64(active) * active;
    const u32 nfRoot = sq > 0xffffffffull / 27ull ? 0xffffffffu : u32(27ull * sq);
    const u32 x = nf ? nfRoot : active;
    const int err = st->error;
    *st = DeviceState{};
    st->error = err;
    st->numActiveParticles = active;
    Control &c = *a.ctl;
    c.levelStart[0] = 0;
    if (x > bucket)
    {
        u32 *row = a.rows;
        row[0] = 0;
        row[1] = 0;
        row[2] = 0;
        row[10] = active;
        row[11] = withUnit(regionWord(0, 0, splitDepth(nf, x, bucket, 0)), 0, kHilbertStart);
        c.levelCount[0] = 1;
        a.offset[0] = 0;
        if (nf)
        {
            // every cell around the root is the root (periodic wrap)
            for (int q = 0; q < 27; ++q) a.nbr[q] = 0;
        }
        st->numLeaves = 0;  // set when the tree is placed
    }
    else
    {
        c.levelCount[0] = 0;
        tb.K[0][0] = 0;
        tb.K[0][1] = kMaxKey;
        tb.B[0][0] = 0;
        tb.B[0][1] = active;
        tb.NF[0][0] = nf ? nfRoot : 0u;
        tb.N[0][0] = active;
        st->numLeaves = 1;
    }
}

static __global__ void rootKernel(Arena a, rb::TreeBufs tb, const u64 *P, size_t n, unsigned bucket)
{
    rootUnit(a, tb, P, n, bucket, true);
}

// Lower bounds of the 7 inner child boundaries key + (d + 1) * cr of a unit
// whose keys are P[lo, hi), searched side by side (7 independent loads per
// step): first among the sampled keys (every 32nd key, a small array that
// stays in L2), then in the window of at most 31 keys the sample leaves.
__device__ __forceinline__ void innerBegins(const KeyIndex &idx, u32 lo, u32 hi, u64 key, u64 cr, u32 (&b)[7])
{
    const u32 jA = (lo + kSampleStride - 1) >> kSampleShift, jB = (hi + kSampleStride - 1) >> kSampleShift;
    u32 len[7];
#pragma unroll
    for (int d = 0; d < 7; ++d)
    {
        b[d] = jA;
        len[d] = jB > jA ? jB - jA : 0;
    }
    for (;;)  // first sample >= target among samples jA..jB-1
    {
        u32 live = 0;
#pragma unroll
        for (int d = 0; d < 7; ++d) live |= len[d];
        if (!live) break;
#pragma unroll
        for (int d = 0; d < 7; ++d)
        {
            if (len[d])
            {
                const u32 half = len[d] >> 1;
                const bool less = __ldg(idx.sample + b[d] + half) < key + u64(d + 1) * cr;
                b[d] = less ? b[d] + half + 1 : b[d];
                len[d] = less ? len[d] - half - 1 : half;
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 7; ++d)
    {
        // the answer lies after the last sample below the target and at or
        // before the first one at or above it
        const u32 wlo = b[d] > jA ? ((b[d] - 1) << kSampleShift) + 1 : lo;
        const u32 whi = b[d] < jB ? (b[d] << kSampleShift) : hi;
        len[d] = whi > wlo ? whi - wlo : 0;  // empty unless the keys are sorted (a failed sort stays in bounds)
        b[d] = wlo;
    }
    for (;;)
    {
        u32 live = 0;
#pragma unroll
        for (int d = 0; d < 7; ++d) live |= len[d];
        if (!live) break;
#pragma unroll
        for (int d = 0; d < 7; ++d)
        {
            if (len[d])
            {
                const u32 half = len[d] >> 1;
                const bool less = __ldg(idx.keys + b[d] + half) < key + u64(d + 1) * cr;
                b[d] = less ? b[d] + half + 1 : b[d];
                len[d] = less ? len[d] - half - 1 : half;
            }
        }
    }
}

// Levels with at most this many units expand by warps (a warp per inner
// child boundary); the chains of dependent loads of the per-thread searches
// dominate there, and the keys of a unit span most of the array.
constexpr u32 kWideUnits = 4096;
// Up to this many units, a lane per inner boundary (8 lanes per unit): more
// searches in flight where the units are too few to fill the GPU one thread
// each.
constexpr u32 kLaneUnits = 1u << 18;

// Lower bound of t among the keys P[lo, hi): first among the sampled keys in
// the range, then in the window of at most 31 keys they leave.
__device__ __forceinline__ u32 boundaryIn(const KeyIndex &idx, u32 lo, u32 hi, u64 t)
{
    const u32 jA = (lo + kSampleStride - 1) >> kSampleShift, jB = (hi + kSampleStride - 1) >> kSampleShift;
    u32 b = jA, len = jB > jA ? jB - jA : 0;
    while (len)
    {
        const u32 half = len >> 1;
        const bool less = __ldg(idx.sample + b + half) < t;
        b = less ? b + half + 1 : b;
        len = less ? len - half - 1 : half;
    }
    const u32 wlo = b > jA ? ((b - 1) << kSampleShift) + 1 : lo;
    const u32 whi = b < jB ? (b << kSampleShift) : hi;
    b = wlo;
    len = whi > wlo ? whi - wlo : 0;
    while (len)
    {
        const u32 half = len >> 1;
        const bool less = __ldg(idx.keys + b + half) < t;
        b = less ? b + half + 1 : b;
        len = less ? len - half - 1 : half;
    }
    return b;
}

// The same by a warp: first sampled key >= t among the samples inside [lo, hi),
// then the window of at most 31 keys before it.
__device__ __forceinline__ u32 warpBoundaryIn(const KeyIndex &idx, u32 lo, u32 hi, u64 t, int lane)
{
    const u32 jA = (lo + kSampleStride - 1) >> kSampleShift, jB = (hi + kSampleStride - 1) >> kSampleShift;
    const u32 sIdx = warpLowerBound(idx.sample, jA, jB > jA ? jB : jA, t, lane);
    const u32 wlo = sIdx > jA ? ((sIdx - 1) << kSampleShift) + 1 : lo;
    const u32 whi = sIdx < jB ? (sIdx << kSampleShift) : hi;
    return warpLowerBound(idx.keys, wlo, whi, t, lane);
}

// The children of units: lanes hold a child each, eight to a unit g in digit
// order, of which `valid` ones take part (whole units; all lanes of the warp
// call).  A child whose value x (its keys, or NF: its near-field count) exceeds
// `bucket` below level 21 becomes a unit of level l + 1 (slots by an atomic add
// per warp; the order of a level's units is free: every later step finds them
// through the child and parent links, and the placement follows the digits),
// the others are leaves, counted into the round history by (arrival, depth,
// relative level): of the CTA (sContrib, sLanded) or, Forest, of the unit's
// system.  key and reg: the unit's key and region word; [begin, end): the
// child's keys; next: first unit of level l + 1.  NFCount units keep their
// children by octant (dec, encNext: the curve's tables).
template <bool NF, bool Hilbert, bool Forest>
__device__ __forceinline__ void growChildren(const Arena &a, int l, unsigned bucket, u32 next, u32 g, bool valid, u32 x,
                                             u32 begin, u32 end, u64 key, u32 reg, const unsigned char *dec,
                                             const unsigned char *encNext, u32 *sContrib, u32 *sLanded)
{
    Control &c = *a.ctl;
    const unsigned m = unsigned(l) + 1;
    const int lane = threadIdx.x & 31, d = lane & 7;
    const bool high = valid && x > bucket && m < kOctLevels;
    const unsigned ballot = __ballot_sync(0xffffffffu, high);
    u32 base = 0;
    if (lane == 0 && ballot) base = atomicAdd(&c.levelCount[l + 1], u32(__popc(ballot)));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (!valid) return;
    const u32 aR = regionArrival(reg), lR = regionLevel(reg), kR = regionDepth(reg);
    const u32 j = m - lR;  // 1 <= j <= kR
    const u32 nHigh = u32(__popc((ballot >> (lane & 24)) & 0xffu));
    const u32 sys = Forest ? a.usys[g] : 0u;
    const u32 state = Hilbert ? unitStateOf(reg) : 0u;
    const u32 oct = Hilbert ? u32(dec[state * 8 + d]) : u32(d);
    u32 slot = kLeaf;
    if (high)
    {
        const u32 gc = next + base + u32(__popc(ballot & sort::laneMaskLt()));
        if (gc < a.cap)
        {
            u32 creg = reg;
            // a landed internal node: a leaf in round aR + 1, splitting at once
            if (j == kR) creg = regionWord(min(aR + 1, u32(kArrivals) - 1), m, splitDepth(NF, x, bucket, m));
            if constexpr (Forest) a.usys[gc] = sys;
            a.parent[gc] = g * 8 + oct;
            a.offset[gc] = kPending;
            const u64 ck = key + u64(d) * octRange(m);
            uint4 *crow = reinterpret_cast<uint4 *>(a.rows + size_t(gc) * kRow);
            crow[0] = make_uint4(u32(ck), u32(ck >> 32), begin, 0u);
            crow[2] = make_uint4(0u, 0u, end, withUnit(creg, m, Hilbert ? u32(encNext[state * 8 + oct]) : u32(kHilbertStart)));
            slot = gc;
        }
        else
        {
            c.overflow = 1;
        }
    }
    a.child[size_t(g) * 8 + oct] = slot;
    if (d != 0) return;
    a.sub[g] = (u64(nHigh) << kSubShift) | (8u - nHigh);
    const u32 bin = (aR * kJumps + kR) * kJumps + j;
    if (nHigh < 8)
    {
        if (Forest) atomicAdd(a.contrib + size_t(sys) * kContribBins + bin, 8ull - nHigh);
        else atomicAdd(&sContrib[bin], 8u - nHigh);
    }
    if (j == kR && nHigh)
    {
        if (aR + 2 >= u32(kArrivals)) c.late = 1;
        else if (Forest) atomicAdd(a.landed + size_t(sys) * kArrivals + aR + 1, (unsigned long long)nHigh);
        else atomicAdd(&sLanded[aR + 1], nHigh);
    }
}

// Expand and classify of a LeafCount level in one step, by a team: on
// levels of few units a CTA per unit, a warp per inner child boundary (sEnds:
// 7 words of the CTA), else a lane per child.
template <bool Forest>
__device__ __forceinline__ void growUnits(const Arena &a, const KeyIndex &idx, int l, unsigned bucket, u32 start,
                                          u32 count, const Team &team, u32 *sEnds, u32 *sContrib, u32 *sLanded)
{
    const u32 next = start + count;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u64 cr = octRange(unsigned(l) + 1);
    if (team.rank == 0 && threadIdx.x == 0) a.ctl->levelStart[l + 1] = next;
    if (count <= kWideUnits)
    {
        static_assert(kThreads / 32 >= 7, "a warp per inner boundary");
        for (u32 i = team.rank; i < count; i += team.size)
        {
            u32 *row = a.rows + size_t(start + i) * kRow;
            const u32 lo = row[2], hi = row[10], reg = row[11];
            const u64 key = rowKey(row);
            if (warp < 7)
            {
                const u32 r = warpBoundaryIn(idx, lo, hi, key + u64(warp + 1) * cr, lane);
                if (lane == 0)
                {
                    row[3 + warp] = r;
                    sEnds[warp] = r;
                }
            }
            __syncthreads();
            if (warp == 0)
            {
                const int d = lane & 7;
                const u32 b = d ? sEnds[d - 1] : lo, e = d < 7 ? sEnds[d] : hi;
                growChildren<false, false, Forest>(a, l, bucket, next, start + i, lane < 8, e - b, b, e, key, reg, nullptr,
                                                   nullptr, sContrib, sLanded);
            }
            __syncthreads();
        }
        return;
    }
    const size_t total = size_t(count) * 8;
    for (size_t e0 = size_t(team.rank) * kThreads + warp * 32; e0 < total; e0 += size_t(team.size) * kThreads)
    {
        const size_t e = e0 + lane;
        const bool valid = e < total;
        const u32 g = start + u32(valid ? e >> 3 : 0);
        const int d = lane & 7;
        u32 *row = a.rows + size_t(g) * kRow;
        const u32 lo = row[2], hi = row[10], reg = row[11];
        const u64 key = rowKey(row);
        u32 end = hi;
        if (valid && d < 7)
        {
            end = boundaryIn(idx, lo, hi, key + u64(d + 1) * cr);
            row[3 + d] = end;
        }
        const u32 prev = __shfl_up_sync(0xffffffffu, end, 1, 8);
        const u32 begin = d ? prev : lo;
        growChildren<false, false, Forest>(a, l, bucket, next, g, valid, end - begin, begin, end, key, reg, nullptr, nullptr,
                                           sContrib, sLanded);
    }
}

// 9 child begins of the units of level l of an NFCount build: one thread per
// unit (the 7 inner ones by innerBegins), one lane per inner boundary on
// levels of fewer units, one warp per inner boundary on levels of few units;
// and the units' child counts as bytes (not on levels of few units, whose
// counts do not fit and which do without), by octant: dec[state * 8 + digit]
// for the Hilbert curve.
template <bool Hilbert>
__device__ __forceinline__ void expandUnits(const Arena &a, const KeyIndex &idx, int l, u32 start, u32 count, u32 rank,
                                            u32 size, const unsigned char *dec)
{
    const u64 cr = octRange(unsigned(l) + 1);
    const int lane = threadIdx.x & 31;
    if (count <= kWideUnits)
    {
        for (u32 w = rank >> 5; w < count * 7; w += size >> 5)
        {
            const u32 i = w / 7, d = w - i * 7;
            u32 *row = a.rows + size_t(start + i) * kRow;
            const u32 r = warpBoundaryIn(idx, row[2], row[10], rowKey(row) + u64(d + 1) * cr, lane);
            if (lane == 0) row[3 + d] = r;
        }
        return;
    }
    if (count <= kLaneUnits)
    {
        for (u32 e = rank; e < count * 8; e += size)  // the 8 lanes of a unit together
        {
            const u32 i = e >> 3, d = e & 7;
            u32 *row = a.rows + size_t(start + i) * kRow;
            const u32 lo = row[2], hi = row[10];
            u32 end = hi;  // of child d
            if (d < 7)
            {
                end = boundaryIn(idx, lo, hi, rowKey(row) + u64(d + 1) * cr);
                row[3 + d] = end;
            }
            const unsigned group = 0xffu << (lane & 24);
            const u32 prev = __shfl_up_sync(group, end, 1, 8);
            const u32 cnt = end - (d ? prev : lo);
            const bool big = __any_sync(group, cnt >= 255u);
            const u32 oct = Hilbert ? u32(dec[unitStateOf(row[11]) * 8 + d]) : d;
            reinterpret_cast<unsigned char *>(a.rec + (start + i))[oct] = big ? 255 : (unsigned char)cnt;
        }
        return;
    }
    for (u32 i = rank; i < count; i += size)
    {
        u32 *row = a.rows + size_t(start + i) * kRow;
        u32 b[7];
        const u32 lo = row[2], hi = row[10];
        innerBegins(idx, lo, hi, rowKey(row), cr, b);
#pragma unroll
        for (int d = 0; d < 7; ++d) row[3 + d] = b[d];
        const u32 st = unitStateOf(row[11]);
        u64 rec = 0;
        bool big = false;
#pragma unroll
        for (int d = 0; d < 8; ++d)
        {
            const u32 cnt = (d < 7 ? b[d] : hi) - (d ? b[d - 1] : lo);
            big |= cnt >= 255u;
            const u32 oct = Hilbert ? u32(dec[st * 8 + d]) : u32(d);
            rec |= u64(cnt & 0xffu) << (8 * oct);
        }
        a.rec[start + i] = big ? kBigRec : rec;
    }
}

template <bool Hilbert>
static __global__ void __launch_bounds__(kThreads) expandKernel(Arena a, KeyIndex idx, int l)
{
    __shared__ __align__(4) unsigned char sDec[48 * 8];
    const Control &c = *a.ctl;
    if (c.overflow | c.late | c.error) return;
    if constexpr (Hilbert)
    {
        copyTable(sDec, gHilbert.decOct);
        __syncthreads();
    }
    expandUnits<Hilbert>(a, idx, l, c.levelStart[l], c.levelCount[l], blockIdx.x * blockDim.x + threadIdx.x,
                              gridDim.x * blockDim.x, sDec);
}

// Near-field counts of the children of the level-l units, a warp per
// kUnitBatch units at a time.
//
// The 27 cells around a unit come from those around its parent U: the cell at
// offset (dx, dy, dz) of the unit (octant o in U) is child o' of the cell at
// offset floor((o + d) / 2) around U, o' = (o + d) mod 2 per axis.  That cell
// is a unit (the child of a unit around U, if internal) or lies in a leaf: a
// leaf child of a unit around U, or the leaf that already holds U's cell.
// (Children are kept by octant, so no curve state is needed on the way.)
//
// The children of those 27 cells form a 6 x 6 x 6 block of cells, a unit's
// own children in its middle; each child's population is its 3 x 3 x 3
// sub-block's.  Cells that are units bring their 8 child counts as one 8-byte
// record, a byte per octant; those in a leaf (one of eight at 16Mi Plummer
// particles, a few keys each) have the leaf's keys counted.  A lane sums two
// children from the record words by byte dot products.  (Levels of few units
// have no records; theirs are made from the rows.)  Units around which a
// count does not fit a byte take the path by rows (nearFieldByRows).
//
// Before: the 27 cells by a kernel of their own, a 48-byte row of begin
// indices and a curve state per cell here, scattered into 4 x 4 x 4 blocks of
// words that eight lanes a unit summed: 387 us (beside the expansion) and
// 786 us for the 1.8 M units of a 16Mi Plummer build, bound by L1 and
// shared memory (79 %).

// Per-warp scratch of the path by rows: the units in flight.
struct RowScratch
{
    u64 pStart[rb::kUnitBatch];
    int childState[rb::kUnitBatch];
    rb::UnitBlocks block;
    unsigned long long pop[rb::kUnitBatch];  // population of the 27 cells around the unit
    u32 slowRef[rb::kUnitBatch * 27];
    unsigned short slowItem[rb::kUnitBatch * 27];
    int nSlow;
};
// Per-warp scratch of the path by records.
struct RecScratch
{
    u64 rec[rb::kUnitBatch * 27];  // child counts of the cells around the units: [unit][27]
    u32 parent[rb::kUnitBatch];
    u32 slowRef[rb::kUnitBatch * 27];
    unsigned short slowItem[rb::kUnitBatch * 27];
};
union NearScratch
{
    RowScratch rows;
    RecScratch recs;
};
struct alignas(4) NearTables
{
    unsigned char enc[48 * 8], next[48 * 8], dec[48 * 8];
    unsigned char step[8 * 27];  // [octant of the unit][offset]: offset around the parent << 3 | octant there
};

// Key range of the leaf `ref` (kLeafRef removed) and, for a cell at level l
// and offset q around the unit with key start `pStart` that lies in it, the
// cell's key and curve state.
template <bool Hilbert>
__device__ __forceinline__ void leafCell(const Arena &a, const NearTables &t, u32 ref, int l, u64 pStart, int q, u32 &lo,
                                         u32 &hi, u64 &qKey, int &qState)
{
    const u32 o = ref & 7u;
    const u32 *row = a.rows + size_t(ref >> 3) * kRow;
    // the whole row at once: its words one after the other were three round
    // trips (with four keys in flight in countedRec: 16Mi near field 586 to 542 us)
    const uint4 *r4 = reinterpret_cast<const uint4 *>(row);
    const uint4 r0 = r4[0], r1 = r4[1], r2 = r4[2];
    const u32 reg = r2.w, st = unitStateOf(reg);
    const u32 d = Hilbert ? u32(t.enc[st * 8 + o]) : o;
    const u32 b[rb::kGroupBegins] = {r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, r2.z};
    lo = b[0];
    hi = b[1];
#pragma unroll
    for (u32 k = 1; k < 8; ++k)
    {
        lo = d == k ? b[k] : lo;
        hi = d == k ? b[k + 1] : hi;
    }
    if (unitLevelOf(reg) + 1 == unsigned(l))
    {
        // the leaf is the cell itself: child o of its parent unit
        qKey = ((u64(r0.y) << 32) | r0.x) + u64(d) * octRange(unsigned(l));
        qState = Hilbert ? int(t.next[st * 8 + o]) : kHilbertStart;
    }
    else if (lo < hi)
    {
        const rb::CellPath path = rb::decodeCell<Hilbert>(pStart, unsigned(l), t.next, t.dec);
        qKey = rb::neighbourCellOf<Hilbert>(path, pStart, unsigned(l), q, qState, t.enc, t.next);
    }
    else
    {
        qKey = 0;
        qState = kHilbertStart;
    }
}

// A unit's child counts as bytes, from its row.
template <bool Hilbert>
__device__ __forceinline__ u64 rowRec(const u32 *row, const unsigned char *dec)
{
    const uint4 *r4 = reinterpret_cast<const uint4 *>(row);
    const uint4 r0 = r4[0], r1 = r4[1], r2 = r4[2];
    const u32 b[rb::kGroupBegins] = {r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, r2.z};
    const u32 st = unitStateOf(r2.w);
    u64 rec = 0;
    bool big = false;
#pragma unroll
    for (int d = 0; d < 8; ++d)
    {
        const u32 cnt = b[d + 1] - b[d];
        big |= cnt >= 255u;
        rec |= u64(cnt & 0xffu) << (8 * (Hilbert ? u32(dec[st * 8 + d]) : u32(d)));
    }
    return big ? kBigRec : rec;
}

// Where the near-field counts go.  Build: into the units' values.  Else (the
// units of a standing tree) to the leaves, with the group flags.
struct NearOut
{
    u32 *NF;
    u8 *G;
    unsigned bucket;
};

// May the 8 leaf children of a unit with `own` particles and `pop` in the 27
// cells around it merge (computeGroupCanMergeKernel, octree_rebalance.cuh:636-700)?
__device__ __forceinline__ u8 canMerge(u64 own, u64 pop, unsigned bucket)
{
    // (pop is below 27 x 2^32: only a product of 37 and 32 bits or more can pass 2^64)
    return own == 0 || (pop <= u64(bucket) && own * pop <= u64(bucket)) ? 1 : 0;
}

// The units [first, first + nb) of level l by rows: any counts.
template <bool Hilbert, bool Build>
__device__ __noinline__ void nearFieldByRows(const Arena &a, const KeyIndex &idx, int l, u32 first, int nb, RowScratch &w,
                                             const NearTables &t, const NearOut &out)
{
    const unsigned m = unsigned(l) + 1;
    const int lane = threadIdx.x & 31;
    const unsigned ltMask = (1u << lane) - 1u;
    if (lane < nb)
    {
        // the cell's path is decoded only where a neighbour lies inside a
        // coarser leaf (phase B); the children's curve state is in the row
        const u32 *row = a.rows + size_t(first + u32(lane)) * kRow;
        w.pStart[lane] = rowKey(row);
        w.childState[lane] = int(unitStateOf(row[11]));
    }
    if (lane == 0) w.nSlow = 0;
    if (!Build && lane < nb) w.pop[lane] = 0;
    __syncwarp();
    // phase A: (unit, Q) pairs over the lanes; a Q that is a unit gives
    // its children's counts from its row
    const int items = nb * 27;
    for (int ib = 0; ib < items; ib += 32)
    {
        const int it = ib + lane;
        const int u = it / 27, q = it - (it / 27) * 27;
        u32 ref = 0;
        bool slow = false;
        if (it < items)
        {
            ref = a.nbr[size_t(first) * 27 + it];
            if (ref & kLeafRef)
            {
                slow = true;
            }
            else
            {
                const uint4 *vr = reinterpret_cast<const uint4 *>(a.rows + size_t(ref) * kRow);
                const uint4 r0 = vr[0], r1 = vr[1], r2 = vr[2];
                const u32 gb[rb::kGroupBegins] = {r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, r2.x, r2.y, r2.z};
                rb::childrenFromPacked<Hilbert>(gb, q, int(unitStateOf(r2.w)), w.block[u]);
                if (!Build) atomicAdd(&w.pop[u], (unsigned long long)(gb[8] - gb[0]));
            }
        }
        const unsigned slowMask = __ballot_sync(0xffffffffu, slow);
        if (slow)
        {
            const int k = w.nSlow + __popc(slowMask & ltMask);
            w.slowRef[k] = ref;
            w.slowItem[k] = (unsigned short)it;
        }
        __syncwarp();
        if (lane == 0) w.nSlow += __popc(slowMask);
        __syncwarp();
    }
    // phase B: Q in a leaf: its children counted among the leaf's keys
    const int nSlow = w.nSlow;
    for (int k = lane; k < nSlow; k += 32)
    {
        const int it = w.slowItem[k];
        const int u = it / 27, q = it - u * 27;
        u32 lo, hi;
        u64 qKey;
        int qState;
        leafCell<Hilbert>(a, t, w.slowRef[k] & ~kLeafRef, l, w.pStart[u], q, lo, hi, qKey, qState);
        u32 begins[rb::kGroupBegins];
        rb::childBeginsWithin(idx.keys, lo, hi, qKey, m, begins);
        rb::childrenFromPacked<Hilbert>(begins, q, qState, w.block[u]);
        if (!Build) atomicAdd(&w.pop[u], (unsigned long long)(begins[8] - begins[0]));
    }
    __syncwarp();
    // phase C: the 8 children of each unit, two per lane
    for (int e = lane; e < nb * 8; e += 32)
    {
        const int u = e >> 3, d = e & 7;
        const u32 g = first + u32(u);
        const u32 *row = a.rows + size_t(g) * kRow;
        const u32 cnt = row[2 + d + 1] - row[2 + d];
        const unsigned o = Hilbert ? unsigned(t.dec[w.childState[u] * 8 + d]) : unsigned(d);
        u32 nf = 0;
        if (cnt)
        {
            const u32 *sub = w.block[u] + (o >> 2) * 16 + ((o >> 1) & 1u) * 4 + (o & 1u);
            u64 pop = 0;
            if (m > 1)
            {
                u32 p32 = 0;
#pragma unroll
                for (int x = 0; x < 3; ++x)
#pragma unroll
                    for (int y = 0; y < 3; ++y)
#pragma unroll
                        for (int z = 0; z < 3; ++z) p32 += sub[x * 16 + y * 4 + z];
                pop = p32;
            }
            else
            {
                // level 1: the periodic wrap repeats cells, the sum may exceed 2^32
                for (int x = 0; x < 3; ++x)
                    for (int y = 0; y < 3; ++y)
                        for (int z = 0; z < 3; ++z) pop += sub[x * 16 + y * 4 + z];
            }
            const u64 v = u64(cnt) * pop;
            nf = v > 0xffffffffull ? 0xffffffffu : u32(v);
        }
        if constexpr (Build)
        {
            a.val[size_t(g) * 8 + d] = nf;
        }
        else
        {
            const u32 ch = a.child[size_t(g) * 8 + o];
            if (ch & kLeafRef) out.NF[ch & ~kLeafRef] = nf;
            // the 8 lanes of a unit together: all its children leaves?
            const unsigned group = 0xffu << (lane & 24);
            if (__all_sync(group, (ch & kLeafRef) != 0) && d == 0)
                out.G[ch & ~kLeafRef] = canMerge(row[10] - row[2], w.pop[u], out.bucket);
        }
    }
    __syncwarp();
}

// Child counts of the level-l cell [qKey, qKey + 8 cr) among the keys
// P[lo, hi) (cr: its children's range), a byte per octant, or kBigRec.
template <bool Hilbert>
__device__ __forceinline__ u64 countedRec(const u64 *P, u32 lo, u32 hi, u64 qKey, int qState, int l,
                                          const unsigned char *dec)
{
    if (hi - lo >= 255u) return kBigRec;
    const unsigned shift = 3u * (kOctLevels - unsigned(l) - 1);
    u64 rec = 0;
    for (u32 k = lo; k < hi; k += 4)  // four keys in flight
    {
        u64 key[4];
#pragma unroll
        for (u32 i = 0; i < 4; ++i) key[i] = __ldg(P + min(k + i, hi - 1));
#pragma unroll
        for (u32 i = 0; i < 4; ++i)
        {
            const u64 d = (key[i] - qKey) >> shift;  // 8 or more: outside the cell
            if (k + i < hi && d < 8) rec += u64(1) << (8 * (Hilbert ? unsigned(dec[qState * 8 + int(d)]) : unsigned(d)));
        }
    }
    return rec;
}

// Build: the values of a build's units, and with them the units of the next
// level and the round history (growChildren; a launch per level that read the
// rows and values back took 178 us at 16Mi and 48 us in 11 launches at 300k);
// else the near-field counts and group flags of the leaves of a standing tree
// (treeUnitsKernel).
template <bool Hilbert, bool Build>
static __global__ void __launch_bounds__(kThreads, 4)
    nearFieldKernel(Arena a, KeyIndex idx, int l, rb::TreeBufs tb, unsigned bucket)
{
    using rb::kUnitBatch;
    __shared__ NearTables t;
    __shared__ NearScratch sWarp[kThreads / 32];
    __shared__ u32 sContrib[Build ? kContribBins : 1], sLanded[Build ? kArrivals : 1];
    Control &c = *a.ctl;
    if (c.overflow | c.late | c.error) return;  // (set by this level's CTAs too: what is left out then does not matter)
    const u32 start = c.levelStart[l], count = c.levelCount[l];
    if (Build && blockIdx.x == 0 && threadIdx.x == 0) c.levelStart[l + 1] = start + count;
    NearOut out{};
    if constexpr (!Build)
    {
        const int active = tb.st->activeBuffer;
        out = {tb.nf(active), tb.g(active), bucket};
    }
    if (count <= blockIdx.x) return;  // no units for this CTA
    if constexpr (Hilbert)
    {
        copyTable(t.enc, gHilbert.enc);
        copyTable(t.next, gHilbert.encNext);
        copyTable(t.dec, gHilbert.decOct);
    }
    for (int k = threadIdx.x; k < 8 * 27; k += blockDim.x)
    {
        const int o = k / 27, q = k - o * 27;
        const int tx = (o >> 2) + q % 3 - 1, ty = ((o >> 1) & 1) + (q / 3) % 3 - 1, tz = (o & 1) + q / 9 - 1;
        const int qp = ((tx + 2) / 2) + 3 * ((ty + 2) / 2) + 9 * ((tz + 2) / 2);  // offset around the parent
        t.step[k] = (unsigned char)(qp << 3 | ((tx & 1) << 2) | ((ty & 1) << 1) | (tz & 1));
    }
    if constexpr (Build)
    {
        for (int k = threadIdx.x; k < kContribBins; k += kThreads) sContrib[k] = 0;
        if (threadIdx.x < kArrivals) sLanded[threadIdx.x] = 0;
    }
    __syncthreads();
    constexpr int kRounds = (kUnitBatch * 27 + 31) / 32;
    const int lane = threadIdx.x & 31;
    const unsigned ltMask = (1u << lane) - 1u;
    const bool byRecs = count > kWideUnits;
    RecScratch &w = sWarp[threadIdx.x >> 5].recs;
    const u32 warpsTotal = gridDim.x * (blockDim.x / 32);
    // levels that do not fill the warps' batches: fewer units per warp, shorter chains
    const u32 per = min(u32(kUnitBatch), (count + warpsTotal - 1) / warpsTotal);
    const u32 w0 = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;  // (a level of few units spreads over the SMs)
    // the units [first, first + nb), whose values are written, four at a time
    const auto classify = [&](u32 first, int nb) {
        for (int e = lane; e < ((nb * 8 + 31) & ~31); e += 32)
        {
            const bool valid = e < nb * 8;
            const u32 g = first + u32(valid ? e >> 3 : 0);
            const int d = e & 7;
            const u32 *row = a.rows + size_t(g) * kRow;
            growChildren<true, Hilbert, false>(a, l, bucket, start + count, g, valid, a.val[size_t(g) * 8 + d], row[2 + d],
                                               row[3 + d], rowKey(row), row[11], t.dec, t.next, sContrib, sLanded);
        }
        __syncwarp();
    };
    for (u32 base = w0 * per; base < count; base += warpsTotal * per)
    {
        const int nb = int(min(per, count - base)), items = nb * 27;
        const u32 first = start + base;
        // the cells around the units, (unit, cell) pairs over the lanes: all
        // loads of a step in flight together
        u32 ref[kRounds];
        if (l > 0)
        {
            if (lane < nb) w.parent[lane] = a.parent[first + u32(lane)];
            __syncwarp();
            u32 oct[kRounds];
#pragma unroll
            for (int i = 0; i < kRounds; ++i)
            {
                const int it = i * 32 + lane, u = it / 27, q = it - u * 27;
                ref[i] = kLeafRef;
                oct[i] = 0;
                if (it < items)
                {
                    const u32 p = w.parent[u], step = t.step[(p & 7u) * 27 + q];
                    ref[i] = a.nbr[size_t(p >> 3) * 27 + (step >> 3)];
                    oct[i] = step & 7u;
                }
            }
            u32 ch[kRounds];
#pragma unroll
            for (int i = 0; i < kRounds; ++i)
                ch[i] = ref[i] & kLeafRef ? kLeaf : a.child[size_t(ref[i]) * 8 + oct[i]];  // (kLeafRef is set in kLeaf)
#pragma unroll
            for (int i = 0; i < kRounds; ++i)
            {
                if (!(ref[i] & kLeafRef)) ref[i] = ch[i] & kLeafRef ? kLeafRef | (ref[i] * 8 + oct[i]) : ch[i];
                const int it = i * 32 + lane;
                if (it < items) a.nbr[size_t(first) * 27 + it] = ref[i];
            }
        }
        bool big = false;
        if (!byRecs)
        {
            // without records: counts that cannot fit a byte are told by the units themselves
            const u32 *row = a.rows + size_t(first + u32(lane < nb ? lane : 0)) * kRow;
            big = l == 0 || __any_sync(0xffffffffu, row[10] - row[2] > 8 * 254u);
        }
        if (!big)
        {
            u64 rec[kRounds];
#pragma unroll
            for (int i = 0; i < kRounds; ++i)
            {
                rec[i] = 0;
                if (i * 32 + lane < items && !(ref[i] & kLeafRef))
                    rec[i] = byRecs ? a.rec[ref[i]] : rowRec<Hilbert>(a.rows + size_t(ref[i]) * kRow, t.dec);
            }
            int nSlow = 0;
#pragma unroll
            for (int i = 0; i < kRounds; ++i)
            {
                const int it = i * 32 + lane;
                const bool slow = it < items && (ref[i] & kLeafRef);
                const unsigned slowMask = __ballot_sync(0xffffffffu, slow);
                if (slow)
                {
                    const int k = nSlow + __popc(slowMask & ltMask);
                    w.slowRef[k] = ref[i];
                    w.slowItem[k] = (unsigned short)it;
                }
                else if (it < items)
                {
                    big |= rec[i] == kBigRec;
                    w.rec[it] = rec[i];
                }
                nSlow += __popc(slowMask);
            }
            __syncwarp();
            for (int k = lane; k < nSlow; k += 32)
            {
                const int it = w.slowItem[k], u = it / 27;
                u32 lo, hi;
                u64 qKey;
                int qState;
                leafCell<Hilbert>(a, t, w.slowRef[k] & ~kLeafRef, l, rowKey(a.rows + size_t(first + u32(u)) * kRow),
                                  it - u * 27, lo, hi, qKey, qState);
                const u64 r = countedRec<Hilbert>(idx.keys, lo, hi, qKey, qState, l, t.dec);
                big |= r == kBigRec;
                w.rec[it] = r;
            }
            big = __any_sync(0xffffffffu, big);  // (also: the records are written)
        }
        __syncwarp();
        if (big)
        {
            nearFieldByRows<Hilbert, Build>(a, idx, l, first, nb, sWarp[threadIdx.x >> 5].rows, t, out);
            if constexpr (Build) classify(first, nb);
            continue;
        }
        // Four lanes a unit: lane (x0, y0) sums the children (x0, y0, 0) and
        // (x0, y0, 1).  A record's word holds the cells (y, z) of one x of its
        // cell: bytes (0,0) (0,1) (1,0) (1,1).  The sub-block's y range is the
        // upper half of cell row 0 and row 1 (y0 = 0), or row 1 and the lower
        // half of row 2; its z range likewise.
        const int u = lane >> 2, x0 = (lane >> 1) & 1, y0 = lane & 1;
        if (u < nb)
        {
            const u32 *words = reinterpret_cast<const u32 *>(w.rec + u * 27);
            const u32 g = first + u32(u);
            const u32 rowA = y0 ? 0x01010101u : 0x01010000u;  // bytes of the two cell rows the range takes
            const u32 rowB = y0 ? 0x00000101u : 0x01010101u;
            u32 z0 = 0, z1 = 0;
#pragma unroll
            for (int i = 0; i < 3; ++i)
            {
                const int x = x0 + 1 + i, qx = x >> 1, ox = x & 1;
#pragma unroll
                for (int j = 0; j < 2; ++j)
                {
                    const u32 row = j ? rowB : rowA;
                    const u32 *cell = words + 2 * (qx + 3 * (y0 + j)) + ox;
                    const u32 below = cell[0], middle = cell[18], above = cell[36];
                    const u32 both = __dp4a(middle, row, 0u);
                    z0 += both + __dp4a(below, row & 0x01000100u, 0u);
                    z1 += both + __dp4a(above, row & 0x00010001u, 0u);
                }
            }
            const u32 own = words[2 * 13 + x0] >> (16 * y0);
            const u32 c0 = own & 0xffu, c1 = (own >> 8) & 0xffu;
            const u32 o0 = u32(x0 * 4 + y0 * 2);
            u32 d0 = o0, d1 = o0 + 1;
            if constexpr (Hilbert)
            {
                const u32 st = unitStateOf(a.rows[size_t(g) * kRow + 11]);
                d0 = t.enc[st * 8 + d0];
                d1 = t.enc[st * 8 + d1];
            }
            // near-field counts: at most 254 x 27 x 254
            if constexpr (Build)
            {
                a.val[size_t(g) * 8 + d0] = c0 * z0;
                a.val[size_t(g) * 8 + d1] = c1 * z1;
            }
            else
            {
                const uint2 ch = *reinterpret_cast<const uint2 *>(a.child + size_t(g) * 8 + o0);
                if (ch.x & kLeafRef) out.NF[ch.x & ~kLeafRef] = c0 * z0;
                if (ch.y & kLeafRef) out.NF[ch.y & ~kLeafRef] = c1 * z1;
                // a complete group's flag: the unit's particles and those of the 27 cells
                const unsigned group = 0xfu << (lane & 28);
                if (__all_sync(group, (ch.x & ch.y & kLeafRef) != 0))
                {
                    u32 pop = 0;
                    for (int k = lane & 3; k < 54; k += 4) pop = __dp4a(words[k], 0x01010101u, pop);
                    pop += __shfl_xor_sync(group, pop, 1);
                    pop += __shfl_xor_sync(group, pop, 2);
                    const u32 mine = __dp4a(words[27], 0x01010101u, __dp4a(words[26], 0x01010101u, 0u));
                    if (d0 == 0 || d1 == 0)
                        out.G[(d0 == 0 ? ch.x : ch.y) & ~kLeafRef] = canMerge(mine, pop, out.bucket);
                }
            }
        }
        __syncwarp();
        if constexpr (Build) classify(first, nb);
    }
    if constexpr (Build)
    {
        __syncthreads();
        for (int k = threadIdx.x; k < kContribBins; k += kThreads)
            if (sContrib[k]) atomicAdd(a.contrib + k, (unsigned long long)sContrib[k]);
        if (threadIdx.x < kArrivals && sLanded[threadIdx.x])
            atomicAdd(a.landed + threadIdx.x, (unsigned long long)sLanded[threadIdx.x]);
    }
}

// ---------------------------------------------------------------------------
// The units of a standing NFCount tree (the full refresh of update()): its
// internal nodes, level by level from the leaf boundaries K, with the begin
// indices B of the moved particles.  A level is one kernel: a node's 7 inner
// child boundaries are found among its leaves, a child of more than one leaf is
// a unit of the next level.  The near field then goes over the units as in a
// build.
// ---------------------------------------------------------------------------
// The root (a tree of one leaf is refreshed here).
static __global__ void treeRootKernel(Arena a, rb::TreeBufs tb)
{
    const DeviceState *st = tb.st;
    if (rb::halted(st)) return;  // no units: the levels find none
    const int active = st->activeBuffer, L = st->numLeaves;
    if (L > 1)
    {
        u32 *row = a.rows;
        row[0] = row[1] = row[2] = 0;
        row[3] = 0;
        row[4] = u32(L);
        row[10] = st->numActiveParticles;
        row[11] = withUnit(0, 0, kHilbertStart);
        for (int q = 0; q < 27; ++q) a.nbr[q] = 0;  // every cell around the root is the root (periodic wrap)
        a.ctl->levelCount[0] = 1;
        return;
    }
    const u64 c = st->numActiveParticles, v = c * c > 0xffffffffull ? 0xffffffffull : c * c * 27ull;
    tb.nf(active)[0] = v > 0xffffffffull ? 0xffffffffu : u32(v);
}

// Levels of at most this many units: a CTA per unit, a warp per boundary.
constexpr u32 kTreeWideUnits = 2048;

// Child d of unit g: leaves [j, jEnd), keys [b, bEnd).  Slots of the warp's
// new units by one atomic add.  All lanes of the warp take part (act: this
// lane holds a child; the 8 children of a unit in the lanes of an aligned
// group of 8).
template <bool Hilbert>
__device__ __forceinline__ void treeChild(const Arena &a, int l, u32 next, bool act, u32 g, int d, u64 key, u32 st, u32 j,
                                          u32 jEnd, u32 b, u32 bEnd, const unsigned char *sNext, const unsigned char *sDec)
{
    Control &c = *a.ctl;
    const int lane = threadIdx.x & 31;
    const unsigned m = unsigned(l) + 1;
    const bool inner = act && jEnd - j > 1;
    const unsigned innerMask = __ballot_sync(0xffffffffu, inner);
    u32 base = 0;
    if (lane == 0 && innerMask) base = atomicAdd(&c.levelCount[l + 1], u32(__popc(innerMask)));
    base = __shfl_sync(0xffffffffu, base, 0);
    const unsigned big = __ballot_sync(0xffffffffu, act && bEnd - b >= 255u) & (0xffu << (lane & 24));
    if (!act) return;
    const u32 oct = Hilbert ? u32(sDec[st * 8 + d]) : u32(d);
    u32 slot = kLeafRef | j;
    if (inner)
    {
        const u32 gc = next + base + u32(__popc(innerMask & ((1u << lane) - 1u)));
        if (gc < a.cap)
        {
            const u64 ck = key + u64(d) * octRange(m);
            const u32 cst = Hilbert ? u32(sNext[st * 8 + oct]) : u32(kHilbertStart);
            uint4 *crow = reinterpret_cast<uint4 *>(a.rows + size_t(gc) * kRow);
            crow[0] = make_uint4(u32(ck), u32(ck >> 32), b, j);
            crow[1] = make_uint4(jEnd, 0u, 0u, 0u);
            crow[2] = make_uint4(0u, 0u, bEnd, withUnit(0, m, cst));
            a.parent[gc] = g * 8 + oct;
            slot = gc;
        }
        else
        {
            c.overflow = 1;
        }
    }
    a.child[size_t(g) * 8 + oct] = slot;
    a.rows[size_t(g) * kRow + 2 + d] = b;
    reinterpret_cast<unsigned char *>(a.rec + g)[oct] = big ? 255 : (unsigned char)(bEnd - b);
}

template <bool Hilbert>
static __global__ void __launch_bounds__(kThreads) treeUnitsKernel(Arena a, rb::TreeBufs tb, int l)
{
    __shared__ __align__(4) unsigned char sNext[48 * 8], sDec[48 * 8];
    __shared__ u32 sCut[9];
    Control &c = *a.ctl;
    if (c.overflow) return;
    const u32 start = c.levelStart[l], count = c.levelCount[l], next = start + count;
    if (blockIdx.x == 0 && threadIdx.x == 0) c.levelStart[l + 1] = next;
    const bool wide = count <= kTreeWideUnits;
    if (wide ? count <= blockIdx.x : count * 8 <= blockIdx.x * kThreads) return;
    if constexpr (Hilbert)
    {
        copyTable(sNext, gHilbert.encNext);
        copyTable(sDec, gHilbert.decOct);
    }
    __syncthreads();
    const int active = tb.st->activeBuffer;
    const u64 *K = tb.k(active);
    const u32 *B = tb.b(active);
    const u64 cr = octRange(unsigned(l) + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (wide)
    {
        for (u32 i = blockIdx.x; i < count; i += gridDim.x)
        {
            const u32 g = start + i;
            const u32 *row = a.rows + size_t(g) * kRow;
            const u64 key = rowKey(row);
            const u32 i0 = row[3], i1 = row[4], st = unitStateOf(row[11]);
            u32 cut = warp == 0 ? i0 : i1;
            if (warp > 0) cut = warpLowerBound(K, i0, i1, key + u64(warp) * cr, lane);
            if (lane == 0) sCut[warp] = cut;
            if (threadIdx.x == 0) sCut[8] = i1;
            __syncthreads();  // (row[3] and row[4] are read by every warp)
            if (warp == 0)
            {
                const bool act = lane < 8;
                const u32 j = sCut[act ? lane : 8], jEnd = sCut[act ? lane + 1 : 8];
                treeChild<Hilbert>(a, l, next, act, g, lane & 7, key, st, j, jEnd, B[j], B[jEnd], sNext, sDec);
            }
            __syncthreads();
        }
        return;
    }
    const u32 total = count * 8;
    for (u32 e0 = blockIdx.x * kThreads + (threadIdx.x & ~31u); e0 < total; e0 += gridDim.x * kThreads)
    {
        const u32 e = e0 + u32(lane);
        const bool act = e < total;
        const int d = int(e & 7);
        const u32 g = start + (act ? e >> 3 : 0);
        const u32 *row = a.rows + size_t(g) * kRow;
        const u64 key = rowKey(row);
        // (lanes without a child look at no unit's leaves: its own warp replaces
        // the two words by begin indices)
        const u32 i0 = act ? row[3] : 0u, i1 = act ? row[4] : 0u, bEnd = row[10], st = unitStateOf(row[11]);
        // first leaf of child d
        u32 j = i0;
        if (d > 0)
        {
            const u64 t = key + u64(d) * cr;
            u32 len = i1 - i0;
            while (len)
            {
                const u32 half = len >> 1;
                const bool less = __ldg(K + j + half) < t;
                j = less ? j + half + 1 : j;
                len = less ? len - half - 1 : half;
            }
        }
        const u32 b = B[j];
        __syncwarp();  // the group's lanes have read row[3] and row[4]
        u32 jEnd = __shfl_down_sync(0xffffffffu, j, 1, 8), bNext = __shfl_down_sync(0xffffffffu, b, 1, 8);
        if (d == 7)
        {
            jEnd = i1;
            bNext = bEnd;
        }
        treeChild<Hilbert>(a, l, next, act, g, d, key, st, j, jEnd, b, bNext, sNext, sDec);
    }
}

// Every unit into the (cleared) node table of the partial refreshes.
static __global__ void __launch_bounds__(kThreads) unitsToTableKernel(Arena a, rb::NodeTable gt)
{
    const Control &c = *a.ctl;
    if (c.overflow) return;
    const u32 total = c.levelStart[kOctLevels];
    for (u32 g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x)
    {
        const uint4 *r4 = reinterpret_cast<const uint4 *>(a.rows + size_t(g) * kRow);
        const uint4 r0 = r4[0], r1 = r4[1], r2 = r4[2];
        u32 *to = rb::nodeRow(gt, rb::cellCode((u64(r0.y) << 32) | r0.x, unitLevelOf(r2.w)));
        if (!to) continue;
        // (rows are 48 bytes: the two words of the code, then the 9 values)
        *reinterpret_cast<uint2 *>(to) = make_uint2(r0.z, r0.w);
        *reinterpret_cast<uint4 *>(to + 2) = r1;
        *reinterpret_cast<uint2 *>(to + 6) = make_uint2(r2.x, r2.y);
        to[8] = r2.z;
    }
}

// The leaves below every unit, all levels at once (the first `total` units): a
// unit whose children are all leaves starts (8 leaves) and adds its count to
// its parent's; the child that comes last takes the parent's total on.
template <bool Forest>
__device__ __forceinline__ void countSubtrees(const Arena &a, u32 total, const Team &team)
{
    for (u32 g = team.rank * blockDim.x + threadIdx.x; g < total; g += team.size * blockDim.x)
    {
        // (a unit with internal children holds 15 leaves or more when they have come)
        u64 n = sort::ldRelaxed(a.sub + g);
        if (n != 8) continue;
        for (u32 u = g; Forest || u != 0;)
        {
            const u32 up = a.parent[u];
            if (Forest && up == kLeaf) break;  // a system's root
            u = up >> 3;
            const u64 old = atomicAdd(reinterpret_cast<unsigned long long *>(a.sub + u),
                                      (unsigned long long)(n - (u64(1) << kSubShift)));
            if ((old >> kSubShift) != 1) break;
            n += old & ((u64(1) << kSubShift) - 1);
        }
    }
}

// The subtree counts of an NFCount build.  (A kernel per level cost its launch
// and tail 11 times at 300k particles, 2.5 us and a gap each.)  `levels` is
// the number of levels the build expanded: units below them mean the build is
// incomplete, and nothing is counted.
static __global__ void __launch_bounds__(kThreads) subtreeKernel(Arena a, int levels)
{
    const Control &c = *a.ctl;
    if (c.levelCount[levels] | c.overflow | c.late | c.error) return;
    countSubtrees<false>(a, c.levelStart[levels], wholeGrid());
}

// Cornerstone entries of the leaf children of every unit (the first `total`),
// and the first leaf index of their internal children.  Eight lanes per unit,
// one per child: a segmented scan of the children's leaf counts gives each
// child's position, so a warp writes the entries of four units at once.
// K, B (and NF, N, SEG where given) are the cornerstone arrays written: N the
// leaf counts, SEG each leaf's tree (system) in a batch of trees.  dec: the
// digit -> octant table of the Hilbert curve (NFCount trees keep their
// children by octant).
//
// A unit waits for its own place, which its parent's warp writes; parents come
// before their children in the arena.  The warps of the team, all resident,
// take units in increasing order, and a warp writes what is ready before it polls again (parent and child may share it), so the
// first unit not placed is always being worked on and the waits end (they are
// bounded all the same).  Bound by the latency of a step: child, its leaf
// count, the poll.  Chunks of units handed out by a counter, with their levels
// looked up, took 43 us for the 32k units of 300k NFCount particles, 166 us for
// the 1.8 M of 16Mi and 51 us for the 133k of an 8Mi k-d tree (a kernel per
// level before that: 36 us and 11 gaps at 300k).
template <bool NF, bool Hilbert, bool Forest>
__device__ __forceinline__ void placeUnits(const Arena &a, const Team &team, u64 *K, u32 *B, u32 *NFo, u32 *N, int *SEG,
                                           u32 total, u32 capacity, const unsigned char *dec,
                                           unsigned spinLimit = kPlaceSpins)
{
    Control &c = *a.ctl;
    const int lane = threadIdx.x & 31, d = lane & 7;
    const u32 stride = team.size * (kThreads / 8);
    for (u32 g0 = team.rank * (kThreads / 8) + (threadIdx.x >> 5) * 4; g0 < total; g0 += stride)
    {
        const u32 g = min(g0 + (lane >> 3), total - 1);
        bool done = g0 + (lane >> 3) >= total;
        const u32 *row = a.rows + size_t(g) * kRow;
        const u32 reg = row[11], begin = row[2 + d], end = row[3 + d];
        const u64 key = rowKey(row) + u64(d) * octRange(unitLevelOf(reg) + 1);
        u32 ch = a.child[size_t(g) * 8 + d];
        u32 val = 0, sys = 0;
        if constexpr (NF) val = a.val[size_t(g) * 8 + d];
        if constexpr (Forest) sys = a.usys[g];
        u32 mine = ch == kLeaf ? 1u : u32(a.sub[ch]);
        if constexpr (NF && Hilbert)
        {
            // from octants to digits within the unit's 8 lanes
            const int from = (lane & 24) | dec[unitStateOf(reg) * 8 + d];
            ch = __shfl_sync(0xffffffffu, ch, from);
            mine = __shfl_sync(0xffffffffu, mine, from);
        }
        // exclusive prefix of the leaf counts within the unit's 8 lanes
        u32 inc = mine;
#pragma unroll
        for (int off = 1; off < 8; off <<= 1)
        {
            const u32 t = __shfl_up_sync(0xffffffffu, inc, off);
            if (d >= off) inc += t;
        }
        for (unsigned spins = 0;; ++spins)
        {
            if (!done)
            {
                const u32 first = vload(a.offset[g]);  // the unit's first leaf
                if (first != kPending)
                {
                    done = true;
                    const u32 o = first + inc - mine;
                    if (ch != kLeaf)
                    {
                        *static_cast<volatile u32 *>(a.offset + ch) = o;
                    }
                    else if (o >= capacity)
                    {
                        c.placeOverflow = 1;  // the host grows the buffers and places again
                    }
                    else
                    {
                        K[o] = key;
                        B[o] = begin;
                        if constexpr (NF) NFo[o] = val;
                        if (N) N[o] = end - begin;
                        if constexpr (Forest) SEG[o] = int(sys);
                    }
                }
            }
            if (__all_sync(0xffffffffu, done)) break;
            if (spins < 64) continue;
            if (spins > spinLimit || vload(c.error))
            {
                c.error = kErrLookback;
                return;
            }
            __nanosleep(64);
        }
    }
}

// (by team)  `levels`: the levels the build expanded.
template <bool NF, bool Hilbert>
static __global__ void __launch_bounds__(kThreads, 4)
    placeKernel(Arena a, u64 *K, u32 *B, u32 *NFo, u32 *N, int levels, u32 capacity)
{
    __shared__ __align__(4) unsigned char sDec[48 * 8];
    Control &c = *a.ctl;
    if (c.levelCount[levels] | c.overflow | c.late | c.error) return;  // (c.error: this launch's, too)
    Team team{enterRoll(&c.bar), 0};
    if (team.rank == kLeftOut) return;
    if constexpr (NF && Hilbert)
    {
        copyTable(sDec, gHilbert.decOct);
        __syncthreads();
    }
    const u32 total = c.levelCount[0] ? c.levelStart[levels] : 0u;
    team.size = closeRoll(&c.bar);
    if (!team.size)
    {
        if (threadIdx.x == 0) c.error = kErrLookback;
        return;
    }
    placeUnits<NF, Hilbert, false>(a, team, K, B, NFo, N, nullptr, total, capacity, sDec);
}

// The finished tree: sentinel boundary and the state of a converged build
// (finishBuildStateKernel, octree.cu:40-47, after `rounds` changing rounds).
__device__ __forceinline__ void finishState(const rb::TreeBufs &tb, int leaves, int rounds)
{
    DeviceState *st = tb.st;
    tb.K[0][leaves] = kMaxKey;
    tb.B[0][leaves] = st->numActiveParticles;
    st->numLeaves = leaves;
    st->newNumLeaves = leaves;
    st->proposal = leaves;
    st->iteration = rounds;
    st->rounds = rounds + 1;
    st->changed = st->converged = st->needsResize = 0;
    st->numNodes = 0;
    st->activeBuffer = 0;
    st->overflow = 0;
    st->dirtyCount = 0;
}

static __global__ void finishKernel(Arena a, rb::TreeBufs tb, int rounds, int levels, u32 capacity)
{
    const Control &c = *a.ctl;
    if (c.levelCount[levels] | c.overflow | c.late | c.error | c.placeOverflow) return;
    const int leaves = c.levelCount[0] ? int(u32(a.sub[0])) : 1;
    if (u32(leaves) <= capacity) finishState(tb, leaves, rounds);
}

struct LeafBuildArgs
{
    Arena a;  // (control block zero on entry)
    KeyIndex idx;
    rb::TreeBufs tb;
    const u64 *P;
    size_t n;
    unsigned bucket, maxDepth;
    u32 capacity;  // leaves the cornerstone buffers hold
};

// A LeafCount build in one launch by team: root, levels, subtree counts,
// placement and final state.  Bound by the latency of the searches and the
// barriers on small trees, of the searches on large ones.  With a launch per
// step and level: 10k particles 74 us in 19 launches, now 49; 1Mi 71 in 15,
// now 75 without their gaps (build() 212 to 160 and 262 to 238 us).
//
// CTAs take the same turns at the barriers: a level's count, and with it the
// room in the arena, is final once its barrier has opened, while the overflow
// flag may already be set by the next level's units and is read after the
// last barrier only.
static __global__ void __launch_bounds__(kThreads, 4) leafBuildKernel(LeafBuildArgs p)
{
    __shared__ u32 sContrib[kContribBins];
    __shared__ u32 sLanded[kArrivals];
    __shared__ u32 sEnds[8];
    __shared__ int sRounds;
    const Arena &a = p.a;
    Control &c = *a.ctl;
    for (int k = threadIdx.x; k < kContribBins; k += kThreads) sContrib[k] = 0;
    if (threadIdx.x < kArrivals) sLanded[threadIdx.x] = 0;
    if (threadIdx.x == 0) sRounds = 0;
    Team team{enterRoll(&c.bar), 0};
    if (team.rank == kLeftOut) return;
    if (team.rank == 0 && threadIdx.x < 32) rootUnit(a, p.tb, p.P, p.n, p.bucket, false);
    team.size = closeRoll(&c.bar);
    if (!team.size || !gridBarrier(&c.bar, team)) return;
    int levels = 0;
    for (; levels < int(kOctLevels); ++levels)
    {
        const u32 start = vload(c.levelStart[levels]), count = vload(c.levelCount[levels]);
        if (count == 0 || count > a.cap - start) break;
        growUnits<false>(a, p.idx, levels, p.bucket, start, count, team, sEnds, sContrib, sLanded);
        if (!gridBarrier(&c.bar, team)) return;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kContribBins; k += kThreads)
        if (sContrib[k]) atomicAdd(a.contrib + k, (unsigned long long)sContrib[k]);
    if (threadIdx.x < kArrivals && sLanded[threadIdx.x])
        atomicAdd(a.landed + threadIdx.x, (unsigned long long)sLanded[threadIdx.x]);
    const u32 total = levels ? vload(c.levelStart[levels]) : 0u;
    countSubtrees<false>(a, total, team);
    if (!gridBarrier(&c.bar, team)) return;
    if (vload(c.overflow) | vload(c.late)) return;
    if (team.rank == 0)
    {
        for (int k = threadIdx.x; k < kContribBins; k += kThreads)
            if (vload(a.contrib[k]))
            {
                const int j = k % kJumps, kk = (k / kJumps) % kJumps, ai = k / (kJumps * kJumps);
                atomicMax(&sRounds, ai + 1 + kk - j);
            }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            const u32 leaves = levels ? u32(vload(a.sub[0])) : 1u;
            c.leaves = leaves;
            c.active = p.tb.st->numActiveParticles;
            c.stateError = p.tb.st->error;
            if (leaves > p.capacity) c.placeOverflow = 1;
            else if (sRounds <= int(p.maxDepth)) finishState(p.tb, int(leaves), sRounds);
        }
    }
    placeUnits<false, false, false>(a, team, p.tb.K[0], p.tb.B[0], nullptr, p.tb.N[0], nullptr, total, p.capacity, nullptr);
}
}  // namespace lb
}  // namespace aot
