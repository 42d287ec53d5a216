// binlevel.cuh -- the converged binary (k-d) tree build, three levels at a time.
//
// The reference builds a binary tree from the root by passes until a pass
// changes nothing (the build loop of kdtree3d.cu:239-249 over
// binaryDecisionKernel, kdtree3d_rebalance.cuh:28-60): a leaf splits in two
// when it holds more than `bucket` particles and its depth is below
// maxDepth, and two sibling leaves merge when together they hold at most
// `bucket`.  A leaf's count never grows from a node to its children, so no
// pair made by a split can merge afterwards, and the tree the passes end with
// is unique: a node is internal exactly when it holds more than `bucket`
// particles below maxDepth.
//
// A "unit" is an internal node at a depth that is a multiple of three,
// together with the nodes of the two depths below it: its slots are its 8
// descendants three depths down.  A slot is an internal node (a unit of the
// next level), a leaf, or part of a wider leaf of 2 or 4 slots, which starts
// at the first of them.  One launch by team (buildKernel, grid_barrier.cuh)
// makes the tree:
//   levels    the 7 inner slot boundaries of each unit among its keys, then
//             its slots (warp-aggregated slots of new units), barrier;
//   subtree   subtree leaf counts, bottom-up, all levels at once;
//   place     every leaf's K, B and count, top-down, all levels at once.
// Each pass of the reference splits one depth, so the passes that change the
// tree number the deepest internal node's depth + 1, and its leaf capacity,
// grown by 25 % steps to the leaf count of every pass (commitIfLast,
// rebalance.cuh), ends at the first step of that chain at or above the final
// leaf count: the counts only grow during a build.
#pragma once

#include "levelbuild.cuh"

namespace aot
{
namespace bl
{
using lb::kLeaf;
using lb::kThreads;
constexpr u32 kInside = 0xfffffffeu;  // child slot: inside a leaf that starts before it
constexpr int kLevels = 21;           // unit depths 0, 3, .. 60
constexpr u32 kWideUnits = 2048;      // levels of at most this many units search by warps

struct Control
{
    u32 levelStart[kLevels + 2];
    u32 levelCount[kLevels + 2];
    int overflow;       // the unit arena is too small
    int placeOverflow;  // more leaves than the leaf arrays hold
    int error;          // a bounded wait gave up
    GridBarrier bar;
    int depths;         // depths holding internal nodes
    u32 leaves;         // leaves of the tree
    u32 units;
    u32 active;         // active particles
    int stateError;     // DeviceState::error
};

struct Arena
{
    u32 *rows;      // [cap][lb::kRow] key (2 words), 9 slot begins, slot masks: leaf or unit starts |
                    // units << 8 | level << 16
    u32 *child;     // [cap][8] unit index of an internal slot, kLeaf or kInside
    u32 *parent;    // [cap] parent unit
    u64 *sub;       // [cap] leaves counted below the unit | units to come << lb::kSubShift
    u32 *offset;    // [cap] leaf index of the unit's first leaf (lb::kPending before it is known)
    Control *ctl;
    u32 cap;
};

// Key range of a node at depth d: 2^(63 - d).
__device__ __forceinline__ u64 depthRange(int d) { return u64(1) << (63 - d); }

// The root (one warp): a unit when it holds more than `bucket` particles (and
// may split), else the single root leaf, written straight to the leaf arrays.
__device__ __forceinline__ void rootUnit(const Arena &a, const rb::TreeBufs &tb, const u64 *P, size_t n, unsigned bucket,
                                         unsigned maxDepth)
{
    const unsigned active = n ? warpLowerBound(P, 0, u32(n), kMaxKey, int(threadIdx.x & 31)) : 0u;
    if (threadIdx.x != 0) return;
    DeviceState *st = tb.st;
    const int err = st->error;
    *st = DeviceState{};
    st->error = err;
    st->numActiveParticles = active;
    Control &c = *a.ctl;
    c.levelStart[0] = 0;
    if (active > bucket && maxDepth > 0)
    {
        a.rows[0] = a.rows[1] = a.rows[2] = 0;
        a.rows[10] = active;
        a.offset[0] = 0;
        c.levelCount[0] = 1;
    }
    else
    {
        c.levelCount[0] = 0;
        tb.K[0][0] = 0;
        tb.K[0][1] = kMaxKey;
        tb.B[0][0] = 0;
        tb.B[0][1] = active;
        tb.N[0][0] = active;
    }
}

// The slots of units: lanes hold one each, eight to a unit g in key order, of
// which `valid` ones take part (whole units; all lanes of the warp call).
// [begin, end): the slot's keys.  deepest: of the CTA.
__device__ __forceinline__ void growSlots(const Arena &a, int level, unsigned bucket, unsigned maxDepth, u32 next, u32 g,
                                          bool valid, u32 begin, u32 end, u64 key, int &deepest)
{
    Control &c = *a.ctl;
    const int l = 3 * level, lane = threadIdx.x & 31, d = lane & 7;
    const auto splits = [&](u32 count, int depth) { return count > bucket && unsigned(depth) < maxDepth; };
    // particles of the slot and of the wider nodes that hold it
    const u32 x1 = end - begin;
    const u32 x2 = x1 + __shfl_xor_sync(0xffffffffu, x1, 1);
    const u32 x4 = x2 + __shfl_xor_sync(0xffffffffu, x2, 2);
    const bool half = valid && splits(x4, l + 1), quarter = half && splits(x2, l + 2);
    const bool high = quarter && splits(x1, l + 3);
    const bool starts = valid && (quarter || (half ? (d & 1) == 0 : (d & 3) == 0));
    const unsigned highs = __ballot_sync(0xffffffffu, high), starting = __ballot_sync(0xffffffffu, starts);
    const unsigned halves = __ballot_sync(0xffffffffu, half), quarters = __ballot_sync(0xffffffffu, quarter);
    if (quarters) deepest = max(deepest, l + 3);
    else if (halves) deepest = max(deepest, l + 2);
    else deepest = max(deepest, l + 1);
    u32 base = 0;
    if (lane == 0 && highs) base = atomicAdd(&c.levelCount[level + 1], u32(__popc(highs)));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (!valid) return;
    u32 slot = starts ? kLeaf : kInside;
    if (high)
    {
        const u32 gc = next + base + u32(__popc(highs & sort::laneMaskLt()));
        if (gc < a.cap)
        {
            const u64 ck = key + u64(d) * depthRange(l + 3);
            uint4 *crow = reinterpret_cast<uint4 *>(a.rows + size_t(gc) * lb::kRow);
            crow[0] = make_uint4(u32(ck), u32(ck >> 32), begin, 0u);
            crow[2] = make_uint4(0u, 0u, end, 0u);
            a.parent[gc] = g;
            a.offset[gc] = lb::kPending;
            slot = gc;
        }
        else
        {
            c.overflow = 1;
        }
    }
    a.child[size_t(g) * 8 + d] = slot;
    if (d != 0) return;
    const u32 s8 = (starting >> lane) & 0xffu, h8 = (highs >> lane) & 0xffu;
    a.rows[size_t(g) * lb::kRow + 11] = s8 | (h8 << 8) | (u32(level) << 16);
    a.sub[g] = (u64(__popc(h8)) << lb::kSubShift) | u32(__popc(s8) - __popc(h8));
}

// The units of a level, by a team: on levels of few units a CTA per
// unit, a warp per inner boundary (sEnds: 7 words of the CTA), else a lane per
// slot.
__device__ __forceinline__ void growUnits(const Arena &a, const KeyIndex &idx, int level, unsigned bucket,
                                          unsigned maxDepth, u32 start, u32 count, const Team &team, u32 *sEnds,
                                          int &deepest)
{
    const u32 next = start + count;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u64 range = depthRange(3 * level + 3);
    if (team.rank == 0 && threadIdx.x == 0) a.ctl->levelStart[level + 1] = next;
    if (count <= kWideUnits)
    {
        static_assert(kThreads / 32 >= 7, "a warp per inner boundary");
        for (u32 i = team.rank; i < count; i += team.size)
        {
            u32 *row = a.rows + size_t(start + i) * lb::kRow;
            const u32 lo = row[2], hi = row[10];
            const u64 key = lb::rowKey(row);
            if (warp < 7)
            {
                const u32 r = lb::warpBoundaryIn(idx, lo, hi, key + u64(warp + 1) * range, lane);
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
                growSlots(a, level, bucket, maxDepth, next, start + i, lane < 8, d ? sEnds[d - 1] : lo,
                          d < 7 ? sEnds[d] : hi, key, deepest);
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
        u32 *row = a.rows + size_t(g) * lb::kRow;
        const u32 lo = row[2], hi = row[10];
        const u64 key = lb::rowKey(row);
        u32 end = hi;
        if (valid && d < 7)
        {
            end = lb::boundaryIn(idx, lo, hi, key + u64(d + 1) * range);
            row[3 + d] = end;
        }
        const u32 prev = __shfl_up_sync(0xffffffffu, end, 1, 8);
        growSlots(a, level, bucket, maxDepth, next, g, valid, d ? prev : lo, end, key, deepest);
    }
}

// The leaves below every unit (lb::countSubtrees): a unit without units below
// it starts, and the unit below another that comes last takes the total on.
__device__ __forceinline__ void countSubtrees(const Arena &a, u32 total, const Team &team)
{
    for (u32 g = team.rank * blockDim.x + threadIdx.x; g < total; g += team.size * blockDim.x)
    {
        if (a.rows[size_t(g) * lb::kRow + 11] & 0xff00u) continue;
        u64 n = sort::ldRelaxed(a.sub + g);
        for (u32 u = g; u != 0;)
        {
            u = a.parent[u];
            const u64 old = atomicAdd(reinterpret_cast<unsigned long long *>(a.sub + u),
                                      (unsigned long long)(n - (u64(1) << lb::kSubShift)));
            if ((old >> lb::kSubShift) != 1) break;
            n += old & ((u64(1) << lb::kSubShift) - 1);
        }
    }
}

// K, B and the count of the leaves that start in every unit, and the first
// leaf index of the units below (lb::placeUnits with a lane per slot).
__device__ __forceinline__ void placeUnits(const Arena &a, const Team &team, u64 *K, u32 *B, u32 *N, u32 total,
                                           u32 capacity, unsigned spinLimit = lb::kPlaceSpins)
{
    Control &c = *a.ctl;
    const int lane = threadIdx.x & 31, d = lane & 7;
    const u32 stride = team.size * (kThreads / 8);
    for (u32 g0 = team.rank * (kThreads / 8) + (threadIdx.x >> 5) * 4; g0 < total; g0 += stride)
    {
        const u32 g = min(g0 + (lane >> 3), total - 1);
        bool done = g0 + (lane >> 3) >= total;
        const u32 *row = a.rows + size_t(g) * lb::kRow;
        const u32 word = row[11], begin = row[2 + d], later = (word & 0xffu) >> (d + 1);  // starts of the slots after d
        const u32 ch = a.child[size_t(g) * 8 + d];
        const u32 mine = ch == kLeaf ? 1u : ch == kInside ? 0u : u32(a.sub[ch]);
        const u32 end = row[2 + (later ? d + __ffs(int(later)) : 8)];
        const u64 key = lb::rowKey(row) + u64(d) * depthRange(3 * int(word >> 16) + 3);
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
                const u32 first = vload(a.offset[g]);
                if (first != lb::kPending)
                {
                    done = true;
                    const u32 o = first + inc - mine;
                    if (ch == kLeaf && o >= capacity)
                    {
                        c.placeOverflow = 1;  // the host grows the leaf arrays and places again
                    }
                    else if (ch == kLeaf)
                    {
                        K[o] = key;
                        B[o] = begin;
                        N[o] = end - begin;
                    }
                    else if (ch != kInside)
                    {
                        *static_cast<volatile u32 *>(a.offset + ch) = o;
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

// (by team)
static __global__ void __launch_bounds__(kThreads, 4) placeKernel(Arena a, u64 *K, u32 *B, u32 *N, u32 total, u32 capacity)
{
    Control &c = *a.ctl;
    if (c.overflow | c.error) return;  // (c.error: this launch's, too)
    Team team{enterRoll(&c.bar), 0};
    if (team.rank == kLeftOut) return;
    team.size = closeRoll(&c.bar);
    if (!team.size)
    {
        if (threadIdx.x == 0) c.error = kErrLookback;
        return;
    }
    placeUnits(a, team, K, B, N, total, capacity);
}

// The finished tree: its sentinel and the state the reference's passes end
// with (the last pass changes nothing: converged, one more pass counted).
__device__ __forceinline__ void finishState(const rb::TreeBufs &tb, int leaves, int passes, long long logicalCap)
{
    DeviceState *st = tb.st;
    tb.K[0][leaves] = kMaxKey;
    tb.B[0][leaves] = st->numActiveParticles;
    st->numLeaves = st->newNumLeaves = leaves;
    st->numNodes = (leaves - 1) * 2 + 1;
    st->proposal = leaves;
    st->iteration = passes;
    st->rounds = passes + 1;
    st->converged = 1;
    st->changed = st->needsResize = 0;
    st->activeBuffer = 0;
    st->overflow = 0;
    st->dirtyCount = 0;
    st->logicalCap = logicalCap;
}

static __global__ void finishKernel(rb::TreeBufs tb, int leaves, int passes, long long logicalCap)
{
    finishState(tb, leaves, passes, logicalCap);
}

// Leaf capacity after a build that ends with `leaves` leaves.
__host__ __device__ __forceinline__ long long grownCapacity(long long c, long long leaves)
{
    if (c < 1) c = 1;
    while (leaves > c) c += (c + 3) / 4;
    return c;
}

struct BuildArgs
{
    Arena a;  // (control block zero on entry)
    KeyIndex idx;
    rb::TreeBufs tb;
    const u64 *P;
    size_t n;
    unsigned bucket, maxDepth;
    u32 capacity;           // leaves the leaf arrays hold
    long long logicalCap;   // the reference's leaf capacity before the build
};

// The whole build in one launch by team.  Bound by the latency of its
// steps: 33 depths of an 8Mi k-d tree are 11 levels here; with a launch per
// depth they took 190 us and 34 gaps, the subtree counts 33 us and the
// placement 28 us, whose chains of dependent steps are a third as long now.
// (CTAs decide at the barriers as in lb::leafBuildKernel.)
static __global__ void __launch_bounds__(kThreads, 4) buildKernel(BuildArgs p)
{
    __shared__ u32 sEnds[8];
    const Arena &a = p.a;
    Control &c = *a.ctl;
    Team team{enterRoll(&c.bar), 0};
    if (team.rank == kLeftOut) return;
    if (team.rank == 0 && threadIdx.x < 32) rootUnit(a, p.tb, p.P, p.n, p.bucket, p.maxDepth);
    team.size = closeRoll(&c.bar);
    if (!team.size || !gridBarrier(&c.bar, team)) return;
    int levels = 0, deepest = 0;
    for (; levels < kLevels; ++levels)
    {
        const u32 start = vload(c.levelStart[levels]), count = vload(c.levelCount[levels]);
        if (count == 0 || count > a.cap - start) break;
        growUnits(a, p.idx, levels, p.bucket, p.maxDepth, start, count, team, sEnds, deepest);
        if (!gridBarrier(&c.bar, team)) return;
    }
    if ((threadIdx.x & 31) == 0 && deepest) atomicMax(&c.depths, deepest);
    const u32 total = levels ? vload(c.levelStart[levels]) : 0u;
    countSubtrees(a, total, team);
    if (!gridBarrier(&c.bar, team)) return;
    if (vload(c.overflow)) return;
    if (team.rank == 0 && threadIdx.x == 0)
    {
        const u32 leaves = levels ? u32(vload(a.sub[0])) : 1u;
        c.leaves = leaves;
        c.units = total;
        c.active = p.tb.st->numActiveParticles;
        c.stateError = p.tb.st->error;
        if (leaves > p.capacity) c.placeOverflow = 1;
        else finishState(p.tb, int(leaves), vload(c.depths), grownCapacity(p.logicalCap, (long long)leaves));
    }
    placeUnits(a, team, p.tb.K[0], p.tb.B[0], p.tb.N[0], total, p.capacity);
}
}  // namespace bl
}  // namespace aot
