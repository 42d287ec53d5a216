// sort_repair.cuh -- the end of a planned sort (sort_plan.cuh): the keys are
// in order of their high digits, stably; each run of equal high digits is
// brought into order of the remaining bits, stably, by one kernel that reads
// every key once.
//
// A CTA takes the runs that start in its tile and holds the tile and kMaxRun
// keys on either side in shared memory.  A bit per key marks the starts of
// runs, so a key finds its run in its word of marks or the next ones; its place in the run is
// the number of the run's keys that come before it, counted in shared memory
// (all lanes of a run read the same word).  Most runs are a handful of keys,
// and in place a key that stands where it belongs is not written.  Runs of more
// than kMaxRun keys are listed and sorted by a CTA each (longRunKernel): with
// the plan's sampling they are rare, so what counts there is that they end.
//
// The passes leave the keys in buffer (passes run) & 1, or in buffer 0
// (endsIn0); the result is in buffer 0.  In place, only the owner of a run
// moves its keys; the others look at the high digits alone, which a move
// inside a run does not change.
#pragma once

#include "radix_sort.cuh"

namespace aot
{
namespace sort
{
constexpr int kRepairThreads = 256;
constexpr int kRepairTile = kRepairThreads * 8;  // keys per CTA of the contiguous sort's repair
constexpr int kMaxRun = 256;  // longest run the tile kernel orders
constexpr int kLongThreads = 512;

// words of the list of long runs: start and end of its segment for each
__host__ __device__ constexpr size_t longRunWords(size_t n) { return 2 * (n / kMaxRun + 1); }

struct RepairArgs
{
    u64 *k[2];
    u32 *v[2];
    size_t n;
    SortControl *ctl;
    u32 *longList;  // the long runs: start, end of the segment [longRunWords(n)]
    u64 *sample;    // every 32nd sorted key (KeyIndex), or nullptr
    const int *error;  // a look-back gave up: the passes' order cannot be relied on
    int beginBit, passes;
    u64 keyMask;    // the sorted bits
    bool endsIn0;
    bool aligned;   // buffers 0 and 1 start at 16-byte addresses
    bool escapes;   // keys of escaped particles (all bits set) share their high digits with no other key
};

template <int Tile>
struct RepairShared
{
    static constexpr int kWindow = Tile + 2 * kMaxRun;
    u32 lo[kWindow], hi[kWindow];  // the words of the window's keys
    u32 val[kWindow];
    u32 mark[kWindow / 32];
    int before[kWindow / 32];  // last mark before the word's second key (kNoMark: none)
    int after[kWindow / 32];   // first mark after the word (-kNoMark: none)
};
// Far enough from every position that a run to or from it is too long.
constexpr int kNoMark = -(1 << 20);

// The runs that start in the tile of (at most) Tile keys from `begin`, in the
// segment [segBegin, segEnd) of keys that are sorted together.  First: the
// plan's first pass, with all 64 bits sorted, so that what tells runs apart
// and what orders a run are known words; or 0: any plan, and the sorted bits
// are those of keyMask.
//
// Window position w is key begin - kMaxRun + w.  The warps take the window's
// words of 32 marks in turn; the runs of a word's keys start and end in the
// word or, the same for all its lanes, at the last mark before it and the
// first one after it (found for all words by two warps first).
template <int First, int Tile>
__device__ __forceinline__ void repairTile(const RepairArgs &a, RepairShared<Tile> &sm, u32 first, bool inPlace,
                                           size_t begin, size_t segBegin, size_t segEnd)
{
    constexpr int kWindow = Tile + 2 * kMaxRun, kWords = kWindow / 32, kSide = kMaxRun / 32;
    static_assert(Tile % (2 * kRepairThreads) == 0 && 2 * kMaxRun % (2 * kRepairThreads) == 0, "whole rounds of loads");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // pointers to the key of window position 0 (used for positions [wBegin, wEnd) only)
    const long long origin = (long long)begin - kMaxRun;
    const u64 *src = (inPlace ? a.k[0] : a.k[1]) + origin;
    const u32 *srcV = (inPlace ? a.v[0] : a.v[1]) + origin;
    u64 *dst = a.k[0] + origin;
    u32 *dstV = a.v[0] + origin;
    const int wBegin = (long long)segBegin > origin ? int((long long)segBegin - origin) : 0;
    const bool atStart = (long long)segBegin >= origin;  // the window's first key starts the segment
    const int wEnd = (long long)segEnd - origin < kWindow ? int((long long)segEnd - origin) : kWindow;
    if (a.aligned && wBegin == 0 && wEnd == kWindow && (begin & 1) == 0)
    {
#pragma unroll
        for (int i = 0; i < kWindow / (2 * kRepairThreads); ++i)
        {
            const int w = 2 * (tid + i * kRepairThreads);  // origin and w are even
            const uint4 k = *reinterpret_cast<const uint4 *>(src + w);
            *reinterpret_cast<uint2 *>(sm.lo + w) = make_uint2(k.x, k.z);
            *reinterpret_cast<uint2 *>(sm.hi + w) = make_uint2(k.y, k.w);
            *reinterpret_cast<uint2 *>(sm.val + w) = *reinterpret_cast<const uint2 *>(srcV + w);
        }
    }
    else if (wBegin == 0 && wEnd == kWindow)
    {
#pragma unroll
        for (int i = 0; i < kWindow / kRepairThreads; ++i)
        {
            const int w = tid + i * kRepairThreads;
            const u64 k = src[w];
            sm.lo[w] = u32(k);
            sm.hi[w] = u32(k >> 32);
            sm.val[w] = srcV[w];
        }
    }
    else
    {
        for (int w = wBegin + tid; w < wEnd; w += kRepairThreads)
        {
            const u64 k = src[w];
            sm.lo[w] = u32(k);
            sm.hi[w] = u32(k >> 32);
            sm.val[w] = srcV[w];
        }
    }
    __syncthreads();
    const u64 mask = a.keyMask;
    const int prefix = a.beginBit + int(first) * kRadixBits;  // bits below are not sorted yet
    const u64 prefixMask = mask & (~u64(0) << prefix);
    const u32 hiMask = u32(prefixMask >> 32), loMask = u32(prefixMask);
    for (int word = warp; word < kWords; word += kRepairThreads / 32)
    {
        // a run starts at the first key and where the high digits change; the
        // first key of the window cannot be told (not marked), and the end of
        // the keys ends the last run
        const int w = word * 32 + lane;
        bool mark = w == wEnd;
        if (w > wBegin && w < wEnd)
        {
            mark = (sm.hi[w] ^ sm.hi[w - 1]) & (First >= 1 && First <= 4 ? ~0u : hiMask);
            if (First < 4) mark |= ((sm.lo[w] ^ sm.lo[w - 1]) & loMask) != 0;
        }
        else if (w == wBegin)
        {
            mark = atStart;
        }
        const u32 m = __ballot_sync(0xffffffffu, mark);
        if (lane == 0) sm.mark[word] = m;
    }
    __syncthreads();
    if (warp < 2)
    {
        // warp 0: the last mark at or before the start of each word; warp 1:
        // the first one after its end (the words mirrored, the marks negated)
        int carry = kNoMark;
        for (int c = 0; c < (kWords + 31) / 32; ++c)
        {
            const int i = c * 32 + lane, word = warp == 0 ? i : kWords - 1 - i;
            const u32 m = i < kWords ? sm.mark[word] : 0u;
            int v = kNoMark;  // of the word itself
            if (m) v = warp == 0 ? word * 32 + 31 - __clz(int(m)) : -(word * 32 + __ffs(int(m)) - 1);
            int inc = v;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1)
            {
                const int t = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc = max(inc, t);
            }
            int excl = __shfl_up_sync(0xffffffffu, inc, 1);
            excl = max(lane ? excl : kNoMark, carry);
            if (i < kWords)
            {
                if (warp == 0) sm.before[word] = (m & 1u) ? word * 32 : excl;
                else sm.after[word] = -excl;
            }
            carry = max(carry, __shfl_sync(0xffffffffu, inc, 31));
        }
    }
    __syncthreads();  // from here on buffers 0 are written: keys and values are read from shared memory
    const unsigned le = laneMaskLt() | (1u << lane);
#pragma unroll 1
    for (int word = kSide + warp; word < kWords; word += kRepairThreads / 32)
    {
        const u32 marks = sm.mark[word];
        if (word >= kSide + Tile / 32 && (marks & 1u)) break;  // past the last run of the tile
        const int w0 = word * 32, w = w0 + lane;
        if (w >= wEnd) break;
        const u32 mh = marks & le, me = marks & ~le;
        const int h = mh ? w0 + 31 - __clz(int(mh)) : sm.before[word];
        const int e = me ? w0 + __ffs(int(me)) - 1 : sm.after[word];
        const u32 lo = sm.lo[w];
        int to = w;
        if (e - h > kMaxRun)
        {
            // part of a long run: its first key's CTA lists it, every key of
            // the tile is brought over as it is (escaped particles are equal
            // keys: nothing to sort)
            if (w >= kMaxRun + Tile) continue;
            if (h == w && !(a.escapes && (lo & sm.hi[w]) == 0xffffffffu))
            {
                const u32 slot = atomicAdd(&a.ctl->longRuns, 1u);
                a.longList[2 * slot] = u32(origin + w);
                a.longList[2 * slot + 1] = u32(segEnd);
            }
        }
        else
        {
            if (unsigned(h - kMaxRun) >= unsigned(Tile)) continue;  // another CTA's run
            if (e - h > 1)
            {
                to = h;
                if (First >= 1 && First <= 4)
                {
                    // at most 32 bits are left: the low words order the run
                    // (with the place as one 64-bit compare; 16Mi keys: 116 us
                    // by two 32-bit ones, 109)
                    const u64 mine = (u64(lo) << 32) | u32(w);
#pragma unroll 2
                    for (int j = h; j < e; ++j) to += ((u64(sm.lo[j]) << 32) | u32(j)) < mine ? 1 : 0;
                }
                else
                {
                    const u64 mine = ((u64(sm.hi[w]) << 32) | lo) & mask;
                    for (int j = h; j < e; ++j)
                    {
                        const u64 o = ((u64(sm.hi[j]) << 32) | sm.lo[j]) & mask;
                        to += (o < mine || (o == mine && j < w)) ? 1 : 0;
                    }
                }
            }
        }
        if (to != w || !inPlace)
        {
            dst[to] = (u64(sm.hi[w]) << 32) | lo;
            dstV[to] = sm.val[w];
        }
    }
    if (!a.sample) return;
    __syncthreads();
    // the sample's keys in the CTA's runs, at every word's start (those of
    // long runs are written again when the run is sorted)
    static_assert(kSampleStride == 32, "a word of marks per sampled key");
    for (int word = kSide + tid; word < kWords; word += kRepairThreads)
    {
        const int w = word * 32, h = sm.before[word];
        const bool inTile = word < kSide + Tile / 32;
        if (w >= wEnd) continue;
        const bool mine = unsigned(h - kMaxRun) < unsigned(Tile);
        const u32 later = sm.mark[word] & ~1u;
        const bool isLong = (later ? w + __ffs(int(later)) - 1 : sm.after[word]) - h > kMaxRun;
        if (isLong ? inTile : mine) a.sample[(origin + w) >> kSampleShift] = dst[w];
    }
}

// Whole: all 64 bits are sorted.
template <bool Whole>
static __global__ void __launch_bounds__(kRepairThreads) repairKernel(RepairArgs a)
{
    __shared__ __align__(16) RepairShared<kRepairTile> sm;
    if (*a.error) return;
    const u32 first = a.ctl->first;
    if (first == 0)
    {
        // every pass has run; only the sample is left
        if (a.sample)
            for (size_t j = size_t(blockIdx.x) * kRepairThreads + threadIdx.x; (j << kSampleShift) < a.n;
                 j += size_t(gridDim.x) * kRepairThreads)
                a.sample[j] = a.k[0][j << kSampleShift];
        return;
    }
    const bool inPlace = a.endsIn0 || ((u32(a.passes) - first) & 1u) == 0;
    const size_t begin = size_t(blockIdx.x) * kRepairTile;
    if (Whole && first == 4) repairTile<4>(a, sm, first, inPlace, begin, 0, a.n);
    else if (Whole && first < 4) repairTile<3>(a, sm, first, inPlace, begin, 0, a.n);
    else repairTile<0>(a, sm, first, inPlace, begin, 0, a.n);
}

template <int Threads>
struct LongShared
{
    u32 start[kRadix];
    u32 warp[Threads / 32][kRadix];
    u32 end;
    u32 differ;  // digits in which the run's keys differ
};

// A long run per CTA: an LSD radix sort of its remaining digits between its
// stretch of buffer 0 and the same stretch of buffer 1.  Digits all keys
// share are left out: the run is read once, eight keys of a thread in flight,
// to find them, and a run of equal keys is done then.  A run of 27k keys, most
// of them equal, took 267 us with a digit counted to see that it is shared and
// a key per thread and step; 17k such keys take 122 now, 50k 327.
template <int Threads>
__device__ __forceinline__ void sortLongRuns(const RepairArgs &a, LongShared<Threads> &sm, int first, u32 runs,
                                             const Team &team)
{
    constexpr int W = Threads / 32;
    constexpr int kLongItems = Threads == kLongThreads ? 4 : 2;  // keys per thread and step (2: no spills in the forest's sort)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int prefix = a.beginBit + first * kRadixBits;
    for (u32 r = team.rank; r < runs; r += team.size)
    {
        const u32 h = a.longList[2 * r], limit = a.longList[2 * r + 1];
        if (warp == 0)
        {
            // end of the run: first key whose high digits are larger
            const u64 mine = (a.k[0][h] & a.keyMask) >> prefix;
            u32 lo = h + 1, hi = limit;
            while (lo < hi)
            {
                const u32 len = hi - lo;
                const u32 p = lo + u32((u64(lane) + 1) * len / 33u);
                const unsigned in = __ballot_sync(0xffffffffu, ((a.k[0][p] & a.keyMask) >> prefix) == mine);
                const int c = __popc(in);  // a prefix of the lanes
                const u32 pLow = __shfl_sync(0xffffffffu, p, c > 0 ? c - 1 : 0);
                const u32 pHigh = __shfl_sync(0xffffffffu, p, c < 32 ? c : 31);
                if (c > 0) lo = pLow + 1;
                if (c < 32) hi = pHigh;
            }
            if (lane == 0)
            {
                sm.end = lo;
                sm.differ = 0;
            }
        }
        __syncthreads();
        const u32 e = sm.end;
        {
            const u64 head = a.k[0][h];
            u64 diff = 0;
            for (u32 i = h + tid; i < e; i += 8 * Threads)
            {
                u64 k[8];
#pragma unroll
                for (u32 q = 0; q < 8; ++q) k[q] = a.k[0][min(i + q * Threads, e - 1)];
#pragma unroll
                for (u32 q = 0; q < 8; ++q) diff |= k[q] ^ head;
            }
            u32 digits = 0;
            for (int d = 0; d < first; ++d)
                if (((diff & a.keyMask) >> (a.beginBit + d * kRadixBits)) & (kRadix - 1)) digits |= 1u << d;
            if (digits) atomicOr(&sm.differ, digits);
        }
        __syncthreads();
        const u32 differ = sm.differ;
        int at = 0;  // buffer that holds the run
        for (int d = 0; d < first; ++d)
        {
            if (!(differ & (1u << d))) continue;
            const int shift = a.beginBit + d * kRadixBits;
            const u64 *in = at ? a.k[1] : a.k[0];
            const u32 *inV = at ? a.v[1] : a.v[0];
            u64 *out = at ? a.k[0] : a.k[1];
            u32 *outV = at ? a.v[0] : a.v[1];
            if (tid < kRadix) sm.start[tid] = 0;
            __syncthreads();
            for (u32 i = h + tid; i < e; i += 4 * Threads)
            {
                u64 k[4];
#pragma unroll
                for (u32 q = 0; q < 4; ++q) k[q] = in[min(i + q * Threads, e - 1)];
#pragma unroll
                for (u32 q = 0; q < 4; ++q)
                    if (i + q * Threads < e) atomicAdd(&sm.start[unsigned(k[q] >> shift) & (kRadix - 1)], 1u);
            }
            __syncthreads();
            if (warp == 0)
            {
                // exclusive scan of the counts, eight per lane
                u32 c[8], sum = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                {
                    c[k] = sm.start[lane * 8 + k];
                    sum += c[k];
                }
                u32 inc = sum;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1)
                {
                    const u32 t = __shfl_up_sync(0xffffffffu, inc, off);
                    if (lane >= off) inc += t;
                }
                u32 run = h + inc - sum;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                {
                    sm.start[lane * 8 + k] = run;
                    run += c[k];
                }
            }
            // tiles of kLongItems keys per thread, a warp's 32 x kLongItems in a row
            for (u32 i0 = h; i0 < e; i0 += Threads * kLongItems)
            {
                for (int k = tid; k < W * kRadix; k += Threads) (&sm.warp[0][0])[k] = 0;
                u64 key[kLongItems];
                u32 val[kLongItems], rank[kLongItems];
                const u32 w0 = i0 + u32(warp) * 32 * kLongItems + lane;
#pragma unroll
                for (int q = 0; q < kLongItems; ++q)
                {
                    const u32 i = min(w0 + q * 32, e - 1);
                    key[q] = in[i];
                    val[q] = inV[i];
                }
                __syncthreads();
#pragma unroll
                for (int q = 0; q < kLongItems; ++q)
                {
                    const unsigned digit = unsigned(key[q] >> shift) & (kRadix - 1);
                    const unsigned validMask = __ballot_sync(0xffffffffu, w0 + q * 32 < e);
                    const unsigned peers = peerLanes<kRadixBits>(digit) & validMask;
                    const u32 before = sm.warp[warp][digit];
                    const unsigned under = __popc(peers & laneMaskLt());
                    rank[q] = before + under;
                    __syncwarp();
                    if ((validMask >> lane & 1u) && under == 0) sm.warp[warp][digit] = before + __popc(peers);
                    __syncwarp();
                }
                __syncthreads();
                if (tid < kRadix)
                {
                    u32 acc = sm.start[tid];
#pragma unroll
                    for (int w = 0; w < W; ++w)
                    {
                        const u32 c = sm.warp[w][tid];
                        sm.warp[w][tid] = acc;
                        acc += c;
                    }
                    sm.start[tid] = acc;
                }
                __syncthreads();
#pragma unroll
                for (int q = 0; q < kLongItems; ++q)
                {
                    if (w0 + q * 32 >= e) break;
                    const u32 to = sm.warp[warp][unsigned(key[q] >> shift) & (kRadix - 1)] + rank[q];
                    out[to] = key[q];
                    outV[to] = val[q];
                }
                __syncthreads();
            }
            at ^= 1;
        }
        __syncthreads();
        if (at)
        {
            for (u32 i = h + tid; i < e; i += Threads)
            {
                const u64 key = a.k[1][i];
                a.k[0][i] = key;
                a.v[0][i] = a.v[1][i];
                if (a.sample && (i & (kSampleStride - 1)) == 0) a.sample[i >> kSampleShift] = key;
            }
        }
        else if (a.sample)
        {
            for (u32 j = ((h + kSampleStride - 1) >> kSampleShift) + tid; (j << kSampleShift) < e; j += Threads)
                a.sample[j] = a.k[0][j << kSampleShift];
        }
        __syncthreads();
    }
}

static __global__ void __launch_bounds__(kLongThreads) longRunKernel(RepairArgs a)
{
    __shared__ LongShared<kLongThreads> sm;
    if (*a.error) return;
    sortLongRuns(a, sm, int(a.ctl->first), a.ctl->longRuns, wholeGrid());
}

// The repair of a planned sort (after its passes).
static inline unsigned repairTiles(size_t n) { return unsigned((n + kRepairTile - 1) / kRepairTile); }
}  // namespace sort
}  // namespace aot
