// radix_sort.cuh -- onesweep LSD radix sort of 64-bit keys carrying 32-bit values.
//
// Replaces cub::DeviceRadixSort::SortPairs on the particle keys
// (octree.cu:301-304, kdtree3d.cu:168-170) and on the view's internal-node keys
// (tree_view.cu:664-689).  Stable: equal keys keep their input order, which
// for the particle sort makes Perm ascend within runs of equal keys.
//
// Structure (one read of the keys per digit):
//   1. a histogram kernel counts all digit positions at once (fused into key
//      generation for the particle sort with 8-bit digits, so the keys are
//      never re-read);
//   2. a tiny kernel turns the counts into per-digit global start offsets;
//   3. one onesweep kernel per digit: each CTA takes a tile of keys in
//      arrival order (atomic tile counter), ranks them per warp with ballots,
//      publishes its per-digit counts, reorders the keys in shared memory,
//      resolves its global offsets by decoupled look-back over earlier tiles
//      (while the tile's values are on their way), reorders the values and
//      writes digit runs out contiguously.
// What bounds a pass is the shared-memory pipe and the issue slots, not HBM
// (16Mi pairs, ncu: shared memory 81 % busy with an atomic-or match, DRAM
// 32 %): about 40 shared-memory wavefronts and 100 instructions per 32 keys.
// Measured at 16Mi pairs, per pass: 156 us before, with the values staged by a
// bulk copy, the ballots left to the compiler and the tile's bounds checked
// for every key; 147 us with the values loaded behind the key reorder; 136 us
// with one lookup for a key's place instead of two and tiles of 3584 keys;
// 120 us with the ballots written out (peerLanes) and tiles of 4096; 117.5 us
// with the warp's counter read by all lanes instead of shuffled (3.4 TB/s).
// Not faster: __match_any_sync (182 us), matching by shared atomic-or (133-138),
// 512 threads (138), tiles of 4608-6144 keys (117-124).
// The digit width and the keys per thread are template parameters; the
// configurations compiled in are listed in kSortConfigs, and the sort tuner
// (sortTune in engine.cu) picks one per device and problem size by timing them.
//
// A sort that has a plan (sort_plan.cuh) runs only the passes of its high
// digits and leaves the rest to a repair of the short runs of equal high
// digits (sort_repair.cuh).  Every pass is launched and reads the plan on the
// device; the ones it leaves out return at once.
// The look-back wait is bounded: after kLookbackSpins polls it records
// kErrLookback in the device error word and proceeds, so a broken invariant
// surfaces as an error status instead of a hung GPU.
#pragma once

#include "common.cuh"
#include "grid_barrier.cuh"

namespace aot
{
namespace sort
{
constexpr int kRadixBits = 8;              // digit width of the default configuration
constexpr int kRadix = 1 << kRadixBits;     // largest radix: stride of every per-pass digit array
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 10;                  // keys per thread of the default configuration
constexpr int kTile = kThreads * kItems;
constexpr int kMaxPasses = 8;               // passes of 8-bit digits over 64-bit keys
constexpr int kPassSlots = 10;              // most passes of any configuration (7-bit digits)
constexpr int kMinTile = kThreads * 8;      // smallest tile of any configuration
constexpr u64 kFlagAgg = u64(1) << 62;
constexpr u64 kFlagPrefix = u64(2) << 62;
constexpr u64 kFlagMask = u64(3) << 62;
// A status word is flag (2 bits) | tag (30 bits) | count (32 bits).  The tag
// numbers the pass that wrote it, so one array serves every pass of every
// sort without being cleared between them: a word of another pass reads as
// not published.  (Cleared arrays of 8 passes were 107 MB of writes and 28 us
// of a 16Mi sort; one pass' words are 13 MB and stay in L2.)
// (The first number is 1: a cleared word carries no pass' tag.)
constexpr u64 kTagMask = ((u64(1) << 30) - 1) << 32;
__host__ __device__ constexpr u64 passTag(u32 number) { return (u64(number + 1) << 32) & kTagMask; }
constexpr unsigned kLookbackSpins = 1u << 22;
constexpr int kLookbackWindow = 8;

__device__ __forceinline__ u64 ldRelaxed(const u64 *p)
{
    u64 v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void stRelaxed(u64 *p, u64 v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned laneMaskLt()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Control block of one sort, in device memory.
struct SortControl
{
    u32 epoch;      // number of the sort: pass slot j writes tag epoch + j (the only word kept between sorts)
    u32 first;      // the passes run are first .. passes - 1 (0: all of them)
    u32 longRuns;   // runs the repair left to the long-run kernel
    u32 keygenDone; // CTAs of the key generation that have added their digit counts
    u32 tileCounters[kPassSlots];
    GridBarrier sortBar;   // of the passes and the repair in one launch
    GridBarrier afterBar;  // of what follows the sort in one launch (update())
};
constexpr u32 kEpochStep = 16;  // tags per sort (>= kPassSlots)
static_assert(kEpochStep >= kPassSlots && (u64(1) << 30) % kEpochStep == 0, "a tag per pass slot");

// Zeroes the barriers of a sort and of what follows it (one CTA, before them).
__device__ __forceinline__ void clearBarriers(SortControl *ctl)
{
    static_assert(sizeof(GridBarrier) % sizeof(u32) == 0, "words");
    constexpr u32 kWords = sizeof(GridBarrier) / sizeof(u32);
    for (u32 i = threadIdx.x; i < kWords; i += blockDim.x)
    {
        reinterpret_cast<u32 *>(&ctl->sortBar)[i] = 0;
        reinterpret_cast<u32 *>(&ctl->afterBar)[i] = 0;
    }
}

// Start of a sort without a plan: every pass runs.
static __global__ void __launch_bounds__(kThreads) beginSortKernel(SortControl *ctl, u32 *hist)
{
    if (hist)
        for (int i = threadIdx.x; i < kPassSlots * kRadix; i += blockDim.x) hist[i] = 0;
    if (threadIdx.x < kPassSlots) ctl->tileCounters[threadIdx.x] = 0;
    clearBarriers(ctl);
    if (threadIdx.x == 0)
    {
        ctl->first = 0;
        ctl->epoch += kEpochStep;
        ctl->longRuns = 0;
        ctl->keygenDone = 0;
    }
}

// Histogram of the Bits-wide digits of keys[0, n) for the passes run of those
// covering [beginBit, endBit); pass p's counts go to hist[p * kRadix + digit].
template <int Bits = kRadixBits>
static __global__ void __launch_bounds__(kThreads) histogramKernel(const u64 *__restrict__ keys, size_t n, int beginBit,
                                                             int passes, u32 *__restrict__ hist, int endBit,
                                                             const SortControl *ctl)
{
    const int first = int(ctl->first);
    constexpr int R = 1 << Bits;
    __shared__ u32 sh[kPassSlots][R];
    for (int i = threadIdx.x; i < kPassSlots * R; i += kThreads) (&sh[0][0])[i] = 0;
    __syncthreads();
    for (size_t i = blockIdx.x * size_t(kThreads) + threadIdx.x; i < n; i += size_t(gridDim.x) * kThreads)
    {
        const u64 k = __ldg(keys + i);
        for (int p = first; p < passes; ++p)
        {
            const int shift = beginBit + p * Bits;
            const int bits = endBit - shift < Bits ? endBit - shift : Bits;
            atomicAdd(&sh[p][(k >> shift) & ((1u << bits) - 1)], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * R; i += kThreads)
    {
        const u32 v = (&sh[0][0])[i];
        if (v) atomicAdd(hist + (i / R) * kRadix + (i % R), v);
    }
}

// Exclusive scan of each pass' 256 digit counts (a narrower radix leaves the
// upper counts zero, so their starts are unused).  A warp per pass, eight
// counts per lane, two an access: the counts and the starts of a pair sort lie
// in the caller's scratch, of which 8-byte alignment is all that is asked.
// __ldcg: the counts may come from other CTAs' atomics.
__device__ __forceinline__ void scanBins(const u32 *hist, u32 *bins, int firstPass, int passes)
{
    static_assert(kRadix == 256, "eight counts per lane");
    const int lane = threadIdx.x & 31;
    for (int p = firstPass + int(threadIdx.x >> 5); p < passes; p += int(blockDim.x >> 5))
    {
        const uint2 *h = reinterpret_cast<const uint2 *>(hist + p * kRadix) + lane * 4;
        uint2 c[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) c[i] = __ldcg(h + i);
        u32 sum = 0, e[8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            e[2 * i] = sum;
            e[2 * i + 1] = sum + c[i].x;
            sum += c[i].x + c[i].y;
        }
        u32 inc = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
        {
            const u32 t = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += t;
        }
        const u32 base = inc - sum;
        uint2 *o = reinterpret_cast<uint2 *>(bins + p * kRadix) + lane * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = make_uint2(base + e[2 * i], base + e[2 * i + 1]);
    }
}

static __global__ void __launch_bounds__(kThreads) binsKernel(const u32 *__restrict__ hist, u32 *__restrict__ bins,
                                                              int passes)
{
    scanBins(hist, bins, 0, passes);
}

template <int Bits, int Items>
struct SharedPass
{
    static constexpr int R = 1 << Bits;
    static constexpr int T = kThreads * Items;
    u64 keys[T];
    u32 vals[T];
    u32 warpStart[kWarps][R];  // per-warp digit counts, then the tile-local start of each warp's digit
    u32 localStart[R];
    u32 gstart[R];             // global position of local index 0 of each digit (mod 2^32)
    u32 warpSums[kWarps];
    u32 tile;
};

// The compiled configurations: digit width, keys per thread and the CTAs per
// SM they are built for (their shared memory and a 64-register budget allow
// 4 CTAs for tiles of up to 3072 keys).  Each gives an even number of passes
// over 64-bit keys (8 or 10), so the sorted data ends where it started.
struct SortConfig
{
    int bits, items;
};
constexpr SortConfig kSortConfigs[] = {{8, 10}, {8, 16}, {8, 8}, {7, 12}, {7, 16}};
constexpr int kNumSortConfigs = int(sizeof(kSortConfigs) / sizeof(kSortConfigs[0]));
constexpr int kDefaultSortConfig = 0;
// The configuration of a sort no tuning has chosen one for: tiles of 4096
// keys from a million keys on (64-bit pair sorts: 700k keys 108 us with 2560,
// 112 with 4096; 1M 125 and 118; 4M 309 and 276; 16Mi 1135 and 1018).
constexpr int defaultSortConfig(size_t n) { return n >= (size_t(1) << 20) ? 1 : kDefaultSortConfig; }
constexpr int configTile(int c) { return kThreads * kSortConfigs[c].items; }
constexpr int configPasses(int c, int bits = 64)
{
    return (bits + kSortConfigs[c].bits - 1) / kSortConfigs[c].bits;
}

// Lanes of the warp whose Bits-wide digit equals this lane's: a ballot per
// digit bit.  Written out as test, ballot, select and one three-input AND-XOR
// per bit: the compiler's version of the same took 16 us more of a 136 us pass.
template <int Bits>
__device__ __forceinline__ unsigned peerLanes(unsigned digit)
{
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < Bits; ++b)
    {
        unsigned lanes, other;  // lanes with the bit set; zero (this lane has it) or all ones
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b32 t;\n\tand.b32 t, %2, %3;\n\tsetp.ne.u32 p, t, 0;\n\t"
            "vote.sync.ballot.b32 %0, p, 0xffffffff;\n\tselp.b32 %1, 0, 0xffffffff, p;\n\t}"
            : "=r"(lanes), "=r"(other)
            : "r"(digit), "r"(1u << b));
        asm("lop3.b32 %0, %0, %1, %2, 0x60;" : "+r"(peers) : "r"(lanes), "r"(other));  // peers & (lanes ^ other)
    }
    return peers;
}

// A tile: the keys [base, base + count) (at most Tile), whether it starts a
// look-back chain (publishes an inclusive prefix at once), the global start
// of each digit, and what is subtracted from a generated value's key index.
struct TileRange
{
    u32 base, count;
    bool chainStart;
    const u32 *digitBase;
    u32 valueOffset;
};

// Tiles of a pass over one contiguous key array keys[0, n).
template <int Tile>
struct ContiguousTiles
{
    size_t n;
    const u32 *bins;  // [radix] global start of each digit
    __device__ __forceinline__ TileRange at(u32 tile) const
    {
        const size_t b = size_t(tile) * Tile, left = n - b;
        return {u32(b), left < size_t(Tile) ? u32(left) : u32(Tile), tile == 0, bins, 0u};
    }
};

// Tiles of a segmented pass (the systems of a forest): tile t holds
// the keys [tileBegin[t], tileEnd[t]) of segment tileSeg[t] (at most one tile,
// never straddling segments); a look-back chain ends at the segment's first
// tile; digit starts are per segment, and generated values are indices within
// the segment.
struct SegmentTiles
{
    const u32 *tileSeg, *tileBegin, *tileEnd, *segFirstTile, *segBase;
    const u32 *bins;  // [segments][kRadix] global start of each digit of this pass
    __device__ __forceinline__ TileRange at(u32 tile) const
    {
        const u32 seg = __ldg(tileSeg + tile), b = __ldg(tileBegin + tile);
        return {b, __ldg(tileEnd + tile) - b, tile == __ldg(segFirstTile + seg), bins + size_t(seg) * kRadix,
                __ldg(segBase + seg)};
    }
};

// One onesweep pass: the digit at bit `shift` (`bits` <= Bits wide) of a tile
// of `tiles`, Items keys per thread.  valsIn == nullptr
// means values are generated (first pass).  Threads below the radix own one
// digit each in the per-digit steps.  The places behind a short tile's keys
// hold the largest digit, so that they rank last, and are not written; their
// counts reach no later tile (a short tile ends its chain).  A look-back that polls an unpublished
// tile more than spinLimit times records kErrLookback and goes on with the
// prefix it has: every write stays inside the output, the result is wrong
// and the host reports the error.  A persistent CTA calls it, with a
// __syncthreads between, until it returns
// false: the tile counter has passed numTiles (which a launch of one CTA per
// tile never reaches).
template <int Bits, int Items, class Tiles>
__device__ __forceinline__ bool onesweepTile(const Tiles &tiles, const u64 *__restrict__ keysIn,
                                             const u32 *__restrict__ valsIn, u64 *__restrict__ keysOut,
                                             u32 *__restrict__ valsOut, int shift, u32 *tileCounter, u64 *status,
                                             u64 tag, int *error, int bits, unsigned spinLimit = kLookbackSpins,
                                             u32 numTiles = 0xffffffffu)
{
    using Smem = SharedPass<Bits, Items>;
    constexpr int R = Smem::R;
    constexpr int T = Smem::T;
    static_assert(R <= kThreads && R <= kRadix, "one digit per thread");
    static_assert(Items % 2 == 0 && T <= 0x10000, "ranks and places are packed in pairs");
    const unsigned dmask = (1u << bits) - 1;
    extern __shared__ __align__(16) unsigned char smemRaw[];
    Smem &sm = *reinterpret_cast<Smem *>(smemRaw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    for (int i = tid; i < kWarps * R; i += kThreads) (&sm.warpStart[0][0])[i] = 0;
    if (tid == 0) sm.tile = atomicAdd(tileCounter, 1u);
    __syncthreads();
    const u32 tile = sm.tile;
    if (tile >= numTiles) return false;
    const TileRange r = tiles.at(tile);
    const u32 at = u32(warp) * (32 * Items) + u32(lane);  // this lane's first key in the tile, then every 32nd
    const bool full = r.count == u32(T);

    u64 key[Items];
    {
        const u64 *in = keysIn + r.base + at;
        if (full)
        {
#pragma unroll
            for (int i = 0; i < Items; ++i) key[i] = __ldcs(in + i * 32);
        }
        else
        {
#pragma unroll
            for (int i = 0; i < Items; ++i) key[i] = at + u32(i) * 32 < r.count ? __ldcs(in + i * 32) : ~u64(0);
        }
    }
    // Rank within the warp, items in memory order (item-major, lane-minor):
    // every lane reads its digit's counter of the warp, then the first lane
    // of each digit group adds the group's size.
    u32 *warpCount = sm.warpStart[warp];
    const unsigned ltMask = laneMaskLt();
    u32 place2[Items / 2];  // rank, later place in the tile: two of 16 bits
#pragma unroll
    for (int i = 0; i < Items; ++i)
    {
        const unsigned d = unsigned(key[i] >> shift) & dmask;
        const unsigned peers = peerLanes<Bits>(d);
        const u32 before = warpCount[d];
        __syncwarp();
        const u32 inGroup = __popc(peers & ltMask);
        if (inGroup == 0) warpCount[d] = before + __popc(peers);
        __syncwarp();
        const u32 rank = before + inGroup;
        if (i & 1) place2[i >> 1] |= rank << 16;
        else place2[i >> 1] = rank;
    }
    __syncthreads();
    // Per digit (thread = digit): the tile's count, published at once (a
    // chain's first tile publishes final prefixes; the look-back comes last,
    // so earlier tiles have had time to publish theirs); the tile-local start
    // of the digit and of each warp's part of it.
    u32 count = 0;
    {
        const int d = tid;
        u32 c[kWarps];
        if (d < R)
        {
#pragma unroll
            for (int w = 0; w < kWarps; ++w) c[w] = sm.warpStart[w][d];
#pragma unroll
            for (int w = 0; w < kWarps; ++w) count += c[w];
            stRelaxed(status + size_t(tile) * R + d, (r.chainStart ? kFlagPrefix : kFlagAgg) | tag | u64(count));
        }
        u32 v = count;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1)
        {
            const u32 t = __shfl_up_sync(0xffffffffu, v, off);
            if (lane >= off) v += t;
        }
        if (lane == 31) sm.warpSums[warp] = v;
        __syncthreads();
        u32 run = v - count;
#pragma unroll
        for (int w = 0; w < kWarps; ++w)
            if (w < warp) run += sm.warpSums[w];
        if (d < R)
        {
            sm.localStart[d] = run;
#pragma unroll
            for (int w = 0; w < kWarps; ++w)
            {
                sm.warpStart[w][d] = run;
                run += c[w];
            }
        }
    }
    __syncthreads();
    // Reorder the keys in shared memory; the values are loaded behind them and
    // arrive during the look-back.
#pragma unroll
    for (int i = 0; i < Items; ++i)
    {
        const unsigned d = unsigned(key[i] >> shift) & dmask;
        const u32 rank = (place2[i >> 1] >> ((i & 1) * 16)) & 0xffffu;
        const u32 place = warpCount[d] + rank;
        sm.keys[place] = key[i];
        if (i & 1) place2[i >> 1] = (place2[i >> 1] & 0xffffu) | (place << 16);
        else place2[i >> 1] = (place2[i >> 1] & 0xffff0000u) | place;
    }
    u32 val[Items];
    if (valsIn)
    {
        const u32 *in = valsIn + r.base + at;
        if (full)
        {
#pragma unroll
            for (int i = 0; i < Items; ++i) val[i] = __ldcs(in + i * 32);
        }
        else
        {
#pragma unroll
            for (int i = 0; i < Items; ++i) val[i] = at + u32(i) * 32 < r.count ? __ldcs(in + i * 32) : 0u;
        }
    }
    else
    {
#pragma unroll
        for (int i = 0; i < Items; ++i) val[i] = r.base + at + u32(i) * 32 - r.valueOffset;
    }
    // Look-back: global start of each digit for this tile.
    if (tid < R)
    {
        const int d = tid;
        u32 excl = 0;  // keys are fewer than 2^32
        if (!r.chainStart)
        {
            // Walk back over earlier tiles, eight status words per round trip,
            // summing aggregates until an inclusive prefix is found (the
            // chain's first tile always holds one).
            long long j = (long long)tile - 1;
            unsigned spins = 0;
            while (j >= 0)
            {
                u64 w8[kLookbackWindow];
#pragma unroll
                for (int k = 0; k < kLookbackWindow; ++k)
                    w8[k] = j - k >= 0 ? ldRelaxed(status + size_t(j - k) * R + d) : (kFlagPrefix | tag);
                int k = 0;
                bool done = false;
#pragma unroll
                for (; k < kLookbackWindow; ++k)
                {
                    if ((w8[k] & kTagMask) != tag) break;  // not published in this pass
                    excl += u32(w8[k]);
                    if ((w8[k] & kFlagMask) == kFlagPrefix)
                    {
                        done = true;
                        break;
                    }
                }
                if (done) break;
                j -= k;
                if (k < kLookbackWindow)  // tile j has not published yet
                {
                    if (++spins > spinLimit)
                    {
                        atomicExch(error, kErrLookback);
                        break;
                    }
                    if (spins > 64) __nanosleep(64);
                }
            }
            stRelaxed(status + size_t(tile) * R + d, kFlagPrefix | tag | u64(excl + count));
        }
        // modulo 2^32: gstart + j is exact for every key of digit d
        sm.gstart[d] = r.digitBase[d] + excl - sm.localStart[d];
    }
#pragma unroll
    for (int i = 0; i < Items; ++i) sm.vals[(place2[i >> 1] >> ((i & 1) * 16)) & 0xffffu] = val[i];
    __syncthreads();
    if (full)
    {
#pragma unroll 4
        for (int i = 0; i < Items; ++i)
        {
            const int j = tid + i * kThreads;
            const u64 k = sm.keys[j];
            const u32 out = sm.gstart[unsigned(k >> shift) & dmask] + u32(j);
            keysOut[out] = k;
            valsOut[out] = sm.vals[j];
        }
    }
    else
    {
        for (int j = tid; j < int(r.count); j += kThreads)
        {
            const u64 k = sm.keys[j];
            const u32 out = sm.gstart[unsigned(k >> shift) & dmask] + u32(j);
            keysOut[out] = k;
            valsOut[out] = sm.vals[j];
        }
    }
    return true;
}

// CTAs per SM each configuration is built for.
template <int Bits, int Items>
constexpr int passMinBlocks()
{
    return Items <= 12 ? 4 : 3;
}

// One contiguous sort: the passes of digits [beginBit, endBit) over n keys.
// Slot j runs pass first + j, from the keys of slot j - 1 (slot 0: keysIn and
// valsIn, or the input indices as values where valsIn is nullptr).  Slot j
// writes buffer (j + 1) & 1; with endsIn0 the buffers alternate backwards from
// the last pass instead, which then writes buffer 0.
struct PassArgs
{
    const u64 *keysIn;
    const u32 *valsIn;
    u64 *k[2];
    u32 *v[2];
    size_t n;
    const u32 *bins;
    SortControl *ctl;
    u64 *status;  // one word per tile and digit of the radix
    int *error;
    int beginBit, endBit, passes;
    bool endsIn0;
};

template <int Bits, int Items>
static __global__ void __launch_bounds__(kThreads, passMinBlocks<Bits, Items>()) onesweepKernel(PassArgs p, int slot)
{
    const int first = int(p.ctl->first), pass = first + slot;
    if (pass >= p.passes) return;
    const int out = (p.endsIn0 ? p.passes - 1 - pass : slot + 1) & 1;
    const int shift = p.beginBit + pass * Bits;
    const u64 *keysIn = slot ? (out ? p.k[0] : p.k[1]) : p.keysIn;
    const u32 *valsIn = slot ? (out ? p.v[0] : p.v[1]) : p.valsIn;
    onesweepTile<Bits, Items>(ContiguousTiles<kThreads * Items>{p.n, p.bins + pass * kRadix}, keysIn, valsIn,
                              out ? p.k[1] : p.k[0], out ? p.v[1] : p.v[0], shift, p.ctl->tileCounters + slot,
                              p.status, passTag(p.ctl->epoch + u32(slot)), p.error, min(Bits, p.endBit - shift));
}

// Pass slot `slot` over the segments of a forest (`passes` in all): every
// segment is sorted on its own (stable within the segment), in place in the
// global arrays.  tiles.bins: [pass][segment][kRadix].
template <int Bits, int Items>
static __global__ void __launch_bounds__(kThreads, passMinBlocks<Bits, Items>())
    segmentOnesweepKernel(SegmentTiles tiles, PassArgs p, int slot, int segments)
{
    const int pass = int(p.ctl->first) + slot;
    if (pass >= p.passes) return;
    tiles.bins += size_t(pass) * size_t(segments) * kRadix;
    const int shift = pass * Bits;
    const bool odd = slot & 1;
    onesweepTile<Bits, Items>(tiles, odd ? p.k[1] : p.k[0], slot == 0 ? nullptr : odd ? p.v[1] : p.v[0],
                              odd ? p.k[0] : p.k[1], odd ? p.v[0] : p.v[1], shift, p.ctl->tileCounters + slot,
                              p.status, passTag(p.ctl->epoch + u32(slot)), p.error, min(Bits, 64 - shift));
}

// ---------------------------------------------------------------------------
// Host-side dispatch over kSortConfigs (one instantiation per configuration):
// X(index, digit bits, keys per thread), in the order of kSortConfigs.
// ---------------------------------------------------------------------------
#define AOT_SORT_CONFIGS(X) X(0, 8, 10) X(1, 8, 16) X(2, 8, 8) X(3, 7, 12) X(4, 7, 16)

inline size_t passSmem(int c)
{
    switch (c)
    {
#define AOT_CASE(i, B, I) \
    case i: return sizeof(SharedPass<B, I>);
        AOT_SORT_CONFIGS(AOT_CASE)
#undef AOT_CASE
    default: throw std::invalid_argument("sort: unknown configuration");
    }
}

// Opts every pass kernel of this translation unit into its dynamic shared
// memory, once per device.
static inline void setPassSmemAll()
{
    static bool done[64] = {};
    int dev = 0;
    AOT_CHECK(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && done[dev]) return;
#define AOT_CASE(i, B, I)                                                                                        \
    AOT_CHECK(cudaFuncSetAttribute(onesweepKernel<B, I>, cudaFuncAttributeMaxDynamicSharedMemorySize,           \
                                   int(sizeof(SharedPass<B, I>))));                                              \
    AOT_CHECK(cudaFuncSetAttribute(segmentOnesweepKernel<B, I>, cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                                   int(sizeof(SharedPass<B, I>))));
    AOT_SORT_CONFIGS(AOT_CASE)
#undef AOT_CASE
    if (dev >= 0 && dev < 64) done[dev] = true;
}

// Pass slot `slot` of a contiguous sort with configuration c.
static inline void launchPass(int c, cudaStream_t s, const PassArgs &p, int slot)
{
    const unsigned tiles = unsigned((p.n + size_t(configTile(c)) - 1) / size_t(configTile(c)));
    switch (c)
    {
#define AOT_CASE(i, B, I)                                                                                        \
    case i: onesweepKernel<B, I><<<tiles, kThreads, sizeof(SharedPass<B, I>), s>>>(p, slot); break;
        AOT_SORT_CONFIGS(AOT_CASE)
#undef AOT_CASE
    default: throw std::invalid_argument("sort: unknown configuration");
    }
}

// Pass slot `slot` of a segmented sort with configuration c over `numTiles` tiles.
static inline void launchSegmentPass(int c, cudaStream_t s, unsigned numTiles, const SegmentTiles &tiles,
                                     const PassArgs &p, int slot, int segments)
{
    switch (c)
    {
#define AOT_CASE(i, B, I)                                                                                        \
    case i:                                                                                                      \
        segmentOnesweepKernel<B, I><<<numTiles, kThreads, sizeof(SharedPass<B, I>), s>>>(tiles, p, slot,         \
                                                                                         segments);              \
        break;
        AOT_SORT_CONFIGS(AOT_CASE)
#undef AOT_CASE
    default: throw std::invalid_argument("sort: unknown configuration");
    }
}

// Histogram of configuration c's digits.
static inline void launchHistogram(int c, cudaStream_t s, unsigned blocks, const u64 *keys, size_t n, int beginBit, int passes,
                            u32 *hist, int endBit, const SortControl *ctl)
{
    if (kSortConfigs[c].bits == 8)
        histogramKernel<8><<<blocks, kThreads, 0, s>>>(keys, n, beginBit, passes, hist, endBit, ctl);
    else
        histogramKernel<7><<<blocks, kThreads, 0, s>>>(keys, n, beginBit, passes, hist, endBit, ctl);
}

}  // namespace sort
}  // namespace aot
