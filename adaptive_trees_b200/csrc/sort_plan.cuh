// sort_plan.cuh -- which digits of the keys a sort has to pass over.
//
// A radix sort of all 64 bits makes 8 passes, but n keys in space-filling
// curve order are told apart by their high digits: 16Mi Plummer particles by
// the first 32 bits, up to runs of a few dozen keys.  A sort with a plan
// passes over the last D digits only (an LSD sort of the high 8 D bits,
// stable), and the repair (sort_repair.cuh) orders the keys inside each run
// of equal high digits.  The result is the sort's whatever the plan is; the
// plan decides the time alone.
//
// The cost of the repair grows with the mean length of the run a key is in,
// R_D = sum of (run length)^2 / n.  It is estimated from M keys at random
// positions: two of them fall into the same run with probability R_D / n, so
// M keys hold about M^2 / 2n x R_D pairs that share their high digits.  Pairs
// of equal keys need no repair and are taken off (also positions drawn
// twice); keys that repeat so often that their runs would be long send the
// sort to all passes.
//
// The sample counts the keys that find an earlier one of their prefix.  That is
// the pairs where a prefix is drawn twice, but k - 1 of k (k - 1) / 2 where it is
// drawn k times, and a run that holds a share p of the keys is drawn p M times:
// R_D has n p^2 of it.  So each CTA also counts the pairs beyond among its own
// keys.  (Without them a tenth of 130k keys in one cell looked like a mean run
// of 34 instead of 1300 keys, and a CTA sorted it: 248 us, all passes take 110.)
#pragma once

#include "radix_sort.cuh"

namespace aot
{
namespace sort
{
constexpr int kPlanThreads = 256;      // a sampled key per thread
constexpr u32 kPlanMaxSamples = 8192;
constexpr int kPlanMinPasses = 2;
constexpr int kPlanMaxPasses = 6;
// Pair sorts of at most this many digits make no plan: it can leave out two
// passes of them at best, and costs a launch and a repair.  Random keys, four
// digits, with a plan and without: replayed 10k keys 33 and 31 us, 700k 68 and
// 66, 5M 187 and 186, queued 2M 132 and 113; three digits 33 and 25, 62 and 53,
// 154 and 145, 103 and 93.  Five digits: 35 and 35, 72 and 76, 189 and 225, 132
// and 135.
constexpr int kUnplannedPasses = 4;
constexpr int kPlanSets = kPlanMaxPasses - kPlanMinPasses + 2;  // a set of prefixes per choice, one of whole keys
// Cost in passes: the repair's fixed part and its part per key of the mean
// run.  Measured at 16Mi keys (a pass 120 us): repairs of mean runs of 3.8,
// 4.7 and 14.4 keys took 116, 130 and 272 us (the first takes 109 now).
constexpr float kRepairCost = 0.55f;
constexpr float kRunCost = 0.11f;
// Mean run of equal keys above which all passes run: they share their run with
// keys that are not equal, and a long run is a CTA's work in the repair.  In
// the sample a single stack of equal keys shows by its share of them, so this
// is 32 of M sampled keys: 0.4 % of 16Mi keys, 4 % of 130k.
constexpr float kMaxRepeats = 16.f;

// splitmix64's finaliser
__host__ __device__ __forceinline__ u64 mix64(u64 x)
{
    x ^= x >> 30;
    x *= 0xBF58476D1CE4E5B9ull;
    x ^= x >> 27;
    x *= 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// Keys sampled of n: about 2 n pairs, so that a mean run of one key more is
// seen about twice (n up to 16Mi).
inline u32 planSamples(size_t n)
{
    u32 m = 64;
    while (m < kPlanMaxSamples && u64(m) * m < 4 * u64(n)) m += 64;
    return m;
}
// slots of one set of the sampled prefixes (2^k, at least four per sample)
inline u32 planSlotBits(size_t n)
{
    u32 bits = 8;
    while ((u32(1) << bits) < 4 * planSamples(n)) ++bits;
    return bits;
}
inline size_t planTableBytes(size_t n) { return (size_t(kPlanSets) << planSlotBits(n)) * sizeof(u64); }

// Counters of one plan (zero between sorts: the last CTA clears them).
struct PlanCounters
{
    u32 repeats[kPlanSets];  // sampled keys whose prefix another one holds already
    u32 more[kPlanSets];     // pairs beyond them among the keys of a CTA
    u32 done;                // CTAs that have counted
};

// The sample and its sets.
struct PlanArgs
{
    u64 *table;  // [kPlanSets][1 << slotBits]: sort number << 32 | the last prefix hashed there
    PlanCounters *counters;
    u32 samples, slotBits;
    int force = -1;  // first pass to run whatever the sample says (self-tests), or -1
};

// The prefixes of a CTA's sampled keys, for the pairs beyond.  Small: with 512
// slots and as many counts, 24 KB, a plan of 16Mi keys took 17 us instead of
// 12, even when it left them alone (another split of the SM's memory).
constexpr u32 kPlanLocalBits = 8;
struct PlanShared
{
    u32 word[kPlanSets][1u << kPlanLocalBits];         // the last prefix hashed there
    u32 finds[kPlanSets][1u << (kPlanLocalBits - 2)];  // keys that found their prefix there
    u32 repeats[kPlanSets], more[kPlanSets];
};

// The first pass to run (0: all `passes`) for n keys, from the counts of each
// set (set 0: whole keys; set s: prefixes of kPlanMinPasses + s - 1 digits).
__host__ __device__ __forceinline__ u32 planFirst(const u32 *repeats, const u32 *more, u32 m, size_t n,
                                                  int passes = kMaxPasses)
{
    const float perPair = 2.f * float(n) / (float(m) * float(m));  // mean run per pair
    if (float(repeats[0]) * perPair > kMaxRepeats) return 0;
    // pairs of sampled keys for each pair within a CTA
    const u32 whole = m / kPlanThreads, rest = m % kPlanThreads;
    const float scale = float(m) * float(m - 1) /
                        (float(whole) * kPlanThreads * (kPlanThreads - 1) + float(rest) * float(rest ? rest - 1 : 0));
    const float equal = float(repeats[0]) + float(more[0]) * scale;
    float best = float(passes);
    u32 first = 0;
    for (int d = kPlanMinPasses; d <= kPlanMaxPasses && d < passes; ++d)
    {
        const int set = d - kPlanMinPasses + 1;
        const float pairs = float(repeats[set]) + float(more[set]) * scale;
        const float run = pairs > equal ? (pairs - equal) * perPair : 0.f;
        const float cost = float(d) + kRepairCost + kRunCost * run;
        if (cost < best)
        {
            best = cost;
            first = u32(passes - d);
        }
    }
    return first;
}

// Position of sampled key i among n: drawn at random, so that the order the
// keys are stored in (often along the curve already) does not matter.
__device__ __forceinline__ size_t planPosition(u32 i, size_t n)
{
    return size_t(__umul64hi(mix64(u64(i) * 0x9E3779B97F4A7C15ull + 0x2545F4914F6CDD1Dull), u64(n)));
}

// This CTA's part of the sample: keyAt(i, group) is the key at position i and
// the segment it is sorted in.  A sample per thread, over many
// CTAs (one CTA took 84 us for 8192: its random loads and shared-memory
// atomics go through one SM), and one exchange per sample and set, all of a
// thread's in flight together: a slot holds the last prefix that was hashed
// to it, so a repeat is missed where another prefix took the slot in between
// (at most a quarter of the slots are used), which an estimate can bear;
// sets with probing took 34-48 us in chains of L2 round trips.  Words of
// earlier sorts (epoch: the number of this one) match no prefix of this one,
// so nothing is cleared.
template <class KeyAt>
__device__ __forceinline__ void planSample(const KeyAt &keyAt, size_t n, const PlanArgs &a, u32 epoch, PlanShared &sm)
{
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    static_assert(sizeof(PlanShared) % sizeof(u32) == 0, "words");
    for (u32 k = threadIdx.x; k < sizeof(PlanShared) / sizeof(u32); k += blockDim.x) reinterpret_cast<u32 *>(&sm)[k] = 0;
    __syncthreads();
    u32 group = 0;
    u64 key = 0;
    const bool valid = i < a.samples;
    if (valid) key = keyAt(planPosition(i, n), group);
    u64 old[kPlanSets], word[kPlanSets];
#pragma unroll
    for (int set = 0; set < kPlanSets; ++set)
    {
        const int shift = set == 0 ? 0 : 64 - (kPlanMinPasses + set - 1) * kRadixBits;
        const u64 h = mix64((key >> shift) * 0x9E3779B97F4A7C15ull + group);
        word[set] = (u64(epoch) << 32) | u32(h);  // the low half stands for the prefix, the high bits pick the slot
        old[set] = 0;
        if (valid)
            old[set] = atomicExch(
                reinterpret_cast<unsigned long long *>(a.table + (size_t(set) << a.slotBits) + (h >> (64 - a.slotBits))),
                (unsigned long long)word[set]);
    }
    // (while the exchanges are on their way)
    static_assert(kPlanSets % 2 == 0 && kPlanThreads <= 256, "two sets' pairs of a warp in a word");
    u32 more[kPlanSets / 2] = {};
#pragma unroll
    for (int set = 0; set < kPlanSets; ++set)
    {
        const u32 mine = u32(word[set]) | 1u, at = mine >> (32 - kPlanLocalBits);
        if (valid && atomicExch(&sm.word[set][at], mine) == mine)
            more[set / 2] += atomicAdd(&sm.finds[set][at / 4], 1u) << (16 * (set % 2));
    }
    u32 any = 0;
#pragma unroll
    for (int k = 0; k < kPlanSets / 2; ++k) any |= more[k];
    if (__any_sync(0xffffffffu, any))
    {
#pragma unroll
        for (int k = 0; k < kPlanSets / 2; ++k)
        {
            const u32 pairs = __reduce_add_sync(0xffffffffu, more[k]);
            if ((threadIdx.x & 31) == 0 && pairs)
            {
                atomicAdd(&sm.more[2 * k], pairs & 0xffffu);
                atomicAdd(&sm.more[2 * k + 1], pairs >> 16);
            }
        }
    }
#pragma unroll
    for (int set = 0; set < kPlanSets; ++set)
    {
        const u32 c = u32(__popc(__ballot_sync(0xffffffffu, old[set] == word[set])));
        if ((threadIdx.x & 31) == 0 && c) atomicAdd(&sm.repeats[set], c);
    }
    __syncthreads();
    if (threadIdx.x < kPlanSets)
    {
        if (sm.repeats[threadIdx.x]) atomicAdd(&a.counters->repeats[threadIdx.x], sm.repeats[threadIdx.x]);
        if (sm.more[threadIdx.x]) atomicAdd(&a.counters->more[threadIdx.x], sm.more[threadIdx.x]);
    }
}

// Start of a sort of n keys: the digit counts are cleared and the keys
// sampled by all CTAs, the plan made and the control block set up by the last.
template <class KeyAt>
__device__ __forceinline__ void planSort(const KeyAt &keyAt, size_t n, const PlanArgs &a, SortControl *ctl, u32 *hist,
                                         size_t histWords, int passes = kMaxPasses)
{
    __shared__ PlanShared sm;
    __shared__ u32 sRepeats[kPlanSets], sMore[kPlanSets];
    __shared__ bool sLast;
    const u32 epoch = ctl->epoch + kEpochStep;  // this sort's number (set at the end)
    for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < histWords; k += size_t(gridDim.x) * blockDim.x)
        hist[k] = 0;
    planSample(keyAt, n, a, epoch, sm);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) sLast = atomicAdd(&a.counters->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!sLast) return;
    __threadfence();
    if (threadIdx.x < kPlanSets)
    {
        sRepeats[threadIdx.x] = __ldcg(&a.counters->repeats[threadIdx.x]);
        sMore[threadIdx.x] = __ldcg(&a.counters->more[threadIdx.x]);
        a.counters->repeats[threadIdx.x] = a.counters->more[threadIdx.x] = 0;
    }
    if (threadIdx.x < kPassSlots) ctl->tileCounters[threadIdx.x] = 0;
    clearBarriers(ctl);
    __syncthreads();
    if (threadIdx.x == 0)
    {
        a.counters->done = 0;
        ctl->first = a.force >= 0 ? u32(a.force) : planFirst(sRepeats, sMore, a.samples, n, passes);
        ctl->epoch = epoch;
        ctl->longRuns = 0;
        ctl->keygenDone = 0;
    }
}

// Start of a planned pair sort by bits [beginBit, beginBit + 8 passes) of
// keyMask: the digits sampled are those of the passes.
static __global__ void __launch_bounds__(kPlanThreads)
    planPairsKernel(const u64 *__restrict__ keys, size_t n, int beginBit, int passes, u64 keyMask, PlanArgs plan,
                    SortControl *ctl)
{
    const int up = 64 - passes * kRadixBits;
    const auto keyAt = [&](size_t i, u32 &) { return ((keys[i] & keyMask) >> beginBit) << up; };
    planSort(keyAt, n, plan, ctl, nullptr, 0, passes);
}
}  // namespace sort
}  // namespace aot
