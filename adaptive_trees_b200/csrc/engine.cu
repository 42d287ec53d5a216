// engine.cu -- host orchestration of the B200 adaptive-tree engine.
//
// Follows the reference's control flow for build/update/views
// (octree.cu:427-551, kdtree3d.cu:227-297, tree_view.cu:814-1134) with
// B200-specific choices:
//   * keygen + onesweep sort replace computeSfcKeys + CUB SortPairs;
//   * builds make the converged tree by levels (levelbuild.cuh, binlevel.cuh);
//   * where that does not apply, the octree build runs its split/merge rounds
//     on the device without a
//     host round-trip per round: rounds are issued in batches, every kernel
//     stops as soon as the device state says the tree converged, and the host
//     reads the state once per batch; the reference's vector capacity growth,
//     which decides leafCapacity, is replayed on the host from the per-round
//     proposals recorded on the device;
//   * the binary build emulates the reference's reject/grow/retry capacity
//     loop on the device (25% steps) instead of a host sync per pass.
#include "engine.hpp"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <thread>
#include <cmath>
#include <cstring>
#include <limits>
#include <map>
#include <tuple>
#include <mutex>
#include <stdexcept>
#include <utility>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "engine_util.cuh"
#include "keygen.cuh"
#include "binlevel.cuh"
#include "levelbuild.cuh"
#include "rebalance.cuh"
#include "sort_fused.cuh"
#include "tree_view.cuh"

namespace aot
{
static_assert(sort::kTile == int(kSortTileItems), "kSortTileItems must match the onesweep tile");
// --------------------------------------------------------------------------
// block cache
// --------------------------------------------------------------------------
namespace blockcache
{
namespace
{
// Misses are served by a stream-ordered pool of this library (cudaMallocAsync
// does not synchronise the device as cudaMalloc does); blocks never go back
// to the pool except through trim().
struct DevicePool
{
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
};
struct Cache
{
    std::mutex mu;
    std::map<std::pair<int, size_t>, std::vector<void *>> dev;  // (device, class) -> blocks
    std::map<size_t, std::vector<void *>> host;
    std::map<int, DevicePool> pools;
    size_t devBytes = 0;
};
Cache &cache()
{
    static Cache *c = new Cache();  // never destroyed: blocks may be given back during process exit
    return *c;
}
// size class: b rounded up to 2^k or 1.5 * 2^k (at most 50% above b), >= 256 bytes
size_t sizeClass(size_t b)
{
    if (b <= 256) return 256;
    const size_t top = size_t(1) << (63 - __builtin_clzll(b));
    if (b == top) return b;
    return b <= top + top / 2 ? top + top / 2 : 2 * top;
}
int currentDevice()
{
    int d = 0;
    AOT_CHECK(cudaGetDevice(&d));
    return d;
}
// with k.mu held
DevicePool &poolOf(Cache &k, int d)
{
    DevicePool &p = k.pools[d];
    if (!p.pool)
    {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = d;
        AOT_CHECK(cudaMemPoolCreate(&p.pool, &props));
        unsigned long long keep = ~0ull;  // keep what it maps until trim()
        AOT_CHECK(cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep));
        AOT_CHECK(cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking));
    }
    return p;
}
}  // namespace

void *take(size_t bytes, size_t *classBytes)
{
    const size_t c = sizeClass(bytes);
    const int d = currentDevice();
    Cache &k = cache();
    cudaStream_t s = nullptr;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(k.mu);
        auto it = k.dev.find({d, c});
        if (it != k.dev.end() && !it->second.empty())
        {
            void *p = it->second.back();
            it->second.pop_back();
            k.devBytes -= c;
            *classBytes = c;
            return p;
        }
        DevicePool &dp = poolOf(k, d);
        s = dp.stream;
        pool = dp.pool;
    }
    void *p = nullptr;
    cudaError_t e = cudaMallocFromPoolAsync(&p, c, pool, s);
    if (e == cudaErrorMemoryAllocation)
    {
        // give the cached blocks back and retry once
        (void)cudaGetLastError();
        trim();
        e = cudaMallocFromPoolAsync(&p, c, pool, s);
    }
    AOT_CHECK(e);
    waitStream(s);  // usable from any stream from here on
    *classBytes = c;
    return p;
}

void give(void *p, size_t classBytes)
{
    if (!p) return;
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess) return;
    Cache &k = cache();
    std::lock_guard<std::mutex> lock(k.mu);
    k.dev[{d, classBytes}].push_back(p);
    k.devBytes += classBytes;
}

void *takeHost(size_t bytes, size_t *classBytes)
{
    const size_t c = sizeClass(bytes);
    Cache &k = cache();
    {
        std::lock_guard<std::mutex> lock(k.mu);
        auto it = k.host.find(c);
        if (it != k.host.end() && !it->second.empty())
        {
            void *p = it->second.back();
            it->second.pop_back();
            *classBytes = c;
            return p;
        }
    }
    void *p = nullptr;
    AOT_CHECK(cudaMallocHost(&p, c));
    *classBytes = c;
    return p;
}

void giveHost(void *p, size_t classBytes)
{
    if (!p) return;
    Cache &k = cache();
    std::lock_guard<std::mutex> lock(k.mu);
    k.host[classBytes].push_back(p);
}

size_t cachedBytes()
{
    Cache &k = cache();
    std::lock_guard<std::mutex> lock(k.mu);
    return k.devBytes;
}

void trim()
{
    Cache &k = cache();
    std::lock_guard<std::mutex> lock(k.mu);
    int cur = 0;
    (void)cudaGetDevice(&cur);
    for (auto &kv : k.dev)
    {
        const int d = kv.first.first;
        auto pit = k.pools.find(d);
        if (pit == k.pools.end()) continue;
        (void)cudaSetDevice(d);
        for (void *p : kv.second) (void)cudaFreeAsync(p, pit->second.stream);
        kv.second.clear();
    }
    for (auto &kv : k.pools)
    {
        (void)cudaSetDevice(kv.first);
        (void)cudaStreamSynchronize(kv.second.stream);
        (void)cudaMemPoolTrimTo(kv.second.pool, 0);
    }
    (void)cudaSetDevice(cur);
    k.dev.clear();
    k.devBytes = 0;
}

namespace
{
struct Handles
{
    std::mutex mu;
    std::map<int, std::vector<cudaStream_t>> streams;
    std::map<int, std::vector<cudaEvent_t>> events;
};
Handles &handles()
{
    static Handles *h = new Handles;  // lives as long as the process (streams outlive static teardown)
    return *h;
}
}  // namespace

cudaStream_t takeStream()
{
    int d = 0;
    AOT_CHECK(cudaGetDevice(&d));
    Handles &h = handles();
    {
        std::lock_guard<std::mutex> lock(h.mu);
        auto &v = h.streams[d];
        if (!v.empty())
        {
            const cudaStream_t s = v.back();
            v.pop_back();
            return s;
        }
    }
    cudaStream_t s = nullptr;
    AOT_CHECK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    return s;
}

void giveStream(cudaStream_t s, int device)
{
    if (!s) return;
    Handles &h = handles();
    std::lock_guard<std::mutex> lock(h.mu);
    h.streams[device].push_back(s);
}

cudaEvent_t takeEvent()
{
    int d = 0;
    AOT_CHECK(cudaGetDevice(&d));
    Handles &h = handles();
    {
        std::lock_guard<std::mutex> lock(h.mu);
        auto &v = h.events[d];
        if (!v.empty())
        {
            const cudaEvent_t e = v.back();
            v.pop_back();
            return e;
        }
    }
    cudaEvent_t e = nullptr;
    AOT_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return e;
}

void giveEvent(cudaEvent_t e, int device)
{
    if (!e) return;
    Handles &h = handles();
    std::lock_guard<std::mutex> lock(h.mu);
    h.events[device].push_back(e);
}
}  // namespace blockcache

namespace
{
thread_local bool t_sleepingWaits = false;
}

void sleepingWaits(bool on) { t_sleepingWaits = on; }

void waitStream(cudaStream_t s)
{
    if (!t_sleepingWaits)
    {
        AOT_CHECK(cudaStreamSynchronize(s));
        return;
    }
    // one blocking-sync event per host thread and device
    thread_local std::map<int, cudaEvent_t> events;
    int d = 0;
    AOT_CHECK(cudaGetDevice(&d));
    cudaEvent_t &ev = events[d];
    if (!ev) AOT_CHECK(cudaEventCreateWithFlags(&ev, cudaEventBlockingSync | cudaEventDisableTiming));
    AOT_CHECK(cudaEventRecord(ev, s));
    // short waits (a tree's own round trips) are polled, yielding the core
    // between polls; long ones sleep in the blocking synchronisation
    const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(1000);
    for (;;)
    {
        const cudaError_t e = cudaEventQuery(ev);
        if (e == cudaSuccess) return;
        if (e != cudaErrorNotReady) AOT_CHECK(e);
        if (std::chrono::steady_clock::now() >= until) break;
        std::this_thread::yield();
    }
    AOT_CHECK(cudaEventSynchronize(ev));
}

// --------------------------------------------------------------------------
// DevMem
// --------------------------------------------------------------------------
DevMem::~DevMem() { release(); }
void DevMem::release()
{
    if (p) blockcache::give(p, bytes);
    p = nullptr;
    bytes = 0;
}
void DevMem::reserve(size_t b, cudaStream_t owner)
{
    if (b <= bytes) return;
    if (p)
    {
        // work queued on the old block must end before another buffer can be
        // handed the block
        if (owner) waitStream(owner);
        else AOT_CHECK(cudaDeviceSynchronize());
        blockcache::give(p, bytes);
    }
    p = nullptr;
    bytes = 0;
    p = blockcache::take(b, &bytes);
}
void DevMem::grow(size_t b, size_t keep, cudaStream_t s)
{
    if (b <= bytes) return;
    size_t nb = 0;
    void *q = blockcache::take(b, &nb);
    keep = std::min(keep, bytes);
    if (keep && p) AOT_CHECK(cudaMemcpyAsync(q, p, keep, cudaMemcpyDeviceToDevice, s));
    if (p)
    {
        // the owner queues its work on this block on s only
        waitStream(s);
        blockcache::give(p, bytes);
    }
    p = q;
    bytes = nb;
}

namespace
{
// Kernel launches issued by this process (all trees); reported by
// ao_tree_get_info so a benchmark can state how many engine kernels ran.
std::atomic<unsigned long long> g_launches{0};
}  // namespace

void noteLaunch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

int smCount()
{
    static int sms = 0;
    if (!sms)
    {
        int dev = 0;
        AOT_CHECK(cudaGetDevice(&dev));
        AOT_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        if (sms <= 0) sms = 148;
    }
    return sms;
}

namespace
{
// makeBinaryGeometry (binary_node.cuh:17-40): the longest side is halved at
// every depth, first axis wins ties.
BinaryGeometry makeGeometry(const double *b, unsigned maxDepth, int real)
{
    if (maxDepth > kBinDepth) throw std::invalid_argument("Binary maxDepth exceeds key precision");
    double bx[6];
    for (int k = 0; k < 6; ++k) bx[k] = real == 0 ? double(float(b[k])) : b[k];
    long double len[3] = {(long double)bx[1] - bx[0], (long double)bx[3] - bx[2], (long double)bx[5] - bx[4]};
    for (auto s : len)
        if (!(s > 0) || !std::isfinite(s)) throw std::invalid_argument("Tree box must have finite positive sides");
    BinaryGeometry g{};
    g.mortonOrder = 1;
    for (unsigned d = 0; d < kBinDepth; ++d)
    {
        unsigned a = 0;
        if (len[1] > len[a]) a = 1;
        if (len[2] > len[a]) a = 2;
        g.axis[d] = (unsigned char)a;
        if (a != d % 3) g.mortonOrder = 0;
        len[a] *= 0.5L;
    }
    g.xmin = bx[0];
    g.xmax = bx[1];
    g.ymin = bx[2];
    g.ymax = bx[3];
    g.zmin = bx[4];
    g.zmax = bx[5];
    return g;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Where a key generation leaves the digit counts of the sort that follows
// (hist == nullptr: nowhere).
struct KeygenSort
{
    u32 *hist = nullptr, *bins = nullptr;
    sort::SortControl *ctl = nullptr;
    const sort::PlanArgs *plan = nullptr;  // make the plan first
};

template <class Real, Curve C>
void launchKeygenT(const Real *x, const Real *y, const Real *z, size_t n, const KeygenParams<Real> &prm, u64 *keys,
                   const KeygenSort &ks, cudaStream_t s)
{
    if (ks.plan)
        planKernel<Real, C><<<ceilDiv(ks.plan->samples, sort::kPlanThreads), sort::kPlanThreads, 0, s>>>(
            x, y, z, n, prm, *ks.plan, ks.ctl, ks.hist), noteLaunch();
    const bool vec = aligned16(x) && aligned16(y) && aligned16(z);
    constexpr int V = sizeof(Real) == 4 ? 4 : 2;
    const size_t groups = vec ? n / V : n;
    const unsigned blocks = std::max(1u, std::min<unsigned>(ceilDiv(std::max<size_t>(groups, 1), kKeygenThreads),
                                                             unsigned(smCount()) * 8u));
    if (vec) keygenKernel<Real, C, V><<<blocks, kKeygenThreads, 0, s>>>(x, y, z, n, prm, keys, ks.hist, ks.bins, ks.ctl), noteLaunch();
    else keygenKernel<Real, C, 1><<<blocks, kKeygenThreads, 0, s>>>(x, y, z, n, prm, keys, ks.hist, ks.bins, ks.ctl), noteLaunch();
    AOT_LAUNCH_CHECK();
}

template <class Real>
void launchKeygen(int kind, bool hilbert, const Real *x, const Real *y, const Real *z, size_t n,
                  const KeygenParams<Real> &prm, u64 *keys, const KeygenSort &ks, cudaStream_t s)
{
    if (kind == 1) launchKeygenT<Real, Curve::Binary>(x, y, z, n, prm, keys, ks, s);
    else if (hilbert) launchKeygenT<Real, Curve::Hilbert>(x, y, z, n, prm, keys, ks, s);
    else launchKeygenT<Real, Curve::Morton>(x, y, z, n, prm, keys, ks, s);
}

__global__ void iotaKernel(u32 *perm, size_t n)
{
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        perm[i] = u32(i);
}

size_t configTiles(int cfg, size_t n) { return std::max<size_t>(1, (n + sort::configTile(cfg) - 1) / sort::configTile(cfg)); }

// Sort scratch in one block: the control block, the plan's counters,
// hist[kPassSlots][256] and bins[kPassSlots][256]; the look-back status words
// (u64) of one pass, with room for every configuration (their tags tell the
// passes apart); and for a planned sort the list of long runs and the
// plan's table.
struct SortArena
{
    DevMem mem;
    size_t longAt = 0, tableAt = 0;
    sort::PlanArgs plan{};
    static size_t up(size_t b) { return (b + 255) & ~size_t(255); }
    static constexpr size_t kPlanAt = (sizeof(sort::SortControl) + 15) & ~size_t(15);
    static constexpr size_t kHistAt = (kPlanAt + sizeof(sort::PlanCounters) + 255) & ~size_t(255);
    static constexpr size_t kHistWords = size_t(sort::kPassSlots) * sort::kRadix;
    static constexpr size_t kStatusAt = kHistAt + 2 * kHistWords * sizeof(u32);
    void ensure(size_t n, cudaStream_t owner, bool planned)
    {
        const size_t tiles = std::max<size_t>(1, (n + sort::kMinTile - 1) / sort::kMinTile);
        longAt = up(kStatusAt + tiles * sort::kRadix * sizeof(u64));
        tableAt = up(longAt + (planned ? sort::longRunWords(n) * sizeof(u32) : 0));
        const void *before = mem.p;
        mem.reserve(tableAt + (planned ? sort::planTableBytes(n) : 0), owner);
        // words left by another owner of the block could carry a tag this
        // arena will use: a new block starts cleared
        if (mem.p != before) AOT_CHECK(cudaMemsetAsync(mem.p, 0, mem.bytes, owner));
        if (!planned) return;
        plan.table = reinterpret_cast<u64 *>(at(tableAt));
        plan.counters = reinterpret_cast<sort::PlanCounters *>(at(kPlanAt));
        plan.samples = sort::planSamples(n);
        plan.slotBits = sort::planSlotBits(n);
    }
    unsigned char *at(size_t offset) const { return mem.as<unsigned char>() + offset; }
    sort::SortControl *ctl() const { return mem.as<sort::SortControl>(); }
    u32 *hist() const { return reinterpret_cast<u32 *>(at(kHistAt)); }
    u32 *bins() const { return hist() + kHistWords; }
    u64 *status() const { return reinterpret_cast<u64 *>(at(kStatusAt)); }
    u32 *longRuns() const { return reinterpret_cast<u32 *>(at(longAt)); }
};

// Sorts of at most this many keys run their passes and repair in one launch,
// unless the stream is being captured: a graph's launches cost less than the
// grid barriers.  Pair sorts of random keys queued directly, launch by launch
// and in one: 10k keys 72 and 57 us, 100k 79 and 61, 1M 113 and 99, 4M 202 and
// 200; from a graph 39 and 46, 48 and 51, 81 and 89, 164 and 190.
constexpr size_t kFusedSort = size_t(1) << 21;
// Pair sorts that make no plan run every pass, and count their digits first, which
// the few CTAs of a small sort do slowly.  Random keys queued directly, launch by
// launch and in one: one digit, 10k keys 21 and 26 us, 50k 24 and 27, 2M 48 and
// 51; four digits 45 and 49, 49 and 51, 200k 62 and 56, 700k 80 and 75, 2M 113
// and 120; eight digits 78 and 79, 84 and 83, 101 and 91, 128 and 128, 197 and
// 210.  (The sorts of views wait for their launches more than for their keys:
// computeViews() of k-d trees of 500, 5k and 50k particles, bucket 64, launch by launch
// 109, 121 and 127 us, in one 97, 102 and 111.)
constexpr int kFusedPasses = 4;
constexpr unsigned kFusedCounting = 32;
constexpr size_t kFusedUnplannedFrom = size_t(1) << 17, kFusedUnplannedTo = size_t(1) << 20;

// The passes and the repair of one launch (sort_fused.cuh), after the plan (or
// beginSortKernel); hist: with the digit counts.  False (nothing done) where
// the passes run launch by launch.
bool launchFusedSort(int cfg, cudaStream_t s, const sort::PassArgs &p, const sort::RepairArgs &r, u32 *hist, u32 *bins,
                     bool repair)
{
    if (p.n > kFusedSort) return false;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    AOT_CHECK(cudaStreamIsCapturing(s, &capture));
    if (capture != cudaStreamCaptureStatusNone) return false;
    size_t smem = 0;
    const void *fn = sort::fusedSort(cfg, smem);
    if (!fn) return false;
    AOT_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    int perSm = 0;
    AOT_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, fn, sort::kThreads, smem));
    if (perSm <= 0) return false;
    const u32 tiles = u32(configTiles(cfg, p.n));
    sort::FusedArgs a{p, r, tiles, hist, bins, repair, r.keyMask == ~u64(0)};
    void *args[] = {&a};
    // (a sort of few tiles counts with more CTAs than pass)
    const unsigned most = hist ? std::max(tiles, std::min(ceilDiv(p.n, 1024), kFusedCounting)) : tiles;
    AOT_CHECK(cudaLaunchKernel(fn, dim3(std::min(most, unsigned(perSm) * unsigned(smCount()))), dim3(sort::kThreads), args,
                               smem, s));
    noteLaunch();
    return true;
}

// The passes of configuration `cfg` over (k[0], v[0]) -> ... for bits [0,
// endBit), the input indices as values; the digit starts must be in bins, or
// hist: are counted first (the counts zero).
// Without a plan all passes run, and the index (0/1) of the buffers holding
// the result is returned; with one, the repair puts it into buffers 0
// (and writes the sample).
int runPasses(int cfg, cudaStream_t s, u64 *k[2], u32 *v[2], size_t n, int endBit, SortArena &a, int *error, bool plan,
              bool hist, u64 *sample = nullptr)
{
    sort::setPassSmemAll();
    const int bitsPer = sort::kSortConfigs[cfg].bits;
    const int passes = (endBit + bitsPer - 1) / bitsPer;
    sort::PassArgs p{k[0], nullptr, {k[0], k[1]}, {v[0], v[1]}, n, a.bins(), a.ctl(), a.status(), error,
                     0, endBit, passes, false};
    const sort::RepairArgs r{{k[0], k[1]}, {v[0], v[1]}, n, a.ctl(), a.longRuns(), sample, error,
                             0, passes, ~u64(0), false, true, true};
    if (launchFusedSort(cfg, s, p, r, hist ? a.hist() : nullptr, a.bins(), plan)) return plan ? 0 : passes & 1;
    if (hist)
    {
        const unsigned blocks = std::max(1u, std::min<unsigned>(ceilDiv(n, sort::kThreads), unsigned(smCount()) * 8u));
        sort::launchHistogram(cfg, s, blocks, k[0], n, 0, passes, a.hist(), endBit, a.ctl()), noteLaunch();
        sort::binsKernel<<<1, sort::kThreads, 0, s>>>(a.hist(), a.bins(), passes), noteLaunch();
        AOT_LAUNCH_CHECK();
    }
    for (int slot = 0; slot < passes; ++slot)
    {
        sort::launchPass(cfg, s, p, slot), noteLaunch();
        AOT_LAUNCH_CHECK();
    }
    if (!plan) return passes & 1;
    sort::repairKernel<true><<<sort::repairTiles(n), sort::kRepairThreads, 0, s>>>(r), noteLaunch();
    sort::longRunKernel<<<unsigned(smCount()) * 2u, sort::kLongThreads, 0, s>>>(r), noteLaunch();
    AOT_LAUNCH_CHECK();
    return 0;
}

// Generic stable sort of (keys, identity indices) by bits [0, 8*passes).
int sortWithIndices(cudaStream_t s, u64 *k[2], u32 *v[2], size_t n, int passes, SortArena &a, int *error)
{
    if (n == 0) return 0;
    const int cfg = sort::defaultSortConfig(n);
    a.ensure(n, s, false);
    sort::beginSortKernel<<<1, sort::kThreads, 0, s>>>(a.ctl(), a.hist()), noteLaunch();
    AOT_LAUNCH_CHECK();
    return runPasses(cfg, s, k, v, n, 8 * passes, a, error, false, true);
}

}  // namespace

unsigned gridFor(size_t n, unsigned threads) { return std::max(1u, ceilDiv(std::max<size_t>(n, 1), threads)); }

unsigned long long TreeEngine::kernelLaunches() { return g_launches.load(std::memory_order_relaxed); }

// --------------------------------------------------------------------------
// sort tuner
// --------------------------------------------------------------------------
namespace
{
struct TunerState
{
    std::mutex mu;
    std::map<std::tuple<int, int, int>, int> chosen;  // (device, segmented, size class) -> configuration
    std::map<std::tuple<int, int, int>, int> timing;  // classes being timed by some thread
    bool autotune = true;
    int forced = -1;
};
TunerState &tuner()
{
    static TunerState t;
    return t;
}
std::tuple<int, int, int> tuneKey(bool segmented, size_t n)
{
    int dev = 0;
    AOT_CHECK(cudaGetDevice(&dev));
    int cls = 0;
    while (cls < 63 && (size_t(1) << (cls + 1)) <= std::max<size_t>(n, 1)) ++cls;
    return {dev, segmented ? 1 : 0, cls};
}
}  // namespace

int sortConfigCount() { return sort::kNumSortConfigs; }

SortTuning sortConfigInfo(int config)
{
    if (config < 0 || config >= sort::kNumSortConfigs) throw std::invalid_argument("sort: unknown configuration");
    return {config, sort::kSortConfigs[config].bits, sort::kSortConfigs[config].items, false};
}

SortTuning sortTuning(bool segmented, size_t n)
{
    TunerState &t = tuner();
    const auto key = tuneKey(segmented, n);
    std::lock_guard<std::mutex> lock(t.mu);
    if (t.forced >= 0) return sortConfigInfo(t.forced);
    const auto it = t.chosen.find(key);
    if (it != t.chosen.end())
    {
        SortTuning r = sortConfigInfo(it->second);
        r.tuned = true;
        return r;
    }
    return sortConfigInfo(sort::defaultSortConfig(n));
}

bool sortNeedsTuning(bool segmented, size_t n)
{
    TunerState &t = tuner();
    const auto key = tuneKey(segmented, n);
    std::lock_guard<std::mutex> lock(t.mu);
    return t.autotune && t.forced < 0 && t.chosen.find(key) == t.chosen.end() && t.timing.find(key) == t.timing.end();
}

int sortTune(bool segmented, size_t n, float (*time)(int, void *), void *ctx)
{
    TunerState &t = tuner();
    const auto key = tuneKey(segmented, n);
    {
        std::lock_guard<std::mutex> lock(t.mu);
        t.timing[key] = 1;  // other threads sort this class with the default meanwhile
    }
    struct Done
    {
        TunerState &t;
        std::tuple<int, int, int> key;
        ~Done()
        {
            std::lock_guard<std::mutex> lock(t.mu);
            t.timing.erase(key);
        }
    } done{t, key};
    int best = sort::kDefaultSortConfig;
    float bestMs = 0.f;
    for (int c = 0; c < sort::kNumSortConfigs; ++c)
    {
        time(c, ctx);  // first launches of a configuration load and set up its kernels
        // the choice stands for every later sort of the class: configurations
        // without a plan (sort_plan.cuh), which always run every pass, are taken
        // only if clearly faster, as on keys whose plan runs every pass they
        // can be by a few percent (a batch of 130k keys, a fifth of them equal:
        // 95 us against 98; without the equal keys 90 against 50)
        const float ms = time(c, ctx) * (sort::kSortConfigs[c].bits == sort::kRadixBits ? 1.f : 1.25f);
        if (c == 0 || ms < bestMs)
        {
            best = c;
            bestMs = ms;
        }
    }
    std::lock_guard<std::mutex> lock(t.mu);
    t.chosen[key] = best;
    return best;
}

void sortSetAutotune(bool on)
{
    std::lock_guard<std::mutex> lock(tuner().mu);
    tuner().autotune = on;
}

void sortForceConfig(int config)
{
    if (config >= sort::kNumSortConfigs) throw std::invalid_argument("sort: unknown configuration");
    std::lock_guard<std::mutex> lock(tuner().mu);
    tuner().forced = config < 0 ? -1 : config;
}

void sortForgetTuning()
{
    std::lock_guard<std::mutex> lock(tuner().mu);
    tuner().chosen.clear();
}

// --------------------------------------------------------------------------
// stand-alone stable pair sort (cub::DeviceRadixSort::SortPairs semantics)
// --------------------------------------------------------------------------
namespace
{
struct PairSortLayout
{
    // altKeys | altVals | counters | status | plan table | long runs, each
    // part 256-byte aligned; from the counters to the plan table they are
    // cleared before a sort.  The
    // counters part starts with the error word (and 3 pad words), so its
    // offset depends on n only and ao_sort_pairs_check can find it whatever
    // configuration ran; then the control block, the plan's counters,
    // hist[passes][256] and bins[passes][256].
    size_t altKeys = 0, altVals = 0, counters = 0, status = 0, table = 0, longRuns = 0, total = 0, tiles = 0;
    int passes = 0;
    static constexpr size_t kCounterHead = 4;  // error word + padding (u32 words)
    static constexpr size_t kCtlWords = (sizeof(sort::SortControl) + 15) / 16 * 4;
    static constexpr size_t kPlanWords = (sizeof(sort::PlanCounters) + 15) / 16 * 4;
    static size_t up(size_t b) { return (b + 255) & ~size_t(255); }
    static size_t countersOffset(size_t n) { return up(up(n * sizeof(u64)) + n * sizeof(u32)); }
    PairSortLayout(size_t n, int cfg)
    {
        tiles = configTiles(cfg, n);
        passes = sort::configPasses(cfg);
        altKeys = 0;
        altVals = up(altKeys + n * sizeof(u64));
        counters = countersOffset(n);
        status = up(counters + counterWords() * sizeof(u32));
        table = up(status + tiles * sort::kRadix * sizeof(u64));
        longRuns = up(table + sort::planTableBytes(n));
        total = up(longRuns + sort::longRunWords(n) * sizeof(u32));
    }
    size_t counterWords() const { return kCounterHead + kCtlWords + kPlanWords + 2 * size_t(passes) * sort::kRadix; }
};
}  // namespace

// The scratch a caller sizes must fit whichever configuration the tuner
// later picks, so the size query answers the largest.
void TreeEngine::sortPairs(void *scratch, size_t *scratchBytes, const unsigned long long *keysIn,
                           unsigned long long *keysOut, const unsigned *valsIn, unsigned *valsOut, size_t n,
                           int beginBit, int endBit, cudaStream_t s)
{
    if (!scratchBytes) throw std::invalid_argument("ao_sort_pairs: scratch_bytes must not be null");
    if (!scratch)
    {
        size_t most = 0;
        for (int c = 0; c < sort::kNumSortConfigs; ++c)
        {
            size_t b = 0;
            sortPairsWith(c, nullptr, &b, keysIn, keysOut, valsIn, valsOut, n, beginBit, endBit, s);
            most = std::max(most, b);
        }
        *scratchBytes = most;
        return;
    }
    sortPairsWith(sortTuning(false, n).config, scratch, scratchBytes, keysIn, keysOut, valsIn, valsOut, n, beginBit,
                  endBit, s);
}

void TreeEngine::sortPairsWith(int cfg, void *scratch, size_t *scratchBytes, const unsigned long long *keysIn,
                               unsigned long long *keysOut, const unsigned *valsIn, unsigned *valsOut, size_t n,
                               int beginBit, int endBit, cudaStream_t s, int forcePlan)
{
    if (!scratchBytes) throw std::invalid_argument("ao_sort_pairs: scratch_bytes must not be null");
    if (beginBit < 0 || endBit > 64 || beginBit > endBit)
        throw std::invalid_argument("ao_sort_pairs: need 0 <= begin_bit <= end_bit <= 64");
    if (n > size_t(std::numeric_limits<std::uint32_t>::max()))
        throw std::invalid_argument("ao_sort_pairs: more than 2^32 - 1 items");
    if (cfg < 0 || cfg >= sort::kNumSortConfigs) throw std::invalid_argument("ao_sort_pairs: unknown configuration");
    const PairSortLayout lay(n, cfg);
    if (!scratch)
    {
        *scratchBytes = lay.total;
        return;
    }
    if (*scratchBytes < lay.total) throw std::invalid_argument("ao_sort_pairs: scratch too small");
    if (n == 0) return;
    if (!keysIn || !keysOut || !valsOut) throw std::invalid_argument("ao_sort_pairs: null array");
    if (keysIn == keysOut) throw std::invalid_argument("ao_sort_pairs: keys_in and keys_out must differ");
    char *base = static_cast<char *>(scratch);
    u64 *altK = reinterpret_cast<u64 *>(base + lay.altKeys);
    u32 *altV = reinterpret_cast<u32 *>(base + lay.altVals);
    u32 *head = reinterpret_cast<u32 *>(base + lay.counters);
    int *error = reinterpret_cast<int *>(head);
    sort::SortControl *ctl = reinterpret_cast<sort::SortControl *>(head + PairSortLayout::kCounterHead);
    u32 *planCounters = head + PairSortLayout::kCounterHead + PairSortLayout::kCtlWords;
    u32 *hist = planCounters + PairSortLayout::kPlanWords;
    u32 *bins = hist + size_t(lay.passes) * sort::kRadix;
    u64 *status = reinterpret_cast<u64 *>(base + lay.status);
    const int bitsPer = sort::kSortConfigs[cfg].bits;
    const int passes = (endBit - beginBit + bitsPer - 1) / bitsPer;
    if (passes == 0)
    {
        AOT_CHECK(cudaMemsetAsync(error, 0, sizeof(int), s));  // ao_sort_pairs_check reads it
        AOT_CHECK(cudaMemcpyAsync(keysOut, keysIn, n * sizeof(u64), cudaMemcpyDeviceToDevice, s));
        if (valsIn) AOT_CHECK(cudaMemcpyAsync(valsOut, valsIn, n * sizeof(u32), cudaMemcpyDeviceToDevice, s));
        else iotaKernel<<<gridFor(n, 256), 256, 0, s>>>(valsOut, n), noteLaunch();
        AOT_LAUNCH_CHECK();
        return;
    }
    AOT_CHECK(cudaMemsetAsync(head, 0, lay.longRuns - lay.counters, s));
    const u64 *in = reinterpret_cast<const u64 *>(keysIn);
    u64 *out = reinterpret_cast<u64 *>(keysOut);
    const u64 keyMask = (endBit - beginBit == 64 ? ~u64(0) : ((u64(1) << (endBit - beginBit)) - 1)) << beginBit;
    // a plan for 8-bit digits, where it can leave passes enough out
    const bool planned = bitsPer == sort::kRadixBits && (passes > sort::kUnplannedPasses || forcePlan >= 0);
    if (planned)
    {
        const sort::PlanArgs plan{reinterpret_cast<u64 *>(base + lay.table),
                                  reinterpret_cast<sort::PlanCounters *>(planCounters), sort::planSamples(n),
                                  sort::planSlotBits(n), std::min(forcePlan, passes - 1)};
        sort::planPairsKernel<<<ceilDiv(plan.samples, sort::kPlanThreads), sort::kPlanThreads, 0, s>>>(
            in, n, beginBit, passes, keyMask, plan, ctl), noteLaunch();
    }
    // (without a plan every pass runs, and the cleared control block says so)
    AOT_LAUNCH_CHECK();
    const sort::PassArgs p{in, valsIn, {out, altK}, {valsOut, altV}, n, bins, ctl, status, error, beginBit, endBit, passes,
                           true};
    const bool aligned = aligned16(out) && (reinterpret_cast<uintptr_t>(valsOut) & 7u) == 0;
    const sort::RepairArgs r{{out, altK}, {valsOut, altV}, n, ctl, reinterpret_cast<u32 *>(base + lay.longRuns), nullptr,
                             error, beginBit, passes, keyMask, true, aligned, false};
    const bool fuse = planned || (passes >= kFusedPasses && n >= kFusedUnplannedFrom && n <= kFusedUnplannedTo);
    if (fuse && launchFusedSort(cfg, s, p, r, hist, bins, planned)) return;
    const unsigned blocks = std::max(1u, std::min<unsigned>(ceilDiv(n, sort::kThreads), unsigned(smCount()) * 8u));
    sort::launchHistogram(cfg, s, blocks, in, n, beginBit, passes, hist, endBit, ctl), noteLaunch();
    sort::binsKernel<<<1, sort::kThreads, 0, s>>>(hist, bins, passes), noteLaunch();
    AOT_LAUNCH_CHECK();
    sort::setPassSmemAll();
    for (int slot = 0; slot < passes; ++slot)
    {
        sort::launchPass(cfg, s, p, slot), noteLaunch();
        AOT_LAUNCH_CHECK();
    }
    if (!planned) return;
    if (keyMask == ~u64(0))
        sort::repairKernel<true><<<sort::repairTiles(n), sort::kRepairThreads, 0, s>>>(r), noteLaunch();
    else
        sort::repairKernel<false><<<sort::repairTiles(n), sort::kRepairThreads, 0, s>>>(r), noteLaunch();
    sort::longRunKernel<<<unsigned(smCount()) * 2u, sort::kLongThreads, 0, s>>>(r), noteLaunch();
    AOT_LAUNCH_CHECK();
}

// Waits for `stream` and reads the error word of a pair sort of n items
// that ran in `scratch` (the bounded look-back of some pass gave up, so its
// output is not a sorted permutation).
bool TreeEngine::sortPairsFailed(const void *scratch, size_t n, cudaStream_t s)
{
    if (!scratch) throw std::invalid_argument("ao_sort_pairs_check: null scratch");
    int error = 0;
    AOT_CHECK(cudaMemcpyAsync(&error, static_cast<const char *>(scratch) + PairSortLayout::countersOffset(n),
                              sizeof(int), cudaMemcpyDeviceToHost, s));
    AOT_CHECK(cudaStreamSynchronize(s));
    return error != 0;
}

namespace
{
TreeEngine::SortPlan readSortPlan(const sort::SortControl *ctl, cudaStream_t s)
{
    u32 words[3];  // epoch, first, longRuns
    static_assert(offsetof(sort::SortControl, longRuns) == 2 * sizeof(u32), "the leading words");
    AOT_CHECK(cudaMemcpyAsync(words, ctl, sizeof(words), cudaMemcpyDeviceToHost, s));
    waitStream(s);
    return {int(words[1]), int(words[2])};
}
}  // namespace

TreeEngine::SortPlan TreeEngine::sortPairsPlan(const void *scratch, size_t n, cudaStream_t s)
{
    if (!scratch) throw std::invalid_argument("ao_selftest_sort_pairs: null scratch");
    return readSortPlan(reinterpret_cast<const sort::SortControl *>(
                            static_cast<const char *>(scratch) + PairSortLayout::countersOffset(n) +
                            PairSortLayout::kCounterHead * sizeof(u32)),
                        s);
}

// Loads every kernel a pair sort with the default configuration can launch
// (lazy module loading would otherwise load one at its first launch).
void TreeEngine::sortPairsPreload()
{
    cudaFuncAttributes a;
    AOT_CHECK(cudaFuncGetAttributes(&a, iotaKernel));
    AOT_CHECK(cudaFuncGetAttributes(&a, sort::beginSortKernel));
    AOT_CHECK(cudaFuncGetAttributes(&a, sort::binsKernel));
    AOT_CHECK(cudaFuncGetAttributes(&a, sort::planPairsKernel));
    AOT_CHECK(cudaFuncGetAttributes(&a, sort::repairKernel<true>));
    AOT_CHECK(cudaFuncGetAttributes(&a, sort::repairKernel<false>));
    AOT_CHECK(cudaFuncGetAttributes(&a, sort::longRunKernel));
    for (int c = 0; c < sort::kNumSortConfigs; ++c)
    {
        size_t smem = 0;
        if (const void *fn = sort::fusedSort(c, smem))
        {
            AOT_CHECK(cudaFuncGetAttributes(&a, fn));
            AOT_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        }
    }
    AOT_CHECK(cudaFuncGetAttributes(&a, sort::histogramKernel<8>));
    AOT_CHECK(cudaFuncGetAttributes(&a, sort::histogramKernel<7>));
#define AOT_CASE(i, B, I) AOT_CHECK(cudaFuncGetAttributes(&a, sort::onesweepKernel<B, I>));
    AOT_SORT_CONFIGS(AOT_CASE)
#undef AOT_CASE
    sort::setPassSmemAll();
}

// --------------------------------------------------------------------------
// Impl
// --------------------------------------------------------------------------
struct TreeEngine::Impl
{
    // particles
    DevMem P[2], Perm[2], sample;
    SortArena sortArena;
    // state
    DevMem stMem;
    DeviceState *st = nullptr;   // device (stMem)
    DeviceState *hst = nullptr;  // pinned mirror (block cache)
    size_t hstBytes = 0;
    cudaStream_t d2h = nullptr;
    cudaEvent_t ready = nullptr;
    int device = 0;  // the device of the pooled streams and events
    cudaEvent_t marks[8] = {};              // stage events (profiling)
    cudaEvent_t tuneStart = nullptr, tuneEnd = nullptr;  // sort tuner timing
    std::vector<cudaEvent_t> nfMarks;       // begin/end pairs around near-field launches
    DevMem history;
    // tree
    DevMem K[2], B[2], NF[2], N[2], G[2], offs, dirty, scan;
    DevMem nodeRows;  // node table of the near-field refresh (NFCount)
    // converged build by levels (levelbuild.cuh): unit arena and its control
    DevMem lvRows, lvVal, lvChild, lvSub, lvOffset, lvCtl, lvNbr, lvParent, lvRec;
    size_t lvCap = 0;
    int lvLevels = int(kOctLevels);  // levels the last level build needed, with one to spare
    DevMem mergeSplits;              // merge-path cuts of the full begin refresh
    unsigned char *lvHost = nullptr; // pinned: the level build's one readback
    size_t lvHostBytes = 0;
    // binary tree by levels (binlevel.cuh)
    DevMem blRows, blChild, blSub, blParent, blOffset, blCtl;
    size_t blCap = 0;
    bl::Control *blHost = nullptr;   // pinned readback
    size_t blHostBytes = 0;
    u32 nodeSlots = 0;
    bool nodeStale = true;         // the keys changed or the table moved: clear before use
    size_t scanTiles = 0;
    // views
    DevMem vBox, vSplit, vDepth, vParent, vChild, vLevelOffset, vPbegin, vPcount, vPmap, vMaxDepth;
    DevMem vLeafLevel, vLeafToNode, vLevels, vCandStart, vCandLevel, vLvKeys[2], vLvVals[2], vLayKeys[2], vLayVals[2];
    DevMem vIntStartSfc, vIntLevelSfc, vIntM, vIntStartLay, vIntLevelLay;
    SortArena viewSort;
    size_t viewLeafCap = 0, viewParticleCap = 0;
    bool viewScratch = false;
    adaptive_octree::ViewConfig viewPrepared{};
    size_t viewNodesLogical = 0, mappingLogical = 0;
    // keys
    KeygenParams<float> kpf{};
    KeygenParams<double> kpd{};

    ~Impl()
    {
        if (hst) blockcache::giveHost(hst, hstBytes);
        if (lvHost) blockcache::giveHost(lvHost, lvHostBytes);
        if (blHost) blockcache::giveHost(blHost, blHostBytes);
        blockcache::giveEvent(ready, device);
        for (cudaEvent_t e : marks)
            if (e) cudaEventDestroy(e);
        if (tuneStart) cudaEventDestroy(tuneStart);
        if (tuneEnd) cudaEventDestroy(tuneEnd);
        for (cudaEvent_t e : nfMarks) cudaEventDestroy(e);
        blockcache::giveStream(d2h, device);
    }

    // device bytes held by this tree
    size_t bytes() const
    {
        const DevMem *all[] = {&P[0],        &P[1],        &Perm[0],        &Perm[1],      &sample,
                               &sortArena.mem, &stMem, &history, &K[0],
                               &K[1],        &B[0],        &B[1],           &NF[0],        &NF[1],
                               &N[0],        &N[1],        &G[0],           &G[1],         &offs,
                               &dirty,       &scan,        &vBox,           &vSplit,       &vDepth,
                               &vParent,     &vChild,      &vLevelOffset,   &vPbegin,      &vPcount,
                               &vPmap,       &vMaxDepth,   &vLeafLevel,     &vLeafToNode,  &vLevels,
                               &vCandStart,  &vCandLevel,  &vLvKeys[0],     &vLvKeys[1],   &vLvVals[0],
                               &vLvVals[1],  &vLayKeys[0], &vLayKeys[1],    &vLayVals[0],  &vLayVals[1],
                               &vIntStartSfc, &vIntLevelSfc, &vIntM,        &vIntStartLay, &vIntLevelLay,
                               &viewSort.mem, &nodeRows, &lvRows, &lvVal, &lvChild,
                               &lvSub, &lvOffset, &lvCtl, &lvNbr, &lvParent, &lvRec,
                               &blRows, &blChild, &blSub, &blParent, &blOffset, &blCtl, &mergeSplits};
        size_t s = 0;
        for (const DevMem *d : all) s += d->bytes;
        return s;
    }

    // the unit arena (levelbuild.cuh)
    static constexpr size_t kUnitHeadBytes = (sizeof(lb::Control) + 255) & ~size_t(255);
    static constexpr size_t kUnitCtlBytes =
        kUnitHeadBytes + (lb::kContribBins + lb::kArrivals) * sizeof(unsigned long long);
    lb::Arena units() const
    {
        lb::Arena a{};
        a.rows = lvRows.as<u32>();
        a.val = lvVal.as<u32>();
        a.nbr = lvNbr.as<u32>();
        a.rec = lvRec.as<u64>();
        a.child = lvChild.as<u32>();
        a.sub = lvSub.as<u64>();
        a.parent = lvParent.as<u32>();
        a.offset = lvOffset.as<u32>();
        a.ctl = lvCtl.as<lb::Control>();
        a.contrib = reinterpret_cast<unsigned long long *>(lvCtl.as<unsigned char>() + kUnitHeadBytes);
        a.landed = a.contrib + lb::kContribBins;
        a.cap = u32(lvCap);
        return a;
    }

    rb::TreeBufs bufs() const
    {
        rb::TreeBufs t{};
        for (int k = 0; k < 2; ++k)
        {
            t.K[k] = K[k].as<u64>();
            t.B[k] = B[k].as<u32>();
            t.NF[k] = NF[k].as<u32>();
            t.G[k] = G[k].as<u8>();
            t.N[k] = N[k].as<u32>();
        }
        t.offs = offs.as<u32>();
        t.dirty = dirty.as<int>();
        t.scanStatus = scan.as<u64>();
        t.scanTile = reinterpret_cast<u32 *>(scan.as<u64>() + scanTiles);
        t.st = st;
        return t;
    }
    KeyIndex keyIndex(size_t n) const
    {
        KeyIndex k{};
        k.keys = P[0].as<u64>();
        k.sample = sample.as<u64>();
        k.n = n;
        k.ns = (n + kSampleStride - 1) >> kSampleShift;
        return k;
    }
    tv::ViewBufs viewBufs() const
    {
        tv::ViewBufs v{};
        v.box = vBox.as<u64>();
        v.split = vSplit.as<u8>();
        v.depth = vDepth.as<u8>();
        v.parent = vParent.as<int>();
        v.child = vChild.as<int>();
        v.levelOffset = vLevelOffset.as<int>();
        v.pbegin = vPbegin.as<u32>();
        v.pcount = vPcount.as<u32>();
        v.pmap = vPmap.as<u64>();
        v.maxDepth = vMaxDepth.as<u8>();
        v.leafLevel = vLeafLevel.as<u8>();
        v.leafToNode = vLeafToNode.as<int>();
        int *lv = vLevels.as<int>();
        v.leavesPerLevel = lv;
        v.internalPerLevel = lv + 66;
        v.nodesPerLevel = lv + 2 * 66;
        v.levelOffsetInternal = lv + 3 * 66;
        v.candStart = vCandStart.as<u64>();
        v.candLevel = vCandLevel.as<u8>();
        v.lvKeys = vLvKeys[0].as<u64>();
        v.lvKeysAlt = vLvKeys[1].as<u64>();
        v.lvVals = vLvVals[0].as<u32>();
        v.lvValsAlt = vLvVals[1].as<u32>();
        v.layKeys = vLayKeys[0].as<u64>();
        v.layKeysAlt = vLayKeys[1].as<u64>();
        v.layVals = vLayVals[0].as<u32>();
        v.layValsAlt = vLayVals[1].as<u32>();
        v.intStartSfc = vIntStartSfc.as<u64>();
        v.intLevelSfc = vIntLevelSfc.as<u8>();
        v.intMBySfc = vIntM.as<int>();
        v.intStartLay = vIntStartLay.as<u64>();
        v.intLevelLay = vIntLevelLay.as<u8>();
        return v;
    }
};

// --------------------------------------------------------------------------
// construction
// --------------------------------------------------------------------------
TreeEngine::TreeEngine(const void *x, const void *y, const void *z, size_t n, const EngineConfig &cfg)
    : m_(std::make_unique<Impl>()), cfg_(cfg), n_(n), x_(x), y_(y), z_(z)
{
    // Backend constructor checks (octree.cu:321-416, kdtree3d.cu:175-216).
    if (n > 0 && (!x || !y || !z))
        throw std::invalid_argument("adaptive_octree: coordinate device pointers must not be null");
    if (cfg.bucket == 0) throw std::invalid_argument("adaptive_octree: particle limit must be positive");
    if (cfg.iterations == 0) throw std::invalid_argument("adaptive_octree: updateIterations must be positive");
    if (cfg.kind == 1) m_->kpd.g = makeGeometry(cfg.box, cfg.maxDepth, cfg.real), m_->kpf.g = m_->kpd.g;
    if (n > size_t(std::numeric_limits<std::uint32_t>::max()))
        throw std::invalid_argument(
            "adaptive_octree: particle count exceeds 32-bit permutation index range");
    m_->kpf.q = makeQuantBox<float>(cfg.box);
    m_->kpd.q = makeQuantBox<double>(cfg.box);
    prepared_ = cfg.views;

    // stream-ordered set-up: nothing here synchronises the device
    m_->stMem.reserve(sizeof(DeviceState));
    m_->st = m_->stMem.as<DeviceState>();
    AOT_CHECK(cudaMemsetAsync(m_->st, 0, sizeof(DeviceState), cfg.stream));
    m_->hst = static_cast<DeviceState *>(blockcache::takeHost(sizeof(DeviceState), &m_->hstBytes));
    std::memset(m_->hst, 0, sizeof(DeviceState));
    AOT_CHECK(cudaGetDevice(&m_->device));
    m_->d2h = blockcache::takeStream();
    m_->ready = blockcache::takeEvent();
    if (n)
    {
        for (int k = 0; k < 2; ++k)
        {
            m_->P[k].reserve(n * sizeof(u64));
            m_->Perm[k].reserve(n * sizeof(u32));
        }
        m_->sample.reserve(((n + kSampleStride - 1) >> kSampleShift) * sizeof(u64));
        m_->sortArena.ensure(n, cfg.stream, true);
    }
    ensurePhysical(16);
    if (cfg.kind == 0)
    {
        const u64 root[2] = {0, kMaxKey};
        AOT_CHECK(cudaMemcpyAsync(m_->K[0].p, root, sizeof(root), cudaMemcpyHostToDevice, cfg.stream));
        waitStream(cfg.stream);
    }
}

size_t TreeEngine::deviceBytes() const { return m_->bytes(); }

void TreeEngine::forceSortPlan(int first)
{
    if (first < -1 || first >= sort::kMaxPasses) throw std::invalid_argument("sort plan: first pass must be -1 to 7");
    m_->sortArena.plan.force = first;
}

TreeEngine::SortPlan TreeEngine::sortPlan() const
{
    if (n_ == 0) return {0, 0};
    return readSortPlan(m_->sortArena.ctl(), cfg_.stream);
}

namespace
{
// dst[i] = src[perm[i]], W-byte words
template <class W>
__global__ void gatherKernel(const W *__restrict__ src, W *__restrict__ dst, const u32 *__restrict__ perm, size_t n)
{
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
        dst[i] = src[perm[i]];
}
__global__ void gatherBytesKernel(const unsigned char *__restrict__ src, unsigned char *__restrict__ dst,
                                  const u32 *__restrict__ perm, size_t n, size_t e)
{
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
    {
        const unsigned char *s = src + size_t(perm[i]) * e;
        for (size_t b = 0; b < e; ++b) dst[i * e + b] = s[b];
    }
}
}  // namespace

void TreeEngine::gather(const void *src, void *dst, size_t elemBytes) const
{
    if (n_ == 0) return;
    if (!src || !dst) throw std::invalid_argument("adaptive_octree: gather needs device source and destination");
    if (elemBytes == 0) throw std::invalid_argument("adaptive_octree: gather element size must be positive");
    if (src == dst) throw std::invalid_argument("adaptive_octree: gather cannot work in place");
    cudaStream_t s = cfg_.stream;
    const u32 *perm = m_->Perm[0].as<u32>();
    const unsigned blocks = std::min<unsigned>(gridFor(n_, 256), unsigned(smCount()) * 16u);
    const uintptr_t align = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst);
    if (elemBytes == 4 && align % 4 == 0)
        gatherKernel<u32><<<blocks, 256, 0, s>>>(static_cast<const u32 *>(src), static_cast<u32 *>(dst), perm, n_), noteLaunch();
    else if (elemBytes == 8 && align % 8 == 0)
        gatherKernel<u64><<<blocks, 256, 0, s>>>(static_cast<const u64 *>(src), static_cast<u64 *>(dst), perm, n_), noteLaunch();
    else if (elemBytes == 16 && align % 16 == 0)
        gatherKernel<uint4><<<blocks, 256, 0, s>>>(static_cast<const uint4 *>(src), static_cast<uint4 *>(dst), perm, n_), noteLaunch();
    else
        gatherBytesKernel<<<blocks, 256, 0, s>>>(static_cast<const unsigned char *>(src), static_cast<unsigned char *>(dst),
                                                 perm, n_, elemBytes), noteLaunch();
    AOT_LAUNCH_CHECK();
}

// The buffers go back to the block cache: no queued work may still use them.
TreeEngine::~TreeEngine()
{
    if (m_)
    {
        (void)cudaStreamSynchronize(cfg_.stream);
        if (m_->d2h) (void)cudaStreamSynchronize(m_->d2h);
    }
}

void TreeEngine::setCoordinates(const void *x, const void *y, const void *z)
{
    if (n_ > 0 && (!x || !y || !z))
        throw std::invalid_argument("adaptive_octree: coordinate device pointers must not be null");
    x_ = x;
    y_ = y;
    z_ = z;
}

// Physical capacity of the leaf buffers (>= leafCapacity at all times).
void TreeEngine::ensurePhysical(size_t capacity)
{
    if (capacity <= physCap_ && m_->K[0].p) return;
    cudaStream_t s = cfg_.stream;
    const size_t c = std::max(capacity, physCap_);
    for (int k = 0; k < 2; ++k)
    {
        m_->K[k].grow((c + 1) * sizeof(u64), m_->K[k].bytes, s);
        m_->B[k].grow((c + 1) * sizeof(u32), m_->B[k].bytes, s);
        m_->N[k].grow((c + 1) * sizeof(u32), m_->N[k].bytes, s);
        if (cfg_.kind == 0 && cfg_.nf)
        {
            m_->NF[k].grow((c + 1) * sizeof(u32), m_->NF[k].bytes, s);
            m_->G[k].grow((c + 1) * sizeof(u8), m_->G[k].bytes, s);
        }
        else
        {
            // nearFieldCounts_d of a LeafCount tree (or a binary tree) is never
            // written: it reads as zeros, as the reference's value-initialised vector
            const size_t before = m_->NF[k].bytes;
            m_->NF[k].grow(sizeof(u32) * (c + 1), m_->NF[k].bytes, s);
            if (m_->NF[k].bytes != before) AOT_CHECK(cudaMemsetAsync(m_->NF[k].p, 0, m_->NF[k].bytes, s));
            m_->G[k].grow(16, m_->G[k].bytes, s);
        }
    }
    m_->offs.reserve((c + 1) * sizeof(u32), s);
    m_->dirty.reserve((c + 1) * sizeof(int), s);
    // the merge-path cuts of the full begin refresh (reserved here: an update
    // may run under stream capture, where nothing may be allocated)
    m_->mergeSplits.reserve(((c + 1 + n_) / rb::kMergeChunk + 3) * sizeof(u32), s);
    // candidate group leaders are first children of distinct internal nodes: <= (L - 1) / 7
    m_->scanTiles = (c + 1 + rb::kScanTile - 1) / rb::kScanTile;
    m_->scan.reserve((m_->scanTiles + 1) * sizeof(u64), s);
    if (cfg_.kind == 0 && cfg_.nf)
    {
        // every internal node of the tree (about a seventh of the leaves) and
        // cells that were internal nodes since the last sort, with room to
        // spare: linear probing stays short
        const size_t slots = std::min<size_t>(c / 4 + 1024, 0xffffffffu);
        if (slots > m_->nodeSlots)
        {
            m_->nodeRows.reserve(slots * rb::kGroupRow * sizeof(u32), s);
            m_->nodeSlots = u32(slots);
            m_->nodeStale = true;
        }
        // the refresh of update() takes a large tree's internal nodes as units: a
        // seventh of its leaves less one.  (Not a unit more: a build that places
        // again, in larger leaf arrays, keeps its units, however full the arena.)
        if (refreshByUnits() && c > 4096) ensureUnits(std::max((c - 1) / 7, n_ / 4 + 4096));
    }
    physCap_ = c;
}

// The unit arena for at least `cap` units.
void TreeEngine::ensureUnits(size_t cap)
{
    Impl &m = *m_;
    cudaStream_t s = cfg_.stream;
    cap = std::max(cap, m.lvCap);
    m.lvRows.reserve(cap * lb::kRow * sizeof(u32), s);
    if (cfg_.nf)
    {
        m.lvVal.reserve(cap * 8 * sizeof(u32), s);
        m.lvNbr.reserve(cap * 27 * sizeof(u32), s);
        m.lvRec.reserve(cap * sizeof(u64), s);
    }
    m.lvChild.reserve(cap * 8 * sizeof(u32), s);
    m.lvSub.reserve(cap * sizeof(u64), s);
    m.lvParent.reserve(cap * sizeof(u32), s);
    m.lvOffset.reserve(cap * sizeof(u32), s);
    m.lvCtl.reserve(Impl::kUnitCtlBytes, s);
    m.lvCap = cap;
}

// --------------------------------------------------------------------------
// keys + sort (octree.cu:285-307, kdtree3d.cu:161-172)
// --------------------------------------------------------------------------
void TreeEngine::sortParticles()
{
    m_->nodeStale = true;  // cell table entries hold indices into the sorted keys
    if (n_ == 0) return;
    cudaStream_t s = cfg_.stream;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    AOT_CHECK(cudaStreamIsCapturing(s, &capture));
    if (capture == cudaStreamCaptureStatusNone && cfg_.tuneSort && sortNeedsTuning(false, n_))
    {
        // every configuration sorts identically, so the keys of the last
        // timed run are the sorted keys
        if (!m_->tuneStart) AOT_CHECK(cudaEventCreate(&m_->tuneStart));
        if (!m_->tuneEnd) AOT_CHECK(cudaEventCreate(&m_->tuneEnd));
        auto time = [](int c, void *ctx) -> float {
            TreeEngine &e = *static_cast<TreeEngine *>(ctx);
            AOT_CHECK(cudaEventRecord(e.m_->tuneStart, e.cfg_.stream));
            e.sortKeys(c);
            AOT_CHECK(cudaEventRecord(e.m_->tuneEnd, e.cfg_.stream));
            AOT_CHECK(cudaEventSynchronize(e.m_->tuneEnd));
            float ms = 0.f;
            AOT_CHECK(cudaEventElapsedTime(&ms, e.m_->tuneStart, e.m_->tuneEnd));
            return ms;
        };
        sortTune(false, n_, time, this);
    }
    else if (capture != cudaStreamCaptureStatusNone && sortConfig_ >= 0)
    {
        sortKeys(sortConfig_);  // under capture: the last sort's configuration and scratch
    }
    else
    {
        sortKeys(sortTuning(false, n_).config);
    }
}

// Keys of every particle, then the stable (key, slot) sort with sort
// configuration `config`; the result lands in P[0] / Perm[0], every 32nd key
// in the sample.
void TreeEngine::sortKeys(int config)
{
    cudaStream_t s = cfg_.stream;
    SortArena &a = m_->sortArena;
    const int passes = sort::configPasses(config);
    if (passes & 1) throw std::logic_error("adaptive_octree: sort configurations must have an even pass count");
    u64 *k[2] = {m_->P[0].as<u64>(), m_->P[1].as<u64>()};
    u32 *v[2] = {m_->Perm[0].as<u32>(), m_->Perm[1].as<u32>()};
    // 8-bit digits: a plan, and the digit counts come with the keys; otherwise
    // every pass, and the counts by a kernel of their own
    const bool planned = sort::kSortConfigs[config].bits == sort::kRadixBits;
    const KeygenSort ks = planned ? KeygenSort{a.hist(), a.bins(), a.ctl(), &a.plan} : KeygenSort{};
    if (cfg_.real == 0)
        launchKeygen<float>(cfg_.kind, cfg_.hilbert, static_cast<const float *>(x_), static_cast<const float *>(y_),
                            static_cast<const float *>(z_), n_, m_->kpf, k[0], ks, s);
    else
        launchKeygen<double>(cfg_.kind, cfg_.hilbert, static_cast<const double *>(x_), static_cast<const double *>(y_),
                             static_cast<const double *>(z_), n_, m_->kpd, k[0], ks, s);
    if (!planned) sort::beginSortKernel<<<1, sort::kThreads, 0, s>>>(a.ctl(), a.hist()), noteLaunch();
    AOT_LAUNCH_CHECK();
    // (without a plan the repair finds all passes run and writes the sample alone)
    runPasses(config, s, k, v, n_, 64, a, &m_->st->error, true, !planned, m_->sample.as<u64>());
    sortConfig_ = config;
}

void TreeEngine::computeKeys(int kind, int real, const void *x, const void *y, const void *z, size_t n,
                             const double *box, bool hilbert, unsigned maxDepth, unsigned long long *keys,
                             unsigned *perm, cudaStream_t s)
{
    if (n == 0) return;
    if (n > size_t(std::numeric_limits<std::uint32_t>::max()))
        throw std::invalid_argument("adaptive_octree: particle count exceeds 32-bit permutation index range");
    KeygenParams<float> pf{};
    KeygenParams<double> pd{};
    if (kind == 1) pd.g = pf.g = makeGeometry(box, maxDepth, real);
    pf.q = makeQuantBox<float>(box);
    pd.q = makeQuantBox<double>(box);
    if (real == 0)
        launchKeygen<float>(kind, hilbert, static_cast<const float *>(x), static_cast<const float *>(y),
                            static_cast<const float *>(z), n, pf, reinterpret_cast<u64 *>(keys), {}, s);
    else
        launchKeygen<double>(kind, hilbert, static_cast<const double *>(x), static_cast<const double *>(y),
                             static_cast<const double *>(z), n, pd, reinterpret_cast<u64 *>(keys), {}, s);
    if (perm)
    {
        iotaKernel<<<gridFor(n, 256), 256, 0, s>>>(perm, n), noteLaunch();
        AOT_LAUNCH_CHECK();
    }
}

// --------------------------------------------------------------------------
// rebalance passes
// --------------------------------------------------------------------------
namespace
{
__global__ void octInitRootKernel(rb::TreeBufs tb, const u64 *P, size_t n)
{
    DeviceState *st = tb.st;
    const unsigned active = n ? unsigned(lowerBoundDev(P, n, kMaxKey)) : 0u;
    tb.K[0][0] = 0;
    tb.K[0][1] = kMaxKey;
    tb.B[0][0] = 0;
    tb.B[0][1] = active;
    const u64 sq = u64(active) * active;
    tb.NF[0][0] = sq > 0xffffffffull / 27ull ? 0xffffffffu : u32(27ull * sq);  // octree.cu:23-38
    const int err = st->error;
    *st = DeviceState{};
    st->error = err;
    st->numLeaves = 1;
    st->newNumLeaves = 1;
    st->numActiveParticles = active;
}

// finishBuildStateKernel (octree.cu:40-47)
__global__ void octFinishBuildKernel(DeviceState *st)
{
    st->newNumLeaves = st->numLeaves;
    st->changed = st->converged = st->needsResize = 0;
    st->numNodes = 0;
    st->activeBuffer = 0;
    st->overflow = 0;
}

// initBinaryRootKernel (kdtree3d.cu:24-30)
__global__ void binInitRootKernel(rb::TreeBufs tb, long long logicalCap)
{
    DeviceState *st = tb.st;
    tb.K[0][0] = 0;
    tb.K[0][1] = kMaxKey;
    const int err = st->error;
    *st = DeviceState{};
    st->error = err;
    st->numLeaves = 1;
    st->newNumLeaves = 1;
    st->numNodes = 1;
    st->logicalCap = logicalCap;
}

__global__ void clearOverflowKernel(DeviceState *st) { st->overflow = 0; }
}  // namespace

void TreeEngine::octreePass(bool buildMode, long long limit)
{
    cudaStream_t s = cfg_.stream;
    const rb::TreeBufs tb = m_->bufs();
    const size_t cap = buildMode ? physCap_ : leafCapacity_;
    const size_t tiles = (cap + 1 + rb::kScanTile - 1) / rb::kScanTile;
    rb::beginPassKernel<<<1, 1, 0, s>>>(m_->st), noteLaunch();
    AOT_CHECK(cudaMemsetAsync(m_->scan.p, 0, (m_->scanTiles + 1) * sizeof(u64), s));
    const int mode = buildMode ? kModeOctreeBuild : kModeUpdate;
    long long *hist = buildMode ? m_->history.as<long long>() : nullptr;
    const unsigned scatterBlocks = std::min(gridFor(cap, rb::kScatterThreads), unsigned(smCount()) * 8u);
    const unsigned refreshBlocks = unsigned(smCount()) * 8u;
    if (cfg_.nf)
    {
        rb::octDecideScanKernel<true><<<unsigned(tiles), rb::kScanThreads, 0, s>>>(tb, cfg_.bucket), noteLaunch();
        rb::octScatterKernel<true><<<scatterBlocks, rb::kScatterThreads, 0, s>>>(tb, limit, mode, hist), noteLaunch();
    }
    else
    {
        rb::octDecideScanKernel<false><<<unsigned(tiles), rb::kScanThreads, 0, s>>>(tb, cfg_.bucket), noteLaunch();
        rb::octScatterKernel<false><<<scatterBlocks, rb::kScatterThreads, 0, s>>>(tb, limit, mode, hist), noteLaunch();
    }
    AOT_LAUNCH_CHECK();
    refreshCounts(false, refreshBlocks);
    AOT_LAUNCH_CHECK();
}

void TreeEngine::binaryPass(bool buildMode, long long limit)
{
    cudaStream_t s = cfg_.stream;
    const rb::TreeBufs tb = m_->bufs();
    const size_t cap = buildMode ? physCap_ : leafCapacity_;
    const size_t tiles = (cap + 1 + rb::kScanTile - 1) / rb::kScanTile;
    rb::beginPassKernel<<<1, 1, 0, s>>>(m_->st), noteLaunch();
    AOT_CHECK(cudaMemsetAsync(m_->scan.p, 0, (m_->scanTiles + 1) * sizeof(u64), s));
    const KeyIndex idx = m_->keyIndex(n_);
    rb::binDecideScanKernel<<<unsigned(tiles), rb::kScanThreads, 0, s>>>(tb, cfg_.bucket, cfg_.maxDepth), noteLaunch();
    rb::binScatterKernel<<<std::min(gridFor(cap, rb::kScatterThreads), unsigned(smCount()) * 8u), rb::kScatterThreads, 0, s>>>(
        tb, limit, buildMode ? kModeBinaryBuild : kModeUpdate), noteLaunch();
    rb::binRefreshKernel<false><<<unsigned(smCount()) * 8u, 256, 0, s>>>(tb, idx), noteLaunch();
    AOT_LAUNCH_CHECK();
}

// Full refresh of the per-leaf quantities of the active tree, after the
// reset of changed/converged/active count (resetRebalanceStateKernel +
// refreshGraphCountsGpu without dirty lists).
void TreeEngine::refreshAll()
{
    cudaStream_t s = cfg_.stream;
    const rb::TreeBufs tb = m_->bufs();
    const KeyIndex idx = m_->keyIndex(n_);
    rb::resetForUpdateKernel<<<1, 32, 0, s>>>(m_->st, m_->P[0].as<u64>(), n_), noteLaunch();
    const unsigned blocks = unsigned(smCount()) * 8u;
    if (cfg_.kind == 1)
    {
        rb::binRefreshKernel<true><<<blocks, 256, 0, s>>>(tb, idx), noteLaunch();
        AOT_LAUNCH_CHECK();
    }
    else
    {
        refreshCounts(true, blocks);
    }
}

// Per-leaf quantities of the active octree: begin indices, then (NFCount)
// near-field counts and group-merge flags.  all = every leaf, else the work
// lists of the last materialisation.
void TreeEngine::refreshCounts(bool all, unsigned blocks)
{
    cudaStream_t s = cfg_.stream;
    const rb::TreeBufs tb = m_->bufs();
    const KeyIndex idx = m_->keyIndex(n_);
    if (all)
    {
        // every leaf: a merge of the leaf keys with the particle keys
        const size_t chunks = (physCap_ + 1 + n_) / rb::kMergeChunk + 2;  // cuts: reserved by ensurePhysical
        const u64 *P = m_->P[0].as<u64>();
        rb::mergeSplitKernel<<<gridFor(chunks + 1, 256), 256, 0, s>>>(tb, P, m_->mergeSplits.as<u32>()), noteLaunch();
        rb::mergeBeginKernel<<<unsigned(std::min<size_t>(chunks, size_t(smCount()) * 8u)), 256, 0, s>>>(
            tb, P, m_->mergeSplits.as<u32>()),
            noteLaunch();
    }
    else
    {
        rb::octBeginKernel<false><<<blocks, rb::kRefreshThreads, 0, s>>>(tb, idx), noteLaunch();
    }
    if (cfg_.nf)
    {
        const rb::NodeTable gt{m_->nodeRows.as<u32>(), m_->nodeSlots};
        if (all && refreshByUnits())
        {
            refreshUnits();
            return;
        }
        // a cleared table takes the nodes of every leaf, else those of the new leaves
        const bool fill = all || m_->nodeStale;
        if (m_->nodeStale)
        {
            AOT_CHECK(cudaMemsetAsync(gt.rows, 0, size_t(gt.slots) * rb::kGroupRow * sizeof(u32), s));
            m_->nodeStale = false;
        }
        if (fill) rb::nodeTableKernel<true><<<blocks, rb::kRefreshThreads, 0, s>>>(tb, gt), noteLaunch();
        else rb::nodeTableKernel<false><<<blocks, rb::kRefreshThreads, 0, s>>>(tb, gt), noteLaunch();
        markNearField(true);
        if (all && cfg_.hilbert)
            rb::octNearFieldKernel<true, true><<<blocks, rb::kRefreshThreads, 0, s>>>(tb, idx, cfg_.bucket, gt), noteLaunch();
        else if (all)
            rb::octNearFieldKernel<false, true><<<blocks, rb::kRefreshThreads, 0, s>>>(tb, idx, cfg_.bucket, gt), noteLaunch();
        else if (cfg_.hilbert)
            rb::octNearFieldKernel<true, false><<<blocks, rb::kRefreshThreads, 0, s>>>(tb, idx, cfg_.bucket, gt), noteLaunch();
        else
            rb::octNearFieldKernel<false, false><<<blocks, rb::kRefreshThreads, 0, s>>>(tb, idx, cfg_.bucket, gt), noteLaunch();
        markNearField(false);
    }
    AOT_LAUNCH_CHECK();
}

// The full refresh of a large NFCount tree: its internal nodes as units, their
// near field level by level, and the node table of the passes from the units.
// (Every level a tree can have is launched: a captured update() serves deeper
// trees too.)
void TreeEngine::refreshUnits()
{
    Impl &m = *m_;
    cudaStream_t s = cfg_.stream;
    const rb::TreeBufs tb = m.bufs();
    const lb::Arena a = m.units();
    const KeyIndex idx = m.keyIndex(n_);
    const unsigned blocks = unsigned(smCount()) * 4u;
    AOT_CHECK(cudaMemsetAsync(a.ctl, 0, sizeof(lb::Control), s));
    lb::treeRootKernel<<<1, 1, 0, s>>>(a, tb), noteLaunch();
    for (int l = 0; l < int(kOctLevels); ++l)
        if (cfg_.hilbert) lb::treeUnitsKernel<true><<<blocks * 2, lb::kThreads, 0, s>>>(a, tb, l), noteLaunch();
        else lb::treeUnitsKernel<false><<<blocks * 2, lb::kThreads, 0, s>>>(a, tb, l), noteLaunch();
    markNearField(true);
    for (int l = 0; l < int(kOctLevels); ++l)
        if (cfg_.hilbert) lb::nearFieldKernel<true, false><<<blocks, lb::kThreads, 0, s>>>(a, idx, l, tb, cfg_.bucket), noteLaunch();
        else lb::nearFieldKernel<false, false><<<blocks, lb::kThreads, 0, s>>>(a, idx, l, tb, cfg_.bucket), noteLaunch();
    markNearField(false);
    const rb::NodeTable gt{m.nodeRows.as<u32>(), m.nodeSlots};
    AOT_CHECK(cudaMemsetAsync(gt.rows, 0, size_t(gt.slots) * rb::kGroupRow * sizeof(u32), s));
    m.nodeStale = false;
    lb::unitsToTableKernel<<<blocks * 2, lb::kThreads, 0, s>>>(a, gt), noteLaunch();
    AOT_LAUNCH_CHECK();
}

// (The units' 42 launches cost about 150 us however small the tree is.)
bool TreeEngine::refreshByUnits() const { return cfg_.kind == 0 && cfg_.nf && n_ >= kUnitRefreshParticles; }

void TreeEngine::materializeCounts()
{
    rb::materializeCountsKernel<<<gridFor(std::max(leafCapacity_, physCap_), 256), 256, 0, cfg_.stream>>>(m_->bufs()), noteLaunch();
    AOT_LAUNCH_CHECK();
}

// --------------------------------------------------------------------------
// state readback (octree.cu:498-537, kdtree3d.cu:127-137)
// --------------------------------------------------------------------------
void TreeEngine::readState()
{
    AOT_CHECK(cudaEventRecord(m_->ready, cfg_.stream));
    AOT_CHECK(cudaStreamWaitEvent(m_->d2h, m_->ready, 0));
    AOT_CHECK(cudaMemcpyAsync(m_->hst, m_->st, sizeof(DeviceState), cudaMemcpyDeviceToHost, m_->d2h));
    waitStream(m_->d2h);
    applyState();
}

// The host's copies of the state from the mirror (filled by a readback, or
// by the host where it knows every value).
void TreeEngine::applyState()
{
    const DeviceState &h = *m_->hst;
    if (h.error) throw std::runtime_error("adaptive_octree: a device scan gave up waiting (bounded look-back)");
    hostActiveBuffer_ = h.activeBuffer;
    hostLeaves_ = size_t(std::max(h.numLeaves, 0));
    hostActive_ = h.numActiveParticles;
    hostNodes_ = size_t(std::max(h.numNodes, 0));
    if (cfg_.kind == 0) capModel_.stateRead(hostLeaves_);
    syncViewSizes();
}

bool TreeEngine::doBuffersNeedResize()
{
    if (!built_) return false;
    readState();
    return m_->hst->needsResize != 0;
}

// --------------------------------------------------------------------------
// capacity (octree.cu:182-241, kdtree3d.cu:96-116)
// --------------------------------------------------------------------------

void TreeEngine::prepareGraphBuffers(size_t capacity)
{
    if (cfg_.kind == 0)
    {
        const size_t maxLeaves = (size_t(std::numeric_limits<int>::max()) - 1) / 8 * 7 + 1;
        if (capacity > maxLeaves) throw std::length_error("adaptive_octree: buffer capacity exceeds node index range");
        leafCapacity_ = capacity;
        capModel_.prepare(capacity);
        ensurePhysical(capacity);
        prepareViews(capacity, prepared_);
        syncViewSizes();
    }
    else
    {
        const size_t maxLeaves = size_t(std::numeric_limits<int>::max()) / 2 + 1;
        if (capacity > maxLeaves) throw std::length_error("adaptive_octree: buffer capacity exceeds node index range");
        leafCapacity_ = capacity;
        ensurePhysical(capacity);
        if (built_ && prepared_.treeStructure | prepared_.particleCountsPerBox | prepared_.particleMapping)
            prepareViews(capacity, prepared_);
        syncViewSizes();
    }
}

void TreeEngine::resizeBuffers()
{
    if (!built_) throw std::logic_error("adaptive_octree: call build() before resizeBuffers()");
    readState();
    prepareGraphBuffers(leafCapacity_ + (leafCapacity_ + 3) / 4);
    AOT_CHECK(cudaMemsetAsync(&m_->st->needsResize, 0, sizeof(int), cfg_.stream));
    waitStream(cfg_.stream);
}

// --------------------------------------------------------------------------
// build / update
// --------------------------------------------------------------------------
void TreeEngine::build()
{
    if (cfg_.kind == 0) octreeBuild();
    else binaryBuild();
}

void TreeEngine::octreeBuild()
{
    cudaStream_t s = cfg_.stream;
    waitStream(s);
    mark(MarkStart, 1);
    capModel_.buildStart();
    sortParticles();
    mark(MarkSorted);
    // Room for the build; grown on overflow.
    const size_t estimate = std::max<size_t>(4096, cfg_.nf ? n_ + 4096 : n_ / 4 + 4096);
    ensurePhysical(std::max(physCap_, estimate));
    std::vector<long long> proposals;
    lastBuildByLevels_ = buildMode_ == 0 && octreeLevelBuild(proposals);
    size_t leaves = 0;
    if (lastBuildByLevels_)
    {
        leaves = hostLeaves_;
    }
    else
    {
        m_->history.reserve(std::max<size_t>(cfg_.maxDepth, 1) * sizeof(long long), cfg_.stream);
        rb::TreeBufs tb = m_->bufs();
        octInitRootKernel<<<1, 1, 0, s>>>(tb, m_->P[0].as<u64>(), n_), noteLaunch();
        AOT_LAUNCH_CHECK();
        // rebalanceBuild (octree.cu:159-180): at most maxDepth decision rounds
        int done = 0;
        const int maxRounds = int(cfg_.maxDepth);
        while (done < maxRounds)
        {
            const int batch = std::min(4, maxRounds - done);
            for (int r = 0; r < batch; ++r) octreePass(true, (long long)physCap_);
            AOT_CHECK(cudaMemcpyAsync(m_->hst, m_->st, sizeof(DeviceState), cudaMemcpyDeviceToHost, s));
            waitStream(s);
            const DeviceState h = *m_->hst;
            if (h.error) throw std::runtime_error("adaptive_octree: a device scan gave up waiting (bounded look-back)");
            done = h.rounds;
            if (h.converged) break;
            if (h.overflow)
            {
                const size_t need = size_t(h.proposal);
                ensurePhysical(std::max(need + need / 4, 2 * physCap_));
                clearOverflowKernel<<<1, 1, 0, s>>>(m_->st), noteLaunch();
                AOT_LAUNCH_CHECK();
            }
        }
        AOT_CHECK(cudaMemcpyAsync(m_->hst, m_->st, sizeof(DeviceState), cudaMemcpyDeviceToHost, s));
        waitStream(s);
        const DeviceState h = *m_->hst;
        proposals.resize(size_t(h.iteration));
        if (h.iteration)
            AOT_CHECK(cudaMemcpy(proposals.data(), m_->history.p, proposals.size() * sizeof(long long),
                                 cudaMemcpyDeviceToHost));
        leaves = size_t(h.numLeaves);
        // The final tree must sit in buffer 0 (finishBuildStateKernel resets the
        // active buffer).
        if (h.activeBuffer == 1)
        {
            AOT_CHECK(cudaMemcpyAsync(m_->K[0].p, m_->K[1].p, (leaves + 1) * sizeof(u64), cudaMemcpyDeviceToDevice, s));
            AOT_CHECK(cudaMemcpyAsync(m_->B[0].p, m_->B[1].p, (leaves + 1) * sizeof(u32), cudaMemcpyDeviceToDevice, s));
            if (cfg_.nf)
            {
                AOT_CHECK(cudaMemcpyAsync(m_->NF[0].p, m_->NF[1].p, leaves * sizeof(u32), cudaMemcpyDeviceToDevice, s));
                AOT_CHECK(cudaMemcpyAsync(m_->G[0].p, m_->G[1].p, leaves * sizeof(u8), cudaMemcpyDeviceToDevice, s));
            }
        }
        octFinishBuildKernel<<<1, 1, 0, s>>>(m_->st), noteLaunch();
        AOT_LAUNCH_CHECK();
    }
    mark(MarkPassed);
    buildRounds_ = int(proposals.size());
    hostLeaves_ = leaves;
    // Replay the reference's K_d/tmpTree capacity history (octree.cu:159-180,
    // 453-457; resizeWithHeadroom, helpers.cuh:122-141).
    const size_t cap = capModel_.finishBuild(proposals.data(), proposals.size(), leaves);
    prepareGraphBuffers(cap);
    built_ = true;
    if (!lastBuildByLevels_) materializeCounts();  // the placement of a build by levels writes the counts
    buildViews(cfg_.views);
    mark(MarkEnd);
    // the state read at the end of a build (doBuffersNeedResize); a build by
    // levels without views already knows every value of the state
    const bool views = cfg_.views.treeStructure | cfg_.views.particleCountsPerBox | cfg_.views.particleMapping;
    if (lastBuildByLevels_ && !views) applyState();
    else (void)doBuffersNeedResize();
}

void TreeEngine::setBuildMode(int mode)
{
    if (mode != 0 && mode != 1) throw std::invalid_argument("adaptive_octree: build mode must be 0 (levels) or 1 (rounds)");
    buildMode_ = mode;
}

namespace
{
// A launch by team (grid_barrier.cuh); grid: as many CTAs as fit at once on an
// idle GPU, or fewer.
void launchTeam(const void *fn, void **args, int threads, unsigned grid, cudaStream_t s)
{
    AOT_CHECK(cudaLaunchKernel(fn, dim3(grid), dim3(unsigned(threads)), args, 0, s));
    noteLaunch();
}
// The grid of a placement: all that fits.
unsigned placeGrid(const void *fn)
{
    int perSm = 0;
    AOT_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, fn, lb::kThreads, 0));
    return unsigned(std::max(1, perSm)) * unsigned(smCount());
}
}  // namespace

// The converged octree, level by level (levelbuild.cuh).  The tree is the
// one the reference's build rounds converge to; the round history (leaves
// after each round that changed the tree) comes from the per-region counts.
bool TreeEngine::octreeLevelBuild(std::vector<long long> &proposals)
{
    if (!cfg_.nf && u64(cfg_.bucket) * 512u > 0xffffffffull) return false;  // wrapping split thresholds
    cudaStream_t s = cfg_.stream;
    Impl &m = *m_;
    const bool nf = cfg_.nf;
    const unsigned blocks = unsigned(smCount()) * 4u;
    unsigned leafGrid = 0;
    if (!nf)
    {
        // one launch by team: a CTA per unit of a typical level (2.5
        // leaves per bucket of particles, 7 leaves per unit), as many as fit;
        // few CTAs meet at a barrier sooner
        int perSm = 0;
        AOT_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, lb::leafBuildKernel, lb::kThreads, 0));
        if (perSm <= 0) return false;
        leafGrid = unsigned(std::min<size_t>(size_t(std::min(perSm, 4)) * size_t(smCount()),
                                             n_ / (2 * std::max<size_t>(cfg_.bucket, 1)) + 16));
    }
    const KeyIndex idx = m.keyIndex(n_);
    const u64 *P = m.P[0].as<u64>();
    size_t cap = std::max<size_t>(m.lvCap, n_ / 4 + 4096);
    constexpr size_t kHeadBytes = Impl::kUnitHeadBytes, kCtlBytes = Impl::kUnitCtlBytes;
    if (!m.lvHost)
        m.lvHost = static_cast<unsigned char *>(blockcache::takeHost(kCtlBytes + 16, &m.lvHostBytes));
    unsigned char *host = m.lvHost;
    const lb::Control &hc = *reinterpret_cast<const lb::Control *>(host);
    for (;;)
    {
        if (cap >= (size_t(1) << 28)) return false;  // neighbour references hold unit * 8 + digit in 31 bits
        ensureUnits(cap);
        const lb::Arena a = m.units();
        AOT_CHECK(cudaMemsetAsync(m.lvCtl.p, 0, kCtlBytes, s));
        // Every kernel reads its level's size on the device, so the whole
        // build is queued without a host wait: the levels the last build
        // needed (all 21 the first time), their subtree counts and the
        // placement; one readback at the end checks that no deeper level
        // was left out.
        const int levels = nf ? std::max(1, std::min(int(kOctLevels), m.lvLevels)) : int(kOctLevels);
        auto place = [&](int expanded) {
            rb::TreeBufs tb = m.bufs();
            u32 room = u32(physCap_);
            lb::Arena arena = a;
            const void *fn = nf && cfg_.hilbert ? reinterpret_cast<const void *>(&lb::placeKernel<true, true>)
                             : nf               ? reinterpret_cast<const void *>(&lb::placeKernel<true, false>)
                                                : reinterpret_cast<const void *>(&lb::placeKernel<false, false>);
            void *args[] = {&arena, &tb.K[0], &tb.B[0], &tb.NF[0], &tb.N[0], &expanded, &room};
            launchTeam(fn, args, lb::kThreads, placeGrid(fn), s);
        };
        u32 rootLeaves = 1;
        if (nf)
        {
            lb::rootKernel<<<1, 32, 0, s>>>(a, m.bufs(), P, n_, cfg_.bucket), noteLaunch();
            AOT_LAUNCH_CHECK();
            for (int l = 0; l < levels; ++l)
            {
                if (cfg_.hilbert) lb::expandKernel<true><<<blocks * 2, lb::kThreads, 0, s>>>(a, idx, l), noteLaunch();
                else lb::expandKernel<false><<<blocks * 2, lb::kThreads, 0, s>>>(a, idx, l), noteLaunch();
                markNearField(true);
                if (cfg_.hilbert) lb::nearFieldKernel<true, true><<<blocks, lb::kThreads, 0, s>>>(a, idx, l, rb::TreeBufs{}, cfg_.bucket), noteLaunch();
                else lb::nearFieldKernel<false, true><<<blocks, lb::kThreads, 0, s>>>(a, idx, l, rb::TreeBufs{}, cfg_.bucket), noteLaunch();
                markNearField(false);
                AOT_LAUNCH_CHECK();
            }
            lb::subtreeKernel<<<blocks * 2, lb::kThreads, 0, s>>>(a, levels), noteLaunch();
            AOT_LAUNCH_CHECK();
            place(levels);
            // the round history is needed before finishKernel writes it; read
            // everything once
            // (with the device state: its active count, set by the root kernel)
            AOT_CHECK(cudaMemcpyAsync(host, m.lvCtl.p, kCtlBytes, cudaMemcpyDeviceToHost, s));
            AOT_CHECK(cudaMemcpyAsync(host + kCtlBytes, a.sub, sizeof(u32), cudaMemcpyDeviceToHost, s));  // the root's leaves
            AOT_CHECK(cudaMemcpyAsync(m.hst, m.st, sizeof(DeviceState), cudaMemcpyDeviceToHost, s));
            waitStream(s);
            std::memcpy(&rootLeaves, host + kCtlBytes, sizeof(u32));
        }
        else
        {
            lb::LeafBuildArgs p{a, idx, m.bufs(), P, n_, cfg_.bucket, cfg_.maxDepth, u32(physCap_)};
            void *args[] = {&p};
            launchTeam(reinterpret_cast<const void *>(&lb::leafBuildKernel), args, lb::kThreads, leafGrid, s);
            AOT_CHECK(cudaMemcpyAsync(host, m.lvCtl.p, kCtlBytes, cudaMemcpyDeviceToHost, s));
            waitStream(s);
            if (hc.bar.error) throw std::runtime_error("adaptive_octree: a grid barrier of the level build gave up waiting");
            rootLeaves = hc.leaves;
            // the device state's other words are set below, as the kernel set them
            *m.hst = DeviceState{};
            m.hst->numActiveParticles = hc.active;
            m.hst->error = hc.stateError;
        }
        if (hc.error) throw std::runtime_error("adaptive_octree: a device scan gave up waiting (bounded look-back)");
        if (hc.overflow)
        {
            cap *= 2;
            continue;
        }
        if (hc.late) return false;
        if (nf && hc.levelCount[levels] != 0)
        {
            m.lvLevels = int(kOctLevels);  // deeper than the last build: all levels again
            continue;
        }
        int deepest = -1;  // deepest level holding units
        for (int l = 0; l < levels; ++l)
            if (hc.levelCount[l]) deepest = l;
        if (deepest < 0) rootLeaves = 1;
        // leaves after every round that changed the tree
        const auto *contrib = reinterpret_cast<const unsigned long long *>(host + kHeadBytes);
        const auto *landed = contrib + lb::kContribBins;
        int rounds = 0;
        for (int ai = 0; ai < lb::kArrivals; ++ai)
            for (int k = 1; k < lb::kJumps; ++k)
                for (int j = 1; j <= k; ++j)
                    if (contrib[(ai * lb::kJumps + k) * lb::kJumps + j]) rounds = std::max(rounds, ai + 1 + (k - j));
        if (rounds > int(cfg_.maxDepth)) return false;  // the rounds stop before converging
        proposals.assign(size_t(rounds), 0);
        for (int t = 1; t <= rounds; ++t)
        {
            unsigned long long leavesAt = landed[t];
            for (int ai = 0; ai + 1 <= t && ai < lb::kArrivals; ++ai)
                for (int k = 1; k < lb::kJumps; ++k)
                    for (int j = 1; j <= k; ++j)
                    {
                        const unsigned long long c = contrib[(ai * lb::kJumps + k) * lb::kJumps + j];
                        if (!c) continue;
                        const int e = k - (t - ai - 1) - j;
                        leavesAt += c << (3 * std::max(e, 0));
                    }
            proposals[size_t(t - 1)] = (long long)leavesAt;
        }
        if (rounds && proposals.back() != (long long)rootLeaves)
            throw std::logic_error("adaptive_octree: level build history does not end at the tree");
        if (hc.placeOverflow)
        {
            ensurePhysical(rootLeaves);
            AOT_CHECK(cudaMemsetAsync(&a.ctl->placeOverflow, 0, sizeof(int), s));
            AOT_CHECK(cudaMemsetAsync(&a.ctl->bar, 0, sizeof(GridBarrier), s));
            place(deepest + 1);
        }
        hostLeaves_ = rootLeaves;
        m.lvLevels = std::min(int(kOctLevels), deepest + 2);
        if (nf || hc.placeOverflow)
        {
            lb::finishKernel<<<1, 1, 0, s>>>(a, m.bufs(), rounds, levels, u32(physCap_)), noteLaunch();
            AOT_LAUNCH_CHECK();
        }
        // the host mirror of what finishKernel writes (the readback above
        // brought the active count), so the build needs no second readback
        DeviceState &h = *m.hst;
        h.numLeaves = h.newNumLeaves = int(rootLeaves);
        h.proposal = (long long)rootLeaves;
        h.iteration = rounds;
        h.rounds = rounds + 1;
        h.changed = h.converged = h.needsResize = 0;
        h.numNodes = 0;
        h.activeBuffer = 0;
        h.overflow = 0;
        h.dirtyCount = 0;
        if (nf) AOT_CHECK(cudaMemsetAsync(m.G[0].p, 0, m.G[0].bytes, s));  // no group of the converged tree may merge
        return true;
    }
}

void TreeEngine::binaryBuild()
{
    cudaStream_t s = cfg_.stream;
    waitStream(s);
    built_ = false;
    hostLeaves_ = 1;
    prepareGraphBuffers(std::max<size_t>(2, leafCapacity_));
    sortParticles();
    const size_t estimate = std::max<size_t>(4096, 4 * (n_ / std::max(1u, cfg_.bucket)) + 4096);
    ensurePhysical(std::max({physCap_, estimate, leafCapacity_}));
    lastBuildByLevels_ = buildMode_ == 0 && binaryLevelBuild();
    if (lastBuildByLevels_)
    {
        built_ = true;
        if (prepared_.treeStructure | prepared_.particleCountsPerBox | prepared_.particleMapping)
            prepareViews(leafCapacity_, prepared_);
        buildViews(cfg_.views);  // the placement wrote the counts
        const bool views = cfg_.views.treeStructure | cfg_.views.particleCountsPerBox | cfg_.views.particleMapping;
        if (views) readState();
        else applyState();  // the finish kernel's state, known on the host
        return;
    }
    rb::TreeBufs tb = m_->bufs();
    binInitRootKernel<<<1, 1, 0, s>>>(tb, (long long)leafCapacity_), noteLaunch();
    AOT_LAUNCH_CHECK();
    refreshAll();
    // build loop (kdtree3d.cu:239-249): passes until converged
    long long passes = 0;
    for (;;)
    {
        const int batch = 8;
        for (int r = 0; r < batch; ++r) binaryPass(true, (long long)physCap_);
        passes += batch;
        AOT_CHECK(cudaMemcpyAsync(m_->hst, m_->st, sizeof(DeviceState), cudaMemcpyDeviceToHost, s));
        waitStream(s);
        const DeviceState h = *m_->hst;
        if (h.error) throw std::runtime_error("adaptive_octree: a device scan gave up waiting (bounded look-back)");
        if (h.converged) break;
        if (h.overflow)
        {
            const size_t need = size_t(h.proposal);
            ensurePhysical(std::max(need + need / 4, 2 * physCap_));
            clearOverflowKernel<<<1, 1, 0, s>>>(m_->st), noteLaunch();
            AOT_LAUNCH_CHECK();
        }
        if (passes > 200000) throw std::runtime_error("adaptive_octree: binary build did not converge");
    }
    buildRounds_ = m_->hst->iteration;
    leafCapacity_ = size_t(m_->hst->logicalCap);
    ensurePhysical(leafCapacity_);
    built_ = true;
    if (prepared_.treeStructure | prepared_.particleCountsPerBox | prepared_.particleMapping)
        prepareViews(leafCapacity_, prepared_);
    materializeCounts();
    buildViews(cfg_.views);
    readState();
}

// The converged binary tree, level by level (binlevel.cuh): the tree the
// reference's build passes end with, its pass count and its leaf capacity.
// False where the passes must run: a depth limit beyond the 63 key bits.
bool TreeEngine::binaryLevelBuild()
{
    if (cfg_.maxDepth > 63) return false;
    cudaStream_t s = cfg_.stream;
    Impl &m = *m_;
    // a CTA per unit of a typical level (as octreeLevelBuild), as many as fit
    int perSm = 0;
    AOT_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, bl::buildKernel, bl::kThreads, 0));
    if (perSm <= 0) return false;
    const size_t buckets = n_ / std::max<size_t>(cfg_.bucket, 1);
    const unsigned grid =
        unsigned(std::min<size_t>(size_t(std::min(perSm, 4)) * size_t(smCount()), buckets / 2 + 16));
    size_t cap = std::max<size_t>(m.blCap, buckets + 4096);
    if (!m.blHost) m.blHost = static_cast<bl::Control *>(blockcache::takeHost(sizeof(bl::Control), &m.blHostBytes));
    const bl::Control &hc = *m.blHost;
    for (;;)
    {
        if (cap >= (size_t(1) << 31)) return false;
        m.blRows.reserve(cap * lb::kRow * sizeof(u32), s);
        m.blChild.reserve(cap * 8 * sizeof(u32), s);
        m.blSub.reserve(cap * sizeof(u64), s);
        m.blParent.reserve(cap * sizeof(u32), s);
        m.blOffset.reserve(cap * sizeof(u32), s);
        m.blCtl.reserve(sizeof(bl::Control), s);
        m.blCap = cap;
        bl::BuildArgs p{};
        bl::Arena &a = p.a;
        a.rows = m.blRows.as<u32>();
        a.child = m.blChild.as<u32>();
        a.sub = m.blSub.as<u64>();
        a.parent = m.blParent.as<u32>();
        a.offset = m.blOffset.as<u32>();
        a.ctl = m.blCtl.as<bl::Control>();
        a.cap = u32(cap);
        p.idx = m.keyIndex(n_);
        p.tb = m.bufs();
        p.P = m.P[0].as<u64>();
        p.n = n_;
        p.bucket = cfg_.bucket;
        p.maxDepth = cfg_.maxDepth;
        p.capacity = u32(physCap_);
        p.logicalCap = (long long)leafCapacity_;
        AOT_CHECK(cudaMemsetAsync(m.blCtl.p, 0, sizeof(bl::Control), s));
        void *args[] = {&p};
        launchTeam(reinterpret_cast<const void *>(&bl::buildKernel), args, bl::kThreads, grid, s);
        AOT_CHECK(cudaMemcpyAsync(m.blHost, m.blCtl.p, sizeof(bl::Control), cudaMemcpyDeviceToHost, s));
        waitStream(s);
        if (hc.bar.error) throw std::runtime_error("adaptive_octree: a grid barrier of the level build gave up waiting");
        if (hc.overflow)
        {
            cap *= 2;
            continue;
        }
        if (hc.stateError | hc.error)
            throw std::runtime_error("adaptive_octree: a device scan gave up waiting (bounded look-back)");
        // one pass per depth of internal nodes
        const u32 leaves = hc.leaves;
        const int passes = hc.depths;
        const long long c = bl::grownCapacity((long long)leafCapacity_, (long long)leaves);
        if (hc.placeOverflow)
        {
            ensurePhysical(leaves);
            rb::TreeBufs tb = m.bufs();
            u32 units = hc.units, room = u32(physCap_);
            void *again[] = {&a, &tb.K[0], &tb.B[0], &tb.N[0], &units, &room};
            AOT_CHECK(cudaMemsetAsync(&a.ctl->bar, 0, sizeof(GridBarrier), s));
            const void *fn = reinterpret_cast<const void *>(&bl::placeKernel);
            launchTeam(fn, again, bl::kThreads, placeGrid(fn), s);
            bl::finishKernel<<<1, 1, 0, s>>>(tb, int(leaves), passes, c), noteLaunch();
            AOT_LAUNCH_CHECK();
        }
        // the host mirror of the finished state
        DeviceState &h = *m.hst;
        h = DeviceState{};
        h.numActiveParticles = hc.active;
        h.numLeaves = h.newNumLeaves = int(leaves);
        h.numNodes = (int(leaves) - 1) * 2 + 1;
        h.proposal = (long long)leaves;
        h.iteration = passes;
        h.rounds = passes + 1;
        h.converged = 1;
        h.logicalCap = c;
        buildRounds_ = passes;
        hostLeaves_ = leaves;
        leafCapacity_ = size_t(c);
        ensurePhysical(leafCapacity_);
        return true;
    }
}

// Trees of at most this many leaves (their capacity) pass in one launch.  An
// update() queued directly, launch by launch and in one, and the same from a
// graph: octrees of 1.2k leaves 109 and 81 us (graph 69 and 69), 33k 150 and
// 127 (125 and 114), 262k 274 and 253 (228 and 228), 2.1M 495 and 516 (440 and
// 494); k-d trees of 1.3k leaves 152 and 85 (118 and 80), 354k 516 and 463 (451
// and 439).
constexpr size_t kFusedLeaves = size_t(1) << 19;

// The refresh, the passes and the counts of an update() in one launch
// (rb::updateKernel).  False (nothing done) where they run launch by launch:
// NFCount trees, trees without particles, and while stages are timed.
bool TreeEngine::passesFused()
{
    if (cfg_.nf || profiling_ || n_ == 0) return false;  // (the sort clears the barrier)
    if (leafCapacity_ > kFusedLeaves) return false;
    const void *fn = cfg_.kind == 0 ? reinterpret_cast<const void *>(&rb::updateKernel<false>)
                                    : reinterpret_cast<const void *>(&rb::updateKernel<true>);
    int perSm = 0;
    AOT_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, fn, rb::kScanThreads, 0));
    if (perSm <= 0) return false;
    rb::UpdateArgs u{m_->bufs(), m_->keyIndex(n_), m_->P[0].as<u64>(), n_, m_->scanTiles + 1, cfg_.bucket, cfg_.maxDepth,
                     cfg_.iterations, (long long)leafCapacity_, &m_->sortArena.ctl()->afterBar};
    // a thread per leaf, as many CTAs as fit; few meet at a barrier sooner
    const unsigned grid = std::min(gridFor(leafCapacity_ + 1, rb::kScanThreads), unsigned(std::min(perSm, 4)) * unsigned(smCount()));
    void *args[] = {&u};
    launchTeam(fn, args, rb::kScanThreads, grid, cfg_.stream);
    return true;
}

void TreeEngine::update()
{
    if (!built_) throw std::logic_error("adaptive_octree: call build() before update()");
    mark(MarkStart, 2);
    sortParticles();
    mark(MarkSorted);
    if (!passesFused())
    {
        refreshAll();
        mark(MarkRefreshed);
        for (unsigned i = 0; i < cfg_.iterations; ++i)
        {
            if (cfg_.kind == 0) octreePass(false, (long long)leafCapacity_);
            else binaryPass(false, (long long)leafCapacity_);
        }
        mark(MarkPassed);
        materializeCounts();
    }
    buildViews(cfg_.views);
    mark(MarkEnd);
}

// --------------------------------------------------------------------------
// stage timing
// --------------------------------------------------------------------------
static const char *const kMarkNames[] = {"keys + sort", "refresh", "passes", "counts + views"};

void TreeEngine::setProfiling(bool on)
{
    if (on)
        for (cudaEvent_t &e : m_->marks)
            if (!e) AOT_CHECK(cudaEventCreate(&e));
    profiling_ = on;
    marksRecorded_ = false;
}

// Records stage mark m on the tree's stream and moves the NVTX range on
// (call: 1 build, 2 update, given with MarkStart).  Nothing is recorded while
// the stream is captured: the events would become graph nodes and time the
// capture, not the work.
void TreeEngine::mark(Mark m, int call)
{
    if (!profiling_) return;
    if (m == MarkStart)
    {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        AOT_CHECK(cudaStreamIsCapturing(cfg_.stream, &cs));
        marking_ = cs == cudaStreamCaptureStatusNone;
        marksRecorded_ = false;
        markCall_ = call;
        nfMarks_ = 0;
        if (!marking_) return;
        nvtxRangePushA(call == 1 ? "build" : "update");
        nvtxRangePushA(kMarkNames[0]);
    }
    if (!marking_) return;
    AOT_CHECK(cudaEventRecord(m_->marks[m], cfg_.stream));
    if (m == MarkSorted && markCall_ == 1)
        AOT_CHECK(cudaEventRecord(m_->marks[MarkRefreshed], cfg_.stream));  // a build has no full refresh
    if (m != MarkStart)
    {
        nvtxRangePop();
        if (m != MarkEnd) nvtxRangePushA(kMarkNames[m]);
    }
    if (m == MarkEnd)
    {
        nvtxRangePop();
        marking_ = false;
        marksRecorded_ = true;
    }
}

// Events around one near-field launch.
void TreeEngine::markNearField(bool begin)
{
    if (!marking_) return;
    std::vector<cudaEvent_t> &ev = m_->nfMarks;
    const size_t k = size_t(nfMarks_) * 2 + (begin ? 0 : 1);
    if (k >= ev.size())
    {
        cudaEvent_t e;
        AOT_CHECK(cudaEventCreate(&e));
        ev.push_back(e);
    }
    AOT_CHECK(cudaEventRecord(ev[k], cfg_.stream));
    if (begin) nvtxRangePushA("near field");
    else
    {
        nvtxRangePop();
        ++nfMarks_;
    }
}

TreeEngine::StageTimes TreeEngine::stageTimes()
{
    StageTimes t;
    if (!marksRecorded_) return t;
    AOT_CHECK(cudaEventSynchronize(m_->marks[MarkEnd]));
    auto ms = [&](cudaEvent_t a, cudaEvent_t b) {
        float v = 0;
        AOT_CHECK(cudaEventElapsedTime(&v, a, b));
        return double(v);
    };
    const cudaEvent_t *e = m_->marks;
    t.keysAndSortMs = ms(e[MarkStart], e[MarkSorted]);
    t.refreshMs = ms(e[MarkSorted], e[MarkRefreshed]);
    t.passesMs = ms(e[MarkRefreshed], e[MarkPassed]);
    t.finishMs = ms(e[MarkPassed], e[MarkEnd]);
    t.totalMs = ms(e[MarkStart], e[MarkEnd]);
    for (int k = 0; k < nfMarks_; ++k)
    {
        const double v = ms(m_->nfMarks[2 * k], m_->nfMarks[2 * k + 1]);
        t.nearFieldMs += v;
        if (k == 0) t.nearFieldFirstMs = v;
    }
    t.nearFieldLaunches = nfMarks_;
    t.call = markCall_;
    t.valid = true;
    return t;
}

// update() runs a fixed number of passes (octree.cu:471-481,
// kdtree3d.cu:259-270), so fast-moving particles can leave overfull or
// mergeable leaves behind.  This variant keeps passing until a pass finds
// nothing to change: passes are launched in groups of cfg.iterations and the
// device state is read between groups.  A pass launched after convergence
// returns at once in every kernel (halted state), so a group may overshoot at
// no cost.  The passes themselves are update()'s, so the result equals
// update() with iterations = maxPasses.
void TreeEngine::updateUntilConverged(unsigned maxPasses, unsigned *changedPasses)
{
    if (!built_) throw std::logic_error("adaptive_octree: call build() before update()");
    if (maxPasses == 0) throw std::invalid_argument("adaptive_octree: updateUntilConverged needs maxPasses >= 1");
    cudaStream_t s = cfg_.stream;
    mark(MarkStart, 2);
    sortParticles();
    mark(MarkSorted);
    refreshAll();
    mark(MarkRefreshed);
    const unsigned group = std::max(1u, cfg_.iterations);
    unsigned launched = 0;
    while (launched < maxPasses)
    {
        const unsigned k = std::min(group, maxPasses - launched);
        for (unsigned i = 0; i < k; ++i)
        {
            if (cfg_.kind == 0) octreePass(false, (long long)leafCapacity_);
            else binaryPass(false, (long long)leafCapacity_);
        }
        launched += k;
        if (launched == maxPasses) break;
        // the raw state only: host-side sizes and the capacity model follow
        // the reference's readbacks, which happen in doBuffersNeedResize()
        AOT_CHECK(cudaMemcpyAsync(m_->hst, m_->st, sizeof(DeviceState), cudaMemcpyDeviceToHost, s));
        waitStream(s);
        if (m_->hst->error) throw std::runtime_error("adaptive_octree: a device scan gave up waiting (bounded look-back)");
        if (m_->hst->converged) break;
    }
    mark(MarkPassed);
    materializeCounts();
    buildViews(cfg_.views);
    mark(MarkEnd);
    if (changedPasses)
    {
        AOT_CHECK(cudaMemcpyAsync(m_->hst, m_->st, sizeof(DeviceState), cudaMemcpyDeviceToHost, s));
        waitStream(s);
        if (m_->hst->error) throw std::runtime_error("adaptive_octree: a device scan gave up waiting (bounded look-back)");
        *changedPasses = unsigned(m_->hst->updatePasses);
    }
}

void TreeEngine::computeViews(const adaptive_octree::ViewConfig &v)
{
    if (!built_) throw std::logic_error("adaptive_octree: call build() before computeViews()");
    buildViews(v);
}

// --------------------------------------------------------------------------
// views (tree_view.cu:755-1134)
// --------------------------------------------------------------------------
void TreeEngine::prepareViews(size_t capacity, const adaptive_octree::ViewConfig &v)
{
    if (!(v.treeStructure | v.particleCountsPerBox | v.particleMapping)) return;
    Impl &m = *m_;
    cudaStream_t s = cfg_.stream;
    m.viewLeafCap = std::max(m.viewLeafCap, capacity);
    m.viewParticleCap = std::max(m.viewParticleCap, n_);
    m.viewPrepared.treeStructure |= v.treeStructure;
    m.viewPrepared.particleCountsPerBox |= v.particleCountsPerBox;
    m.viewPrepared.particleMapping |= v.particleMapping;
    m.viewScratch = true;
    const int b = cfg_.kind == 0 ? 3 : 1;
    const size_t L = std::max<size_t>(m.viewLeafCap, 1);
    const size_t I = (L - 1) / ((size_t(1) << b) - 1);
    const size_t nodes = L + I;
    m.vBox.grow(nodes * 8, m.vBox.bytes, s);
    m.vSplit.grow(nodes, m.vSplit.bytes, s);
    m.vDepth.grow(nodes, m.vDepth.bytes, s);
    m.vParent.grow(nodes * 4, m.vParent.bytes, s);
    m.vChild.grow(nodes * 4, m.vChild.bytes, s);
    m.vLevelOffset.grow(66 * 4, m.vLevelOffset.bytes, s);
    m.vMaxDepth.grow(16, m.vMaxDepth.bytes, s);
    if (m.viewPrepared.particleCountsPerBox)
    {
        m.vPbegin.grow(nodes * 4, m.vPbegin.bytes, s);
        m.vPcount.grow((nodes + 1) * 4, m.vPcount.bytes, s);
    }
    if (m.viewPrepared.particleMapping) m.vPmap.grow(std::max<size_t>(m.viewParticleCap, 1) * 8, m.vPmap.bytes, s);
    m.vLeafLevel.reserve(L, s);
    m.vLeafToNode.reserve(L * 4, s);
    m.vLevels.reserve(4 * 66 * 4, s);
    m.vCandStart.reserve(L * 8, s);
    m.vCandLevel.reserve(L, s);
    for (int k = 0; k < 2; ++k)
    {
        m.vLvKeys[k].reserve(L * 8, s);
        m.vLvVals[k].reserve(L * 4, s);
        m.vLayKeys[k].reserve(std::max<size_t>(I, 1) * 8, s);
        m.vLayVals[k].reserve(std::max<size_t>(I, 1) * 4, s);
    }
    m.vIntStartSfc.reserve(std::max<size_t>(I, 1) * 8, s);
    m.vIntLevelSfc.reserve(std::max<size_t>(I, 1), s);
    m.vIntM.reserve(std::max<size_t>(I, 1) * 4, s);
    m.vIntStartLay.reserve(std::max<size_t>(I, 1) * 8, s);
    m.vIntLevelLay.reserve(std::max<size_t>(I, 1), s);
    m.viewSort.ensure(L, s, false);
}

void TreeEngine::syncViewSizes()
{
    Impl &m = *m_;
    if (!m.viewScratch || hostLeaves_ > m.viewLeafCap) return;
    const size_t k = cfg_.kind == 0 ? 7 : 1;
    m.viewNodesLogical = hostLeaves_ + (hostLeaves_ - 1) / k;
    if (m.viewPrepared.particleMapping) m.mappingLogical = hostActive_;
}

void TreeEngine::buildViews(const adaptive_octree::ViewConfig &v)
{
    prepared_.treeStructure |= v.treeStructure;
    prepared_.particleCountsPerBox |= v.particleCountsPerBox;
    prepared_.particleMapping |= v.particleMapping;
    if (!(v.treeStructure | v.particleCountsPerBox | v.particleMapping)) return;
    Impl &m = *m_;
    cudaStream_t s = cfg_.stream;
    if (!m.viewScratch || (v.particleCountsPerBox && !m.viewPrepared.particleCountsPerBox) ||
        (v.particleMapping && (!m.viewPrepared.particleMapping || n_ > m.viewParticleCap)))
    {
        tv::flagResizeKernel<<<1, 1, 0, s>>>(m.st), noteLaunch();
        AOT_LAUNCH_CHECK();
        return;
    }
    const int b = cfg_.kind == 0 ? 3 : 1;
    const int leafCap = int(m.viewLeafCap);
    const int intCap = (leafCap - 1) / ((1 << b) - 1);
    const tv::ViewBufs vb = m.viewBufs();
    const u64 *K0 = m.K[0].as<u64>(), *K1 = m.K[1].as<u64>();
    const u32 *B0 = m.B[0].as<u32>(), *B1 = m.B[1].as<u32>();
    const KeyIndex idx = m.keyIndex(n_);
    const int counts = v.particleCountsPerBox ? 1 : 0;
    AOT_CHECK(cudaMemsetAsync(vb.leavesPerLevel, 0, 66 * sizeof(int), s));
    if (b == 3)
    {
        tv::classifyKernel<3><<<gridFor(leafCap, tv::kThreads), tv::kThreads, 0, s>>>(K0, K1, m.st, leafCap, vb), noteLaunch();
        tv::metadataKernel<3><<<1, 1, 0, s>>>(m.st, leafCap, vb), noteLaunch();
    }
    else
    {
        tv::classifyKernel<1><<<gridFor(leafCap, tv::kThreads), tv::kThreads, 0, s>>>(K0, K1, m.st, leafCap, vb), noteLaunch();
        tv::metadataKernel<1><<<1, 1, 0, s>>>(m.st, leafCap, vb), noteLaunch();
    }
    AOT_LAUNCH_CHECK();
    if (intCap > 0)
    {
        // stable order of internal nodes by level (non-internal boundaries last)
        u64 *lk[2] = {vb.lvKeys, vb.lvKeysAlt};
        u32 *lv[2] = {vb.lvVals, vb.lvValsAlt};
        const int w1 = sortWithIndices(s, lk, lv, size_t(leafCap - 1), 1, m.viewSort, &m.st->error);
        if (b == 3)
            tv::layoutKeysKernel<3><<<gridFor(intCap, tv::kThreads), tv::kThreads, 0, s>>>(lk[w1], lv[w1], intCap, vb), noteLaunch();
        else
            tv::layoutKeysKernel<1><<<gridFor(intCap, tv::kThreads), tv::kThreads, 0, s>>>(lk[w1], lv[w1], intCap, vb), noteLaunch();
        AOT_LAUNCH_CHECK();
        u64 *yk[2] = {vb.layKeys, vb.layKeysAlt};
        u32 *yv[2] = {vb.layVals, vb.layValsAlt};
        const int w2 = sortWithIndices(s, yk, yv, size_t(intCap), 8, m.viewSort, &m.st->error);
        tv::materializeKernel<<<gridFor(intCap, tv::kThreads), tv::kThreads, 0, s>>>(yk[w2], yv[w2], intCap, vb), noteLaunch();
        if (b == 3)
            tv::internalNodesKernel<3><<<gridFor(intCap, tv::kThreads), tv::kThreads, 0, s>>>(m.st, leafCap, intCap,
                                                                                              idx, counts, vb), noteLaunch();
        else
            tv::internalNodesKernel<1><<<gridFor(intCap, tv::kThreads), tv::kThreads, 0, s>>>(m.st, leafCap, intCap,
                                                                                              idx, counts, vb), noteLaunch();
        AOT_LAUNCH_CHECK();
    }
    if (b == 3)
        tv::leafNodesKernel<3><<<gridFor(leafCap, tv::kThreads), tv::kThreads, 0, s>>>(K0, K1, B0, B1, m.st, leafCap,
                                                                                      counts, vb), noteLaunch();
    else
        tv::leafNodesKernel<1><<<gridFor(leafCap, tv::kThreads), tv::kThreads, 0, s>>>(K0, K1, B0, B1, m.st, leafCap,
                                                                                      counts, vb), noteLaunch();
    AOT_LAUNCH_CHECK();
    if (v.particleMapping && n_ > 0)
    {
        tv::mappingKernel<<<gridFor(n_, tv::kThreads), tv::kThreads, 0, s>>>(B0, B1, m.st, leafCap, n_, vb), noteLaunch();
        AOT_LAUNCH_CHECK();
    }
}

// --------------------------------------------------------------------------
// getters
// --------------------------------------------------------------------------
void TreeEngine::buffer(int which, const void **ptr, size_t *len, size_t *cap, size_t *elem) const
{
    const Impl &m = *m_;
    const int a = hostActiveBuffer_;
    const size_t nodes = m.viewScratch ? m.viewNodesLogical : 0;
    const size_t nodeCap = m.viewScratch ? m.vBox.bytes / 8 : 0;
    const void *p = nullptr;
    size_t l = 0, c = 0, e = 1;
    switch (which)
    {
    case ParticleKeys: p = m.P[0].p; l = c = n_; e = 8; break;
    case Perm: p = m.Perm[0].p; l = c = n_; e = 4; break;
    case Cornerstone: p = m.K[a].p; l = hostLeaves_ + 1; c = physCap_ + 1; e = 8; break;
    case LeafCounts: p = m.N[a].p; l = hostLeaves_; c = physCap_; e = 4; break;
    case NearFieldCounts:
        if (cfg_.kind == 1) throw std::logic_error("Tree: Binary NFCount is not implemented yet");
        p = m.NF[a].p; l = hostLeaves_; c = physCap_; e = 4; break;
    case SfcBoxIndex: p = m.vBox.p; l = nodes; c = nodeCap; e = 8; break;
    case HasBoxSplit: p = m.vSplit.p; l = nodes; c = nodeCap; e = 1; break;
    case BoxDepth: p = m.vDepth.p; l = nodes; c = nodeCap; e = 1; break;
    case ParentIndex: p = m.vParent.p; l = nodes; c = nodeCap; e = 4; break;
    case ChildIndex: p = m.vChild.p; l = nodes; c = nodeCap; e = 4; break;
    case LevelOffset:
        p = m.vLevelOffset.p;
        l = c = m.viewScratch ? (cfg_.kind == 0 ? 23 : 65) : 0;
        e = 4;
        break;
    case ParticleBeginIndex:
        p = m.vPbegin.p;
        l = (m.viewScratch && m.viewPrepared.particleCountsPerBox) ? nodes : 0;
        c = m.vPbegin.bytes / 4;
        e = 4;
        break;
    case ParticleCounts:
        p = m.vPcount.p;
        l = (m.viewScratch && m.viewPrepared.particleCountsPerBox) ? nodes + 1 : 0;
        c = m.vPcount.bytes / 4;
        e = 4;
        break;
    case LeafBegins: p = m.B[a].p; l = hostLeaves_ + 1; c = physCap_ + 1; e = 4; break;
    case SfcParticleIndex:
        p = m.vPmap.p;
        l = (m.viewScratch && m.viewPrepared.particleMapping) ? m.mappingLogical : 0;
        c = m.vPmap.bytes / 8;
        e = 8;
        break;
    default: throw std::invalid_argument("adaptive_octree: unknown buffer");
    }
    if (ptr) *ptr = p;
    if (len) *len = l;
    if (cap) *cap = c;
    if (elem) *elem = e;
}

const int *TreeEngine::numLeavesDevice() const { return &m_->st->numLeaves; }
const int *TreeEngine::numNodesDevice() const { return &m_->st->numNodes; }
const unsigned *TreeEngine::numActiveParticlesDevice() const { return &m_->st->numActiveParticles; }

unsigned TreeEngine::maxAchievedDepth() const
{
    const Impl &m = *m_;
    cudaStream_t s = cfg_.stream;
    if (cfg_.kind == 1 && !(cfg_.views.treeStructure | cfg_.views.particleCountsPerBox | cfg_.views.particleMapping))
    {
        // kdtree3d.cu: maxAchievedDepth from the cornerstone when no view is configured
        std::vector<u64> k(hostLeaves_ + 1);
        AOT_CHECK(cudaMemcpyAsync(k.data(), m.K[hostActiveBuffer_].p, k.size() * 8, cudaMemcpyDeviceToHost, s));
        waitStream(s);
        unsigned d = 0;
        for (size_t i = 0; i + 1 < k.size(); ++i) d = std::max(d, unsigned(clz64(k[i + 1] - k[i])));
        return d;
    }
    if (!m.viewScratch) return 0;
    u8 v = 0;
    AOT_CHECK(cudaMemcpyAsync(&v, m.vMaxDepth.p, 1, cudaMemcpyDeviceToHost, s));
    waitStream(s);
    return v;
}

}  // namespace aot
