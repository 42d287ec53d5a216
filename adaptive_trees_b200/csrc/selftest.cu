// selftest.cu -- checks that the engine's bounded device waits end.
//
// Every decoupled look-back of the engine (the radix sort's per-digit
// prefixes, the rebalance decide+scan) polls earlier tiles for a bounded
// number of rounds; when that runs out the kernel records kErrLookback in its
// error word and finishes, so the host sees an error status instead of a hung
// GPU.  These probes build the one situation in which the limit is reached --
// tile 0 is never processed, so nothing ever publishes its status word -- and
// let the waits of the later tiles run out under a small limit:
//   which 0: one onesweep pass (8-bit digits, 10 keys per thread) over 4
//            tiles of zero keys, launched with 3 CTAs and the tile counter
//            starting at 1, so the CTAs take tiles 1..3;
//   which 1: the decide+scan look-back of tiles 1..3 over a zeroed status
//            array.
// The launches by team (grid_barrier.cuh) wait for the CTAs of their team and,
// in the placements, for a parent's place; teamWaitProbe runs one CTA of them
// where nobody else comes:
//   which 0: a grid barrier of a team of 2, then (a small and a large team
//            count their arrivals in different words) of 400;
//   which 1: the roll of a launch, with nobody on it and no limit but the wait's;
//   which 2: the octree's placement of a unit whose parent never places it;
//   which 3: the same of the binary tree.
// Every index stays inside its buffer (a tile that gave up writes its keys at
// the prefix it has, below the prefix of the full input), and every wait is
// bounded by `spinLimit`, so the probes neither fault nor hang.
#include <stdexcept>
#include <string>

#include "binlevel.cuh"
#include "engine_util.cuh"
#include "radix_sort.cuh"
#include "rebalance.cuh"

namespace aot
{
namespace
{
constexpr int kProbeItems = 10;
constexpr int kProbeTile = sort::kThreads * kProbeItems;
constexpr int kProbeTiles = 4;

__global__ void __launch_bounds__(sort::kThreads, 1)
    sortWaitProbeKernel(const u64 *keysIn, u64 *keysOut, u32 *valsOut, size_t n, const u32 *bins, u32 *tileCounter,
                        u64 *status, int *error, unsigned spinLimit)
{
    sort::onesweepTile<8, kProbeItems>(sort::ContiguousTiles<kProbeTile>{n, bins}, keysIn, nullptr, keysOut,
                                       valsOut, 0, tileCounter, status, sort::passTag(1), error, 8, spinLimit);
}

__global__ void scanWaitProbeKernel(u64 *status, int *error, unsigned spinLimit, i64 *prefix)
{
    const i64 p = rb::lookback(status, blockIdx.x + 1, 1, error, spinLimit);
    if (threadIdx.x == 0) prefix[blockIdx.x] = p;
}

__global__ void __launch_bounds__(lb::kThreads) barrierProbeKernel(GridBarrier *bar, u32 size, unsigned spinLimit, int *error)
{
    if (!gridBarrier(bar, Team{0, size}, spinLimit) && threadIdx.x == 0) *error = kErrLookback;
}

__global__ void __launch_bounds__(lb::kThreads) rollProbeKernel(GridBarrier *bar, unsigned spinLimit, int *error)
{
    if (!closeRoll(bar, spinLimit, 0xffffffffu) && threadIdx.x == 0) *error = kErrLookback;
}

__global__ void __launch_bounds__(lb::kThreads) placeProbeKernel(lb::Arena a, u64 *K, u32 *B, u32 *N, unsigned spinLimit, int *error)
{
    lb::placeUnits<false, false, false>(a, Team{0, 1}, K, B, nullptr, N, nullptr, 1, 8, nullptr, spinLimit);
    __syncthreads();
    if (threadIdx.x == 0) *error = a.ctl->error;
}

__global__ void __launch_bounds__(lb::kThreads) binaryPlaceProbeKernel(bl::Arena a, u64 *K, u32 *B, u32 *N, unsigned spinLimit, int *error)
{
    bl::placeUnits(a, Team{0, 1}, K, B, N, 1, 8, spinLimit);
    __syncthreads();
    if (threadIdx.x == 0) *error = a.ctl->error;
}

// A CTA that fills its SM's shared memory and waits (bounded by the clock and by polls).
constexpr size_t kHoldBytes = 200 * 1024;
constexpr int kHoldMilliseconds = 2000;
__global__ void __launch_bounds__(32) holdKernel(unsigned long long nanoseconds)
{
    extern __shared__ u32 held[];
    unsigned long long start, now;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(start));
    u32 polls = 0;
    do
    {
        __nanosleep(1000);
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    } while (now - start < nanoseconds && ++polls < (1u << 22));
    if (threadIdx.x == 0) held[0] = polls;
}

// Device allocations of the probe, freed on every exit path.
struct ProbeMem
{
    void *p = nullptr;
    explicit ProbeMem(size_t bytes) { AOT_CHECK(cudaMalloc(&p, bytes)); }
    ~ProbeMem() { cudaFree(p); }
    template <class T> T *as() const { return static_cast<T *>(p); }
};

struct ProbeStream
{
    cudaStream_t s = nullptr;
    ProbeStream() { AOT_CHECK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking)); }
    ~ProbeStream() { cudaStreamDestroy(s); }
};
}  // namespace

int TreeEngine::boundedWaitProbe(int which, unsigned spinLimit)
{
    if (which != 0 && which != 1) throw std::invalid_argument("ao_selftest_bounded_wait: which must be 0 or 1");
    if (spinLimit == 0 || spinLimit > (1u << 16))
        throw std::invalid_argument("ao_selftest_bounded_wait: spin_limit must be in [1, 65536]");
    ProbeStream ps;
    const cudaStream_t s = ps.s;
    ProbeMem err(sizeof(int));
    AOT_CHECK(cudaMemsetAsync(err.p, 0, sizeof(int), s));
    if (which == 0)
    {
        const size_t n = size_t(kProbeTiles) * kProbeTile;
        ProbeMem keysIn(n * sizeof(u64)), keysOut(n * sizeof(u64)), valsOut(n * sizeof(u32));
        ProbeMem bins(sort::kRadix * sizeof(u32)), counter(sizeof(u32));
        ProbeMem status(size_t(kProbeTiles) * sort::kRadix * sizeof(u64));
        AOT_CHECK(cudaMemsetAsync(keysIn.p, 0, n * sizeof(u64), s));
        AOT_CHECK(cudaMemsetAsync(bins.p, 0, sort::kRadix * sizeof(u32), s));  // every key has digit 0
        AOT_CHECK(cudaMemsetAsync(status.p, 0, size_t(kProbeTiles) * sort::kRadix * sizeof(u64), s));
        const u32 firstTile = 1;  // tile 0 is never taken, so it never publishes
        AOT_CHECK(cudaMemcpyAsync(counter.p, &firstTile, sizeof(u32), cudaMemcpyHostToDevice, s));
        const int smem = int(sizeof(sort::SharedPass<8, kProbeItems>));
        AOT_CHECK(cudaFuncSetAttribute(sortWaitProbeKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        sortWaitProbeKernel<<<kProbeTiles - 1, sort::kThreads, smem, s>>>(
            keysIn.as<u64>(), keysOut.as<u64>(), valsOut.as<u32>(), n, bins.as<u32>(), counter.as<u32>(),
            status.as<u64>(), err.as<int>(), spinLimit);
        AOT_LAUNCH_CHECK();
        AOT_CHECK(cudaStreamSynchronize(s));
    }
    else
    {
        ProbeMem status(size_t(kProbeTiles) * sizeof(u64)), prefix(size_t(kProbeTiles) * sizeof(i64));
        AOT_CHECK(cudaMemsetAsync(status.p, 0, size_t(kProbeTiles) * sizeof(u64), s));
        scanWaitProbeKernel<<<kProbeTiles - 1, 32, 0, s>>>(status.as<u64>(), err.as<int>(), spinLimit,
                                                           prefix.as<i64>());
        AOT_LAUNCH_CHECK();
        AOT_CHECK(cudaStreamSynchronize(s));
    }
    int error = 0;
    AOT_CHECK(cudaMemcpy(&error, err.p, sizeof(int), cudaMemcpyDeviceToHost));
    return error;
}

int TreeEngine::teamWaitProbe(int which, unsigned spinLimit)
{
    if (which < 0 || which > 3) throw std::invalid_argument("ao_selftest_team_wait: which must be 0 to 3");
    if (spinLimit == 0 || spinLimit > (1u << 16))
        throw std::invalid_argument("ao_selftest_team_wait: spin_limit must be in [1, 65536]");
    ProbeStream ps;
    const cudaStream_t s = ps.s;
    ProbeMem err(2 * sizeof(int)), bar(sizeof(GridBarrier));
    AOT_CHECK(cudaMemsetAsync(err.p, 0, 2 * sizeof(int), s));
    AOT_CHECK(cudaMemsetAsync(bar.p, 0, sizeof(GridBarrier), s));
    // one unit of 8 leaves, whose first leaf's index never comes
    ProbeMem rows(lb::kRow * sizeof(u32)), child(8 * sizeof(u32)), sub(sizeof(u64)), offset(sizeof(u32));
    ProbeMem ctl(std::max(sizeof(lb::Control), sizeof(bl::Control)));
    ProbeMem K(8 * sizeof(u64)), B(8 * sizeof(u32)), N(8 * sizeof(u32));
    AOT_CHECK(cudaMemsetAsync(rows.p, 0, lb::kRow * sizeof(u32), s));
    AOT_CHECK(cudaMemsetAsync(child.p, 0xff, 8 * sizeof(u32), s));  // kLeaf
    AOT_CHECK(cudaMemsetAsync(offset.p, 0xff, sizeof(u32), s));     // kPending
    AOT_CHECK(cudaMemsetAsync(ctl.p, 0, std::max(sizeof(lb::Control), sizeof(bl::Control)), s));
    int *error = err.as<int>();
    if (which == 0)
    {
        barrierProbeKernel<<<1, lb::kThreads, 0, s>>>(bar.as<GridBarrier>(), 2, spinLimit, error);
        AOT_CHECK(cudaMemsetAsync(bar.p, 0, sizeof(GridBarrier), s));
        barrierProbeKernel<<<1, lb::kThreads, 0, s>>>(bar.as<GridBarrier>(), 400, spinLimit, error + 1);
    }
    else if (which == 1)
    {
        rollProbeKernel<<<1, lb::kThreads, 0, s>>>(bar.as<GridBarrier>(), spinLimit, error);
    }
    else if (which == 2)
    {
        lb::Arena a{};
        a.rows = rows.as<u32>();
        a.child = child.as<u32>();
        a.sub = sub.as<u64>();
        a.offset = offset.as<u32>();
        a.ctl = ctl.as<lb::Control>();
        a.cap = 1;
        placeProbeKernel<<<1, lb::kThreads, 0, s>>>(a, K.as<u64>(), B.as<u32>(), N.as<u32>(), spinLimit, error);
    }
    else
    {
        bl::Arena a{};
        a.rows = rows.as<u32>();
        a.child = child.as<u32>();
        a.sub = sub.as<u64>();
        a.offset = offset.as<u32>();
        a.ctl = ctl.as<bl::Control>();
        a.cap = 1;
        binaryPlaceProbeKernel<<<1, lb::kThreads, 0, s>>>(a, K.as<u64>(), B.as<u32>(), N.as<u32>(), spinLimit, error);
    }
    AOT_LAUNCH_CHECK();
    AOT_CHECK(cudaStreamSynchronize(s));
    int e[2] = {0, 0};
    AOT_CHECK(cudaMemcpy(e, err.p, sizeof(e), cudaMemcpyDeviceToHost));
    return which == 0 && e[0] != e[1] ? 0 : e[0];
}

void TreeEngine::holdSms(int sms, int milliseconds, cudaStream_t s)
{
    if (sms < 1 || sms > smCount()) throw std::invalid_argument("ao_selftest_hold_sms: sms must be in [1, the device's]");
    if (milliseconds < 1 || milliseconds > kHoldMilliseconds)
        throw std::invalid_argument("ao_selftest_hold_sms: milliseconds must be in [1, 2000]");
    AOT_CHECK(cudaFuncSetAttribute(holdKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kHoldBytes)));
    holdKernel<<<unsigned(sms), 32, kHoldBytes, s>>>((unsigned long long)milliseconds * 1000000ull);
    AOT_LAUNCH_CHECK();
}
}  // namespace aot
