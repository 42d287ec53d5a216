// keygen.cuh -- particle coordinates -> SFC keys, fused with the sort's digit histogram.
//
// Replaces computeSfcKeysKernel (sfc_keys.cuh:501-532) and
// computeSfcKeysBinaryKernel (kdtree3d_rebalance.cuh:247-273).  Each CTA
// streams coordinates with 128-bit loads (4 floats or 2 doubles per axis per
// thread step), writes the keys with 128-bit stores and accumulates the digit
// counts of the sort's passes in shared memory, so the sort never
// re-reads the keys for its histogram.  The identity permutation is not
// written: the first sort pass generates it from the input index.  A plan
// kernel before it (planKernel) samples the keys and picks the passes; the
// last CTA to add its counts turns them into the passes' digit starts.
#pragma once

#include "sfc.cuh"
#include "sort_plan.cuh"

namespace aot
{
enum class Curve : int { Morton = 0, Hilbert = 1, Binary = 2 };

template <class Real>
struct KeygenParams
{
    QuantBox<Real> q;
    BinaryGeometry g;
};

// What a thread keeps for the keys of its particles.  sPair: the two-level
// Hilbert table in shared memory.
template <class Real, Curve C>
struct KeyMaker
{
    QuantAxis<Real> x, y, z;
    const u32 *sPair;
    const BinaryGeometry &g;
    __device__ __forceinline__ KeyMaker(const KeygenParams<Real> &p, const u32 *pair)
        : x(quantAxis(p.q.xmin, p.q.ilx, p.q.bx)), y(quantAxis(p.q.ymin, p.q.ily, p.q.by)),
          z(quantAxis(p.q.zmin, p.q.ilz, p.q.bz)), sPair(pair), g(p.g)
    {
    }
    __device__ __forceinline__ u64 operator()(Real px, Real py, Real pz) const
    {
        if constexpr (C == Curve::Binary)
        {
            return binaryKey<Real>(px, py, pz, g);
        }
        else
        {
            const u32 ix = quantise(px, x), iy = quantise(py, y), iz = quantise(pz, z);
            u64 k;
            if constexpr (C == Curve::Hilbert) k = hilbertKeyPairs(ix, iy, iz, sPair);
            else k = mortonKey(ix, iy, iz);
            return isEscaped<Real>(px, py, pz) ? kInvalidKey : k;
        }
    }
};

// Counts the digits of passes firstPass to 7 of a key in
// sh[kMaxPasses][kRadix] (shared memory).
__device__ __forceinline__ void countDigits(u64 k, int firstPass, u32 *sh)
{
    static_assert(sort::kMaxPasses == 8 && sort::kRadixBits == 8, "a byte per digit");
    const u32 half[2] = {u32(k), u32(k >> 32)};
#pragma unroll
    for (int h = 0; h < 2; ++h)
    {
        if (firstPass >= 4 * (h + 1)) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (4 * h + b >= firstPass) atomicAdd(sh + (4 * h + b) * sort::kRadix + ((half[h] >> (8 * b)) & 0xffu), 1u);
    }
}

constexpr int kKeygenThreads = 256;

// The two-level Hilbert table to shared memory.
__device__ __forceinline__ void loadPairTable(u32 *sPair)
{
    for (int i = threadIdx.x; i < kHilbertPairEntries; i += blockDim.x) sPair[i] = __ldg(gHilbertPairs.entry + i);
}

// Start of a planned sort: the control block, zeroed digit counts and the
// plan, from the keys of particles at random positions.
template <class Real, Curve C>
static __global__ void __launch_bounds__(sort::kPlanThreads)
    planKernel(const Real *__restrict__ x, const Real *__restrict__ y, const Real *__restrict__ z, size_t n,
               const KeygenParams<Real> prm, sort::PlanArgs plan, sort::SortControl *ctl, u32 *hist)
{
    __shared__ u32 sPair[C == Curve::Hilbert ? kHilbertPairEntries : 1];
    if constexpr (C == Curve::Hilbert) loadPairTable(sPair);
    __syncthreads();
    const KeyMaker<Real, C> make(prm, sPair);
    const auto keyAt = [&](size_t i, u32 &) { return make(x[i], y[i], z[i]); };
    sort::planSort(keyAt, n, plan, ctl, hist, size_t(sort::kPassSlots) * sort::kRadix);
}

// Vec: particles per thread step (4 for float4, 2 for double2, 1 scalar).
// hist (with bins and ctl) or nullptr: the digit counts of the plan's passes
// and their starts.
template <class Real, Curve C, int Vec>
static __global__ void __launch_bounds__(kKeygenThreads)
    keygenKernel(const Real *__restrict__ x, const Real *__restrict__ y, const Real *__restrict__ z, size_t n,
                 const KeygenParams<Real> prm, u64 *__restrict__ keys, u32 *__restrict__ hist,
                 u32 *__restrict__ bins, sort::SortControl *ctl)
{
    __shared__ u32 sh[sort::kMaxPasses][sort::kRadix];
    __shared__ u32 sPair[C == Curve::Hilbert ? kHilbertPairEntries : 1];
    for (int i = threadIdx.x; i < sort::kMaxPasses * sort::kRadix; i += blockDim.x) (&sh[0][0])[i] = 0;
    if constexpr (C == Curve::Hilbert) loadPairTable(sPair);
    const int firstPass = hist ? int(ctl->first) : sort::kMaxPasses;
    __syncthreads();

    const KeyMaker<Real, C> make(prm, sPair);
    const size_t groups = n / Vec;
    const size_t stride = size_t(gridDim.x) * blockDim.x;
    for (size_t gi = blockIdx.x * size_t(blockDim.x) + threadIdx.x; gi < groups; gi += stride)
    {
        const size_t base = gi * Vec;
        Real vx[Vec], vy[Vec], vz[Vec];
        if constexpr (Vec == 4)
        {
            const float4 a = __ldcs(reinterpret_cast<const float4 *>(x) + gi);
            const float4 b = __ldcs(reinterpret_cast<const float4 *>(y) + gi);
            const float4 c = __ldcs(reinterpret_cast<const float4 *>(z) + gi);
            vx[0] = a.x; vx[1] = a.y; vx[2] = a.z; vx[3] = a.w;
            vy[0] = b.x; vy[1] = b.y; vy[2] = b.z; vy[3] = b.w;
            vz[0] = c.x; vz[1] = c.y; vz[2] = c.z; vz[3] = c.w;
        }
        else if constexpr (Vec == 2)
        {
            const double2 a = __ldcs(reinterpret_cast<const double2 *>(x) + gi);
            const double2 b = __ldcs(reinterpret_cast<const double2 *>(y) + gi);
            const double2 c = __ldcs(reinterpret_cast<const double2 *>(z) + gi);
            vx[0] = a.x; vx[1] = a.y;
            vy[0] = b.x; vy[1] = b.y;
            vz[0] = c.x; vz[1] = c.y;
        }
        else
        {
            vx[0] = x[base];
            vy[0] = y[base];
            vz[0] = z[base];
        }
        u64 k[Vec];
#pragma unroll
        for (int j = 0; j < Vec; ++j)
        {
            k[j] = make(vx[j], vy[j], vz[j]);
            countDigits(k[j], firstPass, &sh[0][0]);
        }
        if constexpr (Vec == 4)
        {
            ulonglong2 *o = reinterpret_cast<ulonglong2 *>(keys + base);
            o[0] = make_ulonglong2(k[0], k[1]);  // default policy: the sort reads the keys next
            o[1] = make_ulonglong2(k[2], k[3]);
        }
        else if constexpr (Vec == 2)
        {
            *reinterpret_cast<ulonglong2 *>(keys + base) = make_ulonglong2(k[0], k[1]);
        }
        else
        {
            keys[base] = k[0];
        }
    }
    // tail particles that do not fill a vector
    for (size_t i = groups * Vec + blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += stride)
    {
        const u64 k = make(x[i], y[i], z[i]);
        keys[i] = k;
        countDigits(k, firstPass, &sh[0][0]);
    }
    if (!hist) return;
    __syncthreads();
    for (int i = firstPass * sort::kRadix + threadIdx.x; i < sort::kMaxPasses * sort::kRadix; i += blockDim.x)
    {
        const u32 v = (&sh[0][0])[i];
        if (v) atomicAdd(hist + i, v);
    }
    // the last CTA: the digit starts of every pass
    __shared__ bool sLast;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) sLast = atomicAdd(&ctl->keygenDone, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!sLast) return;
    __threadfence();
    sort::scanBins(hist, bins, firstPass, sort::kMaxPasses);
}

}  // namespace aot
