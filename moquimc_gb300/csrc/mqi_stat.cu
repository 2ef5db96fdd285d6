// Statistics kernels: the reference's uncertainty estimator, a batch estimator, and tally scaling.
//
// The reference computes, per stat-ROI voxel, sigma_i = sqrt((S2_i/n - (S1_i/n)^2) / (n - 1)) and
// mean_i = S1_i/n from per-step dose and dose^2 tallies (calculate_standard_deviation,
// moqui/kernel_functions/mqi_variables.hpp:19-48), then averages sigma_i/mean_i over the voxels
// whose mean exceeds threshold * max on the host (tps_env::calculate_stat,
// moqui/base/environments/mqi_tps_env.hpp:1338-1426).  Here both passes are device reductions
// over the dense tallies (one max pass, one sum pass), so only two numbers cross to the host.
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "mqi_internal.h"

namespace mqi_gpu
{

namespace
{

/// Positive doubles order like their bit patterns.  The sweeps below compare those: GB300's FP64
/// pipe is narrow, and an FP64 comparison per voxel alone would take as long as the voxel's bytes.
/// 0 for a value that is not above zero (NaN included).
__device__ inline unsigned long long
positive_bits(double v) {
    const unsigned long long b = (unsigned long long) __double_as_longlong(v);
    return b - 1ull < 0x7FF0000000000000ull ? b : 0ull;
}

__device__ inline double
warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    return v;
}

/// Per-voxel mean and relative sigma of the reference estimator (mqi_variables.hpp:38-45):
/// sigma is evaluated in double and rounded to float before the square root, as the reference
/// stores it in a float array; a negative variance from rounding gives 0 (the reference's sqrtf
/// of it would be NaN).
__device__ inline void
ref_mean_sigma(double s1, double s2, double n, float& mean, float& sigma) {
    const double m = s1 / n;
    float        v = (float) ((s2 / n - m * m) / (n - 1.0));
    if (!(v > 0.0f)) v = 0.0f;
    sigma = sqrtf(v);
    mean  = (float) m;
}

/// Batch estimator: relative standard error of the mean over B batches.
__device__ inline void
batch_mean_rel(double s1, double s2, double B, double& mean, double& rel) {
    mean = s1 / B;
    double var = (s2 / B - mean * mean) / (B - 1.0);   // variance of one batch
    if (!(var > 0.0)) var = 0.0;
    rel = (mean > 0.0) ? sqrt(var / B) / mean : 0.0;
}

/// Both estimators' means are monotone in s1 (a division by nh, then at most one rounding to float),
/// so the largest mean is that of the largest s1: the pass over the volume is an integer maximum,
/// and one division follows it.  Block (x, y) sweeps a share of scenario y's n voxels.
constexpr int kStatBlock = 256;

/// The first value (s1) of voxel i, and with kPair the second beside it: one 16-byte load.
template<bool kPair>
__device__ __forceinline__ double
stat_s1(const double* __restrict__ s1, uint64_t i, uint32_t stride, double& s2) {
    if constexpr (kPair) {
        const double2 v = reinterpret_cast<const double2*>(s1)[i];
        s2              = v.y;
        return v.x;
    } else {
        return s1[i * stride];
    }
}

template<bool kPair>
__global__ void __launch_bounds__(kStatBlock)
k_stat_max(const double* __restrict__ s1, uint64_t n, uint32_t stride, unsigned long long* __restrict__ scratch) {
    __shared__ unsigned long long best;
    if (threadIdx.x == 0) best = 0ull;
    __syncthreads();
    s1 += blockIdx.y * n * stride;
    unsigned long long m    = 0ull;
    const uint64_t     step = (uint64_t) gridDim.x * blockDim.x;
    double             s2;
#pragma unroll 4
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += step)
        m = max(m, positive_bits(stat_s1<kPair>(s1, i, stride, s2)));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xFFFFFFFFu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(&best, m);
    __syncthreads();
    if (threadIdx.x == 0 && best) atomicMax(scratch + 3 * blockIdx.y, best);
}

/// The sum over the voxels above the threshold.  A voxel's division and square root run only when
/// s1 can be above the cut (an integer comparison with a bound that allows for the roundings of
/// the mean); those that are decide it as the reference does.
template<bool kPair>
__global__ void __launch_bounds__(kStatBlock)
k_stat_sum(const double* __restrict__ s1, const double* __restrict__ s2, uint64_t n, uint32_t stride, double nh,
           int mode, float threshold, unsigned long long* __restrict__ scratch) {
    __shared__ double             part[kStatBlock / 32], s_cut;
    __shared__ unsigned long long s_low, count;
    s1 += blockIdx.y * n * stride;
    s2 += blockIdx.y * n * stride;
    scratch += 3 * blockIdx.y;
    if (threadIdx.x == 0) {
        const double top  = __longlong_as_double((long long) scratch[0]) / nh;
        const double cut  = (mode == 0 ? (double) (float) top : top) * (double) threshold;
        // below the normal floats the mean's rounding is not relative: every positive s1 is looked at
        const double low  = cut > 1e-30 ? cut * nh * (1.0 - 1e-6) : 0.0;
        s_cut             = cut;
        s_low             = positive_bits(low);
        count             = 0ull;
    }
    __syncthreads();
    const double             cut = s_cut;
    const unsigned long long low = s_low;
    double                   acc = 0.0;
    unsigned int             cnt = 0;
    const uint64_t           step = (uint64_t) gridDim.x * blockDim.x;
#pragma unroll 4
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += step) {
        double       b = 0.0;
        const double a = stat_s1<kPair>(s1, i, stride, b);
        if (!(positive_bits(a) > low)) continue;
        if (!kPair) b = s2[i * stride];
        if (mode == 0) {
            float mean, sigma;
            ref_mean_sigma(a, b, nh, mean, sigma);
            if ((double) mean > cut) {   // dose_mean[i] > dose_max * stat_threshold (mqi_tps_env.hpp:1418)
                acc += (double) (sigma / mean);
                ++cnt;
            }
        } else {
            double mean, rel;
            batch_mean_rel(a, b, nh, mean, rel);
            if (mean > cut) {
                acc += rel;
                ++cnt;
            }
        }
    }
    acc = warp_sum(acc);
    cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
    if ((threadIdx.x & 31) == 0) {
        part[threadIdx.x >> 5] = acc;
        if (cnt) atomicAdd(&count, (unsigned long long) cnt);
    }
    __syncthreads();
    if (threadIdx.x == 0 && count) {
        double sum = 0.0;
        for (int w = 0; w < kStatBlock / 32; ++w) sum += part[w];
        atomicAdd(reinterpret_cast<double*>(scratch + 2), sum);
        atomicAdd(scratch + 1, count);
    }
}

__global__ void
k_batch_fold(double* __restrict__ tally, uint32_t stride, double* __restrict__ s1, double* __restrict__ s2, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x) {
        const double t = tally[i * stride];
        if (t != 0.0) {
            s1[i] += t;
            s2[i] += t * t;
            tally[i * stride] = 0.0;
        }
    }
}

__global__ void
k_scale(double* __restrict__ a, uint32_t stride, uint64_t n, double w) {
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x)
        a[i * stride] *= w;
}

__global__ void
k_copy_strided(const double* __restrict__ a, uint32_t stride, double* __restrict__ out, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x)
        out[i] = a[i * stride];
}

__global__ void
k_copy_scaled(const double* __restrict__ a, double* __restrict__ out, uint64_t n, double w) {
    for (uint64_t i = blockIdx.x * (uint64_t) blockDim.x + threadIdx.x; i < n; i += (uint64_t) gridDim.x * blockDim.x)
        out[i] = a[i] * w;
}

unsigned
grid_for(uint64_t n, int sms) {
    const uint64_t b = (n + 255) / 256;
    const uint64_t cap = (uint64_t) sms * 16;
    return (unsigned) (b < cap ? (b ? b : 1) : cap);
}

}   // namespace

/// The estimate of each of `copies` scenarios, n voxels each, one behind the other.  Bound by HBM:
/// two passes over s1 (16 B a voxel each for the interleaved pair).  One launch a pass for all
/// scenarios: 0.76 and 1.12 ms for both of the 512 x 512 x 200 CT and 21 scenarios of 256 x 256 x 200
/// together.  On the CT alone the passes took 0.78 and 1.81 ms with the FP64 divisions done
/// for every voxel, and each scenario waited for the one before it.
cudaError_t
launch_stat(const double* s1, const double* s2, uint64_t n, uint32_t stride, uint32_t copies, double nh, int mode,
            float threshold, int sms, unsigned long long* scratch, cudaStream_t s) {
    // scratch, per scenario: [0] bits of the largest s1, [1] count, [2] sum (as double bits)
    cudaError_t e = cudaMemsetAsync(scratch, 0, 3 * copies * sizeof(unsigned long long), s);
    if (e != cudaSuccess || n == 0) return e;
    const uint64_t need = (n + kStatBlock - 1) / kStatBlock, share = std::max<uint64_t>((uint64_t) sms * 8 / copies, 1);
    const dim3     g((unsigned) std::min(need, share), copies);
    if (stride == 2 && s2 == s1 + 1 && reinterpret_cast<uintptr_t>(s1) % 16 == 0) {
        k_stat_max<true><<<g, kStatBlock, 0, s>>>(s1, n, stride, scratch);
        k_stat_sum<true><<<g, kStatBlock, 0, s>>>(s1, s2, n, stride, nh, mode, threshold, scratch);
    } else {
        k_stat_max<false><<<g, kStatBlock, 0, s>>>(s1, n, stride, scratch);
        k_stat_sum<false><<<g, kStatBlock, 0, s>>>(s1, s2, n, stride, nh, mode, threshold, scratch);
    }
    return cudaGetLastError();
}

cudaError_t
launch_batch_fold(double* tally, uint32_t stride, double* s1, double* s2, uint64_t n, int sms, cudaStream_t s) {
    k_batch_fold<<<grid_for(n, sms), 256, 0, s>>>(tally, stride, s1, s2, n);
    return cudaGetLastError();
}

cudaError_t
launch_scale(double* a, uint32_t stride, uint64_t n, double w, int sms, cudaStream_t s) {
    k_scale<<<grid_for(n, sms), 256, 0, s>>>(a, stride, n, w);
    return cudaGetLastError();
}

cudaError_t
launch_copy_strided(const double* a, uint32_t stride, double* out, uint64_t n, int sms, cudaStream_t s) {
    k_copy_strided<<<grid_for(n, sms), 256, 0, s>>>(a, stride, out, n);
    return cudaGetLastError();
}

cudaError_t
launch_copy_scaled(const double* a, double* out, uint64_t n, double w, int sms, cudaStream_t s) {
    k_copy_scaled<<<grid_for(n, sms), 256, 0, s>>>(a, out, n, w);
    return cudaGetLastError();
}

}   // namespace mqi_gpu
