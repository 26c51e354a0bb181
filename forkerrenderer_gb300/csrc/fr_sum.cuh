// Sums of a gradient's partial sums (k_grad_reduce). The host test compiles the same code.
#pragma once

#include <stddef.h>

#include "fr_exact.cuh"

namespace frx
{

// (hi, lo) += x: hi the rounded running sum, lo the sum of its rounding errors.
FR_HD void two_sum_add(float& hi, float& lo, float x)
{
    const float s = hi + x;
    const float b = s - hi;
    const float e = (hi - (s - b)) + (x - b);
    hi = s;
    lo = lo + e;
}

// The sum in FP64 (term c into sum c mod 8), for what the FP32 form cannot hold.
#ifdef __CUDACC__
__host__ __device__ __noinline__
#else
inline
#endif
float sum_fp64(const float* src, size_t stride, int n)
{
    double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int c = 0; c < n; ++c) acc[c & 7] += src[c * stride];
    return (float)(((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7])));
}

// src[0] + src[stride] + ... (n terms). FP64 is slow on this GPU (a convert and an add per
// term made the kernel 91 us of a 16 x 256 x 256 step), so the sum is compensated FP32:
// every add's exact rounding error (Knuth's TwoSum) goes into a second float, and the
// pair rounds to the result. Term c goes into sum c mod 4, the four are combined pairwise
// at the end; 32 loads are in flight. An infinite or NaN term, and a running sum that
// overflows, leave no finite pair: then the sum is taken in FP64, which has the range.
FR_HD float sum_terms(const float* src, size_t stride, int n)
{
    constexpr int kLoads = 32;
    float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < n; c += kLoads)
    {
        float v[kLoads];
#pragma unroll
        for (int j = 0; j < kLoads; ++j) v[j] = c + j < n ? src[(c + j) * stride] : 0.f;
#pragma unroll
        for (int j = 0; j < kLoads; ++j) two_sum_add(hi[j & 3], lo[j & 3], v[j]);  // adding 0 is exact
    }
#pragma unroll
    for (int j = 2; j > 0; j >>= 1)
#pragma unroll
        for (int k = 0; k < j; ++k)
        {
            two_sum_add(hi[k], lo[k], hi[k + j]);
            two_sum_add(hi[k], lo[k], lo[k + j]);
        }
    const float total = hi[0] + lo[0];
    return total - total == 0.f ? total : sum_fp64(src, stride, n);  // 0 only where it is finite
}

}  // namespace frx
