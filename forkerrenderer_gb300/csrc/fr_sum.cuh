// Sums of a gradient's partial sums (k_grad_reduce). The host test compiles the same code.
#pragma once

#include <stddef.h>

#include "fr_exact.cuh"

namespace frx
{

// A running sum as three floats: hi the rounded sum, mid the rounded sum of its adds'
// exact rounding errors (Knuth's TwoSum), lo the sum of mid's.
struct Sum3
{
    float hi, mid, lo;
};

// a = RN(a + x); the rounding error, exactly.
FR_HD float two_sum(float& a, float x)
{
    const float s = a + x;
    const float b = s - a;
    const float e = (a - (s - b)) + (x - b);
    a = s;
    return e;
}

FR_HD void add(Sum3& t, float x) { t.lo += two_sum(t.mid, two_sum(t.hi, x)); }

// The sum in FP64 (term c into sum c mod 8), for what the FP32 form cannot hold.
FR_HD float sum_fp64(const float* src, size_t stride, int n)
{
    double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int c = 0; c < n; c += 8)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += c + j < n ? src[(c + j) * stride] : 0.f;
    return (float)(((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7])));
}

// src[0] + src[stride] + ... (n terms, at most 152: a chain per SM), rounded once. FP64 is
// slow on this GPU (a convert and an add per term made the kernel 91 us of a 16 x 256 x 256
// step), so the sum is compensated FP32: 19 us, 16 with a pair of floats. Term c goes into
// sum c mod 4, the four are combined pairwise; the loads of 32 terms are independent.
// With u = 2^-24 and m terms in a sum (m <= 38): an add to hi rounds by at most
// u sum|x|, one to mid by at most u (m u sum|x|), and only those to lo are lost, each at
// most u (m^2 u^2 sum|x|): m^3 u^3 sum|x| < 2^-56 sum|x| in all, and less than 2^-54 with
// the combining. FP64 sums of every eighth term, combined pairwise, may lose 22 2^-53. (A
// pair of floats, without lo, loses up to 2^-37.6 sum|x|: where the terms cancel, bits of
// the result.) An infinite or NaN term, and a running sum that overflows, leave no finite
// sum: then it is taken in FP64, which has the range.
FR_HD float sum_terms(const float* src, size_t stride, int n)
{
    constexpr int kLoads = 32;
    Sum3 t[4] = {};
    for (int c = 0; c < n; c += kLoads)
    {
        float v[kLoads];
#pragma unroll
        for (int j = 0; j < kLoads; ++j) v[j] = c + j < n ? src[(c + j) * stride] : 0.f;
#pragma unroll
        for (int j = 0; j < kLoads; ++j) add(t[j & 3], v[j]);  // adding 0 is exact
    }
#pragma unroll
    for (int j = 2; j > 0; j >>= 1)
#pragma unroll
        for (int k = 0; k < j; ++k)
        {
            add(t[k], t[k + j].hi);
            add(t[k], t[k + j].mid);
            add(t[k], t[k + j].lo);
        }
    const float total = (float)((double)t[0].hi + ((double)t[0].mid + (double)t[0].lo));
    return total - total == 0.f ? total : sum_fp64(src, stride, n);  // 0 only where it is finite
}

}  // namespace frx
