// compensated.cuh — sums to twice the float precision without the FP64 pipe.
// The operations are spelled as intrinsics, so that they round one by one
// whatever the file's contraction setting is.
#pragma once

#include <cstdint>

namespace facetcu {

// Compensated FP32 sum of count x B terms: each product split exactly into
// p + e (TwoProduct with an explicit fmaf) and each addition into s + err
// (Neumaier's TwoSum); the errors accumulate in c.  sum + c then carries
// about twice the float precision, as close to the reference's FP64 sum as
// its conversion back to float can tell, at FP32 throughput (GB300's FP64
// rate is a small fraction of it).
struct Csum {
    float s, c;
};
__device__ __forceinline__ void csum_add(Csum& a, float t, float e)
{
    const float s = __fadd_rn(a.s, t);
    const float err = fabsf(a.s) >= fabsf(t) ? __fadd_rn(__fsub_rn(a.s, s), t)
                                             : __fadd_rn(__fsub_rn(t, s), a.s);
    a.s = s;
    a.c = __fadd_rn(a.c, __fadd_rn(err, e));
}
__device__ __forceinline__ void csum_term(Csum& a, uint32_t count, float v)
{
    const float n = float(count);  // exact below 2^24
    const float p = __fmul_rn(n, v);
    csum_add(a, p, fmaf(n, v, -p));
}
__device__ __forceinline__ double csum_value(const Csum& a) { return double(a.s) + double(a.c); }

// (skyc L + sum) / d to twice the float precision, which rounds to the float
// that the double division gives but for halfway cases.  In doubles it is some
// twenty instructions of a pipe that was 83 % busy with nothing else: 43 us for
// one column of 400,000 sides, 7 so.  (Its error and that of the doubles, each
// against long double, are both below 0.5000005 units of the last place from 1e-37
// to 1e36: tests/cpp/mean_check.cpp.)
__device__ __forceinline__ float diffuse_mean(Csum a, uint32_t skyc, float L, uint32_t d)
{
    // counts that floats don't hold, products that overflow them or whose errors
    // they don't hold
    const float most = fmaxf(fabsf(a.s), fabsf(float(skyc) * L));
    if (max(d, skyc) >= 1u << 24 || !(most < 1.0e37f) || (most < 1.0e-30f && most != 0.0f))
        return float((double(skyc) * double(L) + csum_value(a)) / double(d));
    csum_term(a, skyc, L);
    const float hi = __fadd_rn(a.s, a.c), lo = __fsub_rn(a.c, __fsub_rn(hi, a.s)), n = float(d);
    const float q = __fdiv_rn(hi, n);
    return __fadd_rn(q, __fdiv_rn(__fadd_rn(fmaf(-q, n, hi), lo), n));
}

}  // namespace facetcu
