// Division by a number that many divisions share.  Plain C++ beside the device
// code, so that the host can check it.
#pragma once
#include <cfloat>
#include <cmath>

#ifndef MV_HD
#ifdef __CUDACC__
#define MV_HD __host__ __device__ __forceinline__
#else
#define MV_HD inline
#endif
#endif

namespace mv {

// x / c where r = 1 / c, correctly rounded: x r, corrected by its remainder
// (Markstein's division step), which gives the rounded quotient; infinities and
// NaNs as x r has them.  c and r have to be normal numbers.  The remainder has
// to be exact: below 2^-80, where it may lie between the least subnormal
// numbers (x from 2^-108 down at c = 1e-29 gave other quotients), and for
// quotients that small, the division itself.
MV_HD float divide_by(float x, float c, float r) {
    const float q = x * r;
    if (fminf(fabsf(x), fabsf(q)) < 0x1p-80f && x != 0.f) return x / c;
    const float q1 = fmaf(fmaf(-q, c, x), r, q);
    return fabsf(q1) <= FLT_MAX ? q1 : q;
}

}  // namespace mv
