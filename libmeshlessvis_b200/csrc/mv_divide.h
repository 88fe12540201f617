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
// (Markstein's division step), which gives the rounded quotient.  c and r have to
// be normal numbers, the quotient finite and the remainder exact: x = 0 or |x| and
// |x / c| at least 2^-80 (from 2^-108 down it may lie between the least subnormal
// numbers, and the quotient be another).
MV_HD float divide_finite(float x, float c, float r) {
    const float q = x * r;
    return fmaf(fmaf(-q, c, x), r, q);
}

// The same of any x; infinities and NaNs as x r has them.
MV_HD float divide_by(float x, float c, float r) {
    const float q = divide_finite(x, c, r);
    return fabsf(q) <= FLT_MAX ? q : x * r;
}

// From which x on divide_by(x, c, 1 / c) holds, 0 < c < 1e30, and for its
// quotient as x again, c then from 2^-20 to 1.
MV_HD float divide_by_least(float c) { return fmaxf(0x1p-80f, c * 0x1p-79f); }

}  // namespace mv
