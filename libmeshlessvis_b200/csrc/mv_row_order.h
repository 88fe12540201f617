// The order in which the folded table sums (mv_sum.cu) take a lattice's rows.
// Plain C++ beside the device code, so that the host can check it.
#pragma once
#include <cmath>

#ifndef MV_HD
#ifdef __CUDACC__
#define MV_HD __host__ __device__ __forceinline__
#else
#define MV_HD inline
#endif
#endif

namespace mv {

// Whether a sum of n particles is worth the order.  `cells`: the cells of Phi^'s
// table that one step of k spans at the largest radius (negative: not known).
// Sorted rows save bank conflicts, a part of a particle's time that grows with
// the cells between the lanes' rows, and the order costs 2 to 6 us, so small sums
// and those of few cells lose by it.  us a group of 8, rows as they lie and
// sorted:
//   cells      1.2                  5.8                  23
//   62         34.3  40.6           34.3  42.0           38.4  42.6   100 x 90 x 70
//   250        73.4  80.5           77.4  81.5           86.7  81.6
//   2000       186   194            191   195            229   196
//   4000       349   358            359   358            429   362
//   250        71.3  75.5           75.5  76.1           84.7  77.5   92 x 76 x 58
//   2000       122   127            131   127            151   128
// The line, n cells^2 = 45,000, is within 3% of the better one in all of these.
constexpr double kRowOrderWorth = 45000.0;

MV_HD bool rows_worth_sorting(long long n, double cells) {
    return cells < 0.0 || (double)n * cells * cells >= kRowOrderWorth;
}

// The rows (yp, z) of a folded lattice sorted by their distance from the x
// axis (ties by yp, then z): a row's place is the number of rows before it,
// found for each yp by bisection over z >= 0, along which the distance grows.
struct RowOrder {
    int* rows;       // [yrows * nz], null: none wanted
    int yrows, nz, z0;
    double ky, kz;
    int first_block;
};

// The squared distance.  The places are a permutation only if a row's distance
// has one value wherever it is computed, and ry * ry + rz * rz has not: the
// compiler may contract either product into a fused multiply-add, and in a
// loop it takes another one than outside of it (steps such as 0.1 then leave
// some of the list unwritten).  So the fused operation is spelled out: the
// product rz * rz is its addend, rounded, and monotone in z.
MV_HD double row_key(const RowOrder& o, int y, int z) {
    const double ry = o.ky * y, rz = o.kz * (o.z0 + z);
    return fma(ry, ry, rz * rz);
}

// How many rows of yp = first, first + stride, ... come before row (y, z).
MV_HD int rows_before(const RowOrder& o, int y, int z, int first, int stride) {
    const double key = row_key(o, y, z);
    int place = 0;
    for (int yy = first; yy < o.yrows; yy += stride) {
        int lo = 0, hi = o.nz;  // z' < lo: before the row, z' >= hi: not
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const double k = row_key(o, yy, mid);
            const bool before = k < key || (k == key && (yy < y || (yy == y && mid < z)));
            if (before) lo = mid + 1;
            else hi = mid;
        }
        place += lo;
    }
    return place;
}

}  // namespace mv
