// Direct slice sum of one group (vis_fourier_volume_rendering: the reference's
// sample_fourier_transform_over_grid on its 2D lattice, meshless_vis/
// fourier_transform.cu:67-141, with reduce_partial_sums, arrange_samples and the
// cudaMemset before them, meshless_vis.cu:301-338, in one finalize).
//
// The lattice is x in (-cx, cx), y in [0, cy).  As in the folded plain form
// (mv_sum.cu) a representative x >= 0 gives both signs of x: with c = e^{i x Qx}
// and d = w e^{i y Qy} the sums
//   A0 = sum cr dr, A1 = sum ci di, A2 = sum cr di, A3 = sum ci dr
// give T(+x) = (A0 - A1, A2 + A3) and T(-x) = (A0 + A1, A2 - A3).  Positions are
// 32-bit fixed-point turns, phases exact wrapping integers.
//
// Two kernels:
//   slice_gemm_kernel   groups whose amplitude separates over x and y (no
//       radii, one radius for all particles, Gaussians): the four sums are a
//       real matrix product over the particles, done as a register-tiled FP32
//       one;
//   slice_table_kernel  SPH and Wendland with varying radii on square slices
//       (cx = cy, one step): |k| is the same at (x, y) and (y, x), so one
//       table lookup of Phi^ serves four lattice points.
// Other slices (SPH or Wendland with varying radii, cx != cy or two steps) take
// the folded plain form.
//
// Both split the particles over blocks until the chip is full, down to 64 a block
// (the plain form's four tiles of 256 leave a small slice on a few SMs); a tile is
// summed in FP32 registers, tiles in FP64 running sums in global scratch (none
// for blocks of one tile), splits in FP64 by the finalize.
#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>

#include "mv_device.cuh"
#include "mv_internal.h"
#include "mv_split_rules.h"

namespace mv {
namespace {

constexpr int kThreads = 256;  // threads per block == particles per tile

struct SliceSumArgs {
    const float4* particles;
    const float* radii;
    int n;
    int chunk;     // particles per split (whole tiles if more than one)
    int cx, cy;    // representatives x < cx (cx > 0), y < cy
    double m[6];   // turns of a particle along x and y: rows of M
    float gamma;   // Gaussians: +-pi log2(e); the exponent is gamma h^2 |k|^2
    float kx2, ky2;  // step.x^2, step.y^2
    double step;   // table: the step (|k| = step sqrt(x^2 + y^2))
    const float4* table;  // cubic cells; cell table_n is all zero
    int table_n;
    float inv_ds;
    double2* sums;    // [split][values][blocks x threads] running sums
    float2* partial;  // [split][(x + cx - 1) cy + y]
    size_t plane;
};

// exp(2 pi i q / 2^32), correctly rounded but for the last bit: a chain's steps
// multiply its error.
__device__ __forceinline__ float2 unit_rotation(uint32_t q) {
    double sn, cs;
    sincospi((double)(int32_t)q * (1.0 / 2147483648.0), &sn, &cs);
    return make_float2((float)cs, (float)sn);
}

// Adds a tile's packed FP32 sums to the thread's running sums.
template <int COUNT>
__device__ __forceinline__ void add_tile(double2* sums, size_t stride, const float2* acc, bool first) {
#pragma unroll
    for (int i = 0; i < COUNT; ++i) {
        double2* p = sums + (size_t)i * stride;
        const double2 o = first ? make_double2(0.0, 0.0) : *p;
        *p = make_double2(o.x + (double)acc[i].x, o.y + (double)acc[i].y);
    }
}

// ------------------------------------------------------------ separable groups
// Block: 64 x 64 representatives (x, y), thread: 4 x 4 of them (16 x 16 threads,
// a warp's lanes along y).  Per stage of 32 particles the block computes the
// factors c gx of 64 x and d gy of 64 y in shared memory (8-step rotations from
// an exact start), and every thread adds 4 x 4 products of each particle: 32
// packed FMAs and 4 16-byte loads for 32 lattice points, where a thread of the
// folded plain form spends about 5 instructions a point (rotation, phases, one
// packed FMA).  Bound: the FP32 pipes (two FMAs a point).
constexpr int kTile = 64, kStage = 32;
constexpr int kFRow = kTile + 4;  // floats of a particle's 64 factors' re (or im), padded against bank conflicts
constexpr size_t kGemmSmem = (size_t)kStage * 4 * kFRow * sizeof(float);
static_assert(kGemmSmem + kThreads * (sizeof(uint4) + sizeof(float4)) <= 48 << 10, "within what a launch may take");

template <bool GAUSS>
__global__ void __launch_bounds__(kThreads, 2) slice_gemm_kernel(SliceSumArgs a) {
    extern __shared__ float4 s_dyn[];
    float* s_f = reinterpret_cast<float*>(s_dyn);  // x factors' re and im, y factors' re and im: [kStage][kFRow] each
    __shared__ uint4 s_q[kThreads];    // Qx, Qy, w, gamma h^2
    __shared__ float4 s_rot[kThreads];  // the unit rotations of Qx and Qy
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int x_tiles = (a.cx + kTile - 1) / kTile;
    const int xt = (int)(blockIdx.x % x_tiles) * kTile, yt = (int)(blockIdx.x / x_tiles) * kTile;
    const int tx = tid >> 4, ty = tid & 15;
    const int beg = blockIdx.y * a.chunk, end = min(a.n, beg + a.chunk);
    const size_t stride = (size_t)gridDim.x * kThreads;
    double2* sums = a.sums + (size_t)blockIdx.y * 32 * stride + (size_t)blockIdx.x * kThreads + tid;

    // [x][y pair][A0 .. A3], packed over the pair's two y
    float2 acc[32];  // [(x * 2 + pair) * 4 + kind]
    auto clear = [&]() {
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] = make_float2(0.f, 0.f);
    };
    clear();
    for (int t0 = beg; t0 < end; t0 += kThreads) {
        __syncthreads();
        {
            const int idx = t0 + tid;
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
            float g = 0.f;
            if (idx < end) {
                p = a.particles[idx];
                if constexpr (GAUSS) {
                    const float h = a.radii[idx];
                    g = a.gamma * h * h;
                }
            }
            const double px = p.x, py = p.y, pz = p.z;
            const uint32_t qx = fixed_turns(a.m[0] * px + a.m[1] * py + a.m[2] * pz);
            const uint32_t qy = fixed_turns(a.m[3] * px + a.m[4] * py + a.m[5] * pz);
            s_q[tid] = make_uint4(qx, qy, __float_as_uint(p.w), __float_as_uint(g));
            const float2 rx = unit_rotation(qx), ry = unit_rotation(qy);
            s_rot[tid] = make_float4(rx.x, rx.y, ry.x, ry.y);
        }
        const int count = min(kThreads, end - t0);
        for (int s0 = 0; s0 < count; s0 += kStage) {
            __syncthreads();
            // the stage's factors: lane = particle, warp = 8 of the 64 x and y
            // (particles past the end have weight 0)
            const uint4 q = s_q[s0 + lane];
            const float4 R = s_rot[s0 + lane];
            const float gam = __uint_as_float(q.w);
#pragma unroll 1
            for (int axis = 0; axis < 2; ++axis) {  // a loop, four factors at a time: the sums stay in registers
                const int f0 = (axis ? yt : xt) + warp * 8;
                const float k2 = axis ? a.ky2 : a.kx2;
                const float rx = axis ? R.z : R.x, ry = axis ? R.w : R.y;
                float im, re;
                __sincosf(turns_to_radians((uint32_t)f0 * (axis ? q.y : q.x)), &im, &re);
                const float w = axis ? __uint_as_float(q.z) : 1.f;
                re *= w;
                im *= w;
#pragma unroll 1
                for (int i0 = 0; i0 < 8; i0 += 4) {
                    float vr[4], vi[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int f = f0 + i0 + i;
                        float g = 1.f;
                        if constexpr (GAUSS) g = exp2f(gam * (k2 * (float)(f * f)));
                        vr[i] = GAUSS ? g * re : re;
                        vi[i] = GAUSS ? g * im : im;
                        const float nr = fmaf(re, rx, -im * ry);
                        im = fmaf(re, ry, im * rx);
                        re = nr;
                    }
                    float* at = s_f + (axis * 2 * kStage + lane) * kFRow + warp * 8 + i0;
                    *reinterpret_cast<float4*>(at) = make_float4(vr[0], vr[1], vr[2], vr[3]);
                    *reinterpret_cast<float4*>(at + kStage * kFRow) = make_float4(vi[0], vi[1], vi[2], vi[3]);
                }
            }
            __syncthreads();
#pragma unroll 2
            for (int j = 0; j < kStage; ++j) {
                const float* at = s_f + j * kFRow;
                const float4 xr = *reinterpret_cast<const float4*>(at + tx * 4);
                const float4 xi = *reinterpret_cast<const float4*>(at + kStage * kFRow + tx * 4);
                const float4 dr = *reinterpret_cast<const float4*>(at + 2 * kStage * kFRow + ty * 4);
                const float4 di = *reinterpret_cast<const float4*>(at + 3 * kStage * kFRow + ty * 4);
                const float2 r[2] = {make_float2(dr.x, dr.y), make_float2(dr.z, dr.w)};
                const float2 m[2] = {make_float2(di.x, di.y), make_float2(di.z, di.w)};
                const float re[4] = {xr.x, xr.y, xr.z, xr.w}, im[4] = {xi.x, xi.y, xi.z, xi.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 cr = make_float2(re[i], re[i]), ci = make_float2(im[i], im[i]);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        acc[(i * 2 + k) * 4 + 0] = __ffma2_rn(cr, r[k], acc[(i * 2 + k) * 4 + 0]);
                        acc[(i * 2 + k) * 4 + 1] = __ffma2_rn(ci, m[k], acc[(i * 2 + k) * 4 + 1]);
                        acc[(i * 2 + k) * 4 + 2] = __ffma2_rn(cr, m[k], acc[(i * 2 + k) * 4 + 2]);
                        acc[(i * 2 + k) * 4 + 3] = __ffma2_rn(ci, r[k], acc[(i * 2 + k) * 4 + 3]);
                    }
                }
            }
        }
        if (a.chunk > kThreads) {
            add_tile<32>(sums, stride, acc, t0 == beg);
            clear();
        }
    }
    float2* out = a.partial + blockIdx.y * a.plane;
    const bool scratch = a.chunk > kThreads && beg < end;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int x = xt + tx * 4 + i;
        if (x >= a.cx) continue;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            double2 A[4];
#pragma unroll
            for (int v = 0; v < 4; ++v)
                A[v] = scratch ? sums[(size_t)((i * 2 + k) * 4 + v) * stride]
                               : make_double2(acc[(i * 2 + k) * 4 + v].x, acc[(i * 2 + k) * 4 + v].y);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int y = yt + ty * 4 + 2 * k + e;
                if (y >= a.cy) continue;
                const double a0 = e ? A[0].y : A[0].x, a1 = e ? A[1].y : A[1].x;
                const double a2 = e ? A[2].y : A[2].x, a3 = e ? A[3].y : A[3].x;
                out[(size_t)(a.cx - 1 + x) * a.cy + y] = make_float2((float)(a0 - a1), (float)(a2 + a3));
                if (x > 0) out[(size_t)(a.cx - 1 - x) * a.cy + y] = make_float2((float)(a0 + a1), (float)(a2 - a3));
            }
        }
    }
}

// ------------------------------------------- SPH, Wendland with varying radii
// Square slices.  A thread owns kL x values from kL g and a row y of the triangle
// x >= y, and sums the points (+-x, y) and (+-y, x) together: a table lookup
// (one 16-byte shared-memory read) serves four points, where the folded form's
// serves two.  Lanes run along y (neighbours in |k|, whose lookups often share a
// cell; along x a lookup took 12 shared-memory cycles).  Per stage of 32
// particles a warp computes, a lane a particle, the factors of every other x
// value of its chunks -- c = e^{i x Qx} for the first pair of points, d' = w e^{i
// x Qy} for the second -- and keeps them packed in shared memory; the loop over
// particles rotates them once, and takes the next particle's sines at y while it
// sums one.  No one pipe binds it: shared memory, the packed operations' FMA
// pipe and issue are each about half busy.  Indices past the table and of
// negative radii read its last, all-zero cell (a NaN radius reads it too, but its
// offset in the cell is a NaN, and so are its terms); a tile whose radii all lie
// in the table's range (a group's usually do: the table reaches its largest
// radius) uses the index as it is.
constexpr int kL = 4;
constexpr int kTableResident = 24;  // warps an SM, of 80 registers
constexpr int kXRow = kL / 2;      // float4 of a particle's x factors
constexpr int kSpan = 4;           // chunks a warp's 32 rows lie in at most (4 + 8 + 12 rows, then more)

// Threads of the triangle: chunk g has rows y < kL (g + 1).
__host__ __device__ inline int triangle_threads(int c) {
    const int g = (c + kL - 1) / kL;
    return kL * g * (g + 1) / 2;
}

// Shared memory of a block of `warps` warps beside the table, with the 1 KB the
// system keeps.
constexpr int table_block_smem(int warps) { return 8192 + warps * kSpan * 32 * kXRow * 16 + 1024; }

template <int kTableWarps>
__global__ void __launch_bounds__(32 * kTableWarps, kTableResident / kTableWarps) slice_table_kernel(SliceSumArgs a) {
    constexpr int kTableThreads = 32 * kTableWarps;
    extern __shared__ float4 s_tab[];  // table cells
    __shared__ uint4 s_q[kThreads];    // Qx, Qy, w, h / ds
    __shared__ float4 s_rot[kThreads];  // the unit rotations of Qx and Qy: their re, their im
    __shared__ float4 s_x[kTableWarps][kSpan][32 * kXRow];  // (c re, d' re, c im, d' im)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i <= a.table_n; i += kTableThreads) s_tab[i] = a.table[i];

    const int c = a.cx;
    // thread t: chunk g begins at thread kL g (g + 1) / 2; the last one's rows
    // are repeated past the end
    const int threads = triangle_threads(c);
    const int t = min((int)blockIdx.x * kTableThreads + tid, threads - 1);
    const bool active = (int)blockIdx.x * kTableThreads + tid < threads;
    int g = (int)((sqrtf(1.f + 8.f / kL * (float)t) - 1.f) * 0.5f);
    while (kL * g * (g + 1) / 2 > t) --g;
    while (kL * (g + 1) * (g + 2) / 2 <= t) ++g;
    const int x0 = kL * g, y = t - kL * g * (g + 1) / 2;
    const int g0 = __shfl_sync(0xffffffffu, g, 0), spans = __shfl_sync(0xffffffffu, g, 31) - g0 + 1;
    float r[kL];  // |k| (0 off the triangle, which stays in the table)
#pragma unroll
    for (int m = 0; m < kL; ++m)
        r[m] = x0 + m < c && y <= x0 + m ? (float)(a.step * sqrt((double)(x0 + m) * (x0 + m) + (double)y * y)) : 0.f;
    const float r_most = (float)(a.step * sqrt(2.0) * (c - 1)) * 1.000001f;

    const int beg = blockIdx.y * a.chunk, end = min(a.n, beg + a.chunk);
    const size_t stride = (size_t)gridDim.x * kTableThreads;
    double2* sums = a.sums + (size_t)blockIdx.y * 4 * kL * stride + (size_t)blockIdx.x * kTableThreads + tid;
    const uint32_t uy = (uint32_t)y;
    // byte address of cell 0, less the bits of the rounding constant
    const uint32_t tab = (uint32_t)__cvta_generic_to_shared(s_tab) - (0x4B400000u << 4);

    // (A0, A0'), (A1, A1'), (A2, A3'), (A3, A2'): unprimed at (x, y), primed at (y, x)
    float2 acc[4 * kL];
    auto clear = [&]() {
#pragma unroll
        for (int i = 0; i < 4 * kL; ++i) acc[i] = make_float2(0.f, 0.f);
    };
    clear();
    // a particle's factors at y: d for (x, y), c' for (y, x), packed
    struct AtY {
        float2 D1, D2;
        float h;
    };
    auto at_y = [&](int j) {
        const uint4 q = s_q[j];
        const float w = __uint_as_float(q.z);
        float sn, cs, s2, c2;
        __sincosf(turns_to_radians(uy * q.y), &sn, &cs);
        __sincosf(turns_to_radians(uy * q.x), &s2, &c2);
        AtY d;
        d.D1 = make_float2(w * cs, c2);
        d.D2 = make_float2(w * sn, s2);
        d.h = __uint_as_float(q.w);
        return d;
    };
    auto add_particle = [&](int j, const float4* xf, const AtY& d, auto clamp) {
        const float2 D1 = d.D1, D2 = d.D2;
        const float h = d.h;
        const float4 R = s_rot[j];  // (Re Rx, Re Ry, Im Rx, Im Ry)
        float2 X, Y;
#pragma unroll
        for (int m = 0; m < kL; ++m) {
            if (m % 2 == 0) {
                const float4 v = xf[m / 2];
                X = make_float2(v.x, v.y);
                Y = make_float2(v.z, v.w);
            } else {
                const float2 RX = make_float2(R.x, R.y), RY = make_float2(R.z, R.w);
                const float2 nx = __ffma2_rn(X, RX, __fmul2_rn(make_float2(-Y.x, -Y.y), RY));
                Y = __ffma2_rn(X, RY, __fmul2_rn(Y, RX));
                X = nx;
            }
            // |k| h / ds: nearest cell and offset (1.5 * 2^23 rounds)
            const float tt = fmaf(r[m], h, 12582912.0f);
            const float fr = fmaf(r[m], h, -(tt - 12582912.0f));
            float4 t;
            if constexpr (decltype(clamp)::value) {
                t = s_tab[min((unsigned)(__float_as_int(tt) - 0x4B400000), (unsigned)a.table_n)];
            } else {
                const uint32_t at = ((uint32_t)__float_as_int(tt) << 4) + tab;
                asm("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                    : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w)
                    : "r"(at));
            }
            const float amp = fmaf(fmaf(fmaf(t.w, fr, t.z), fr, t.y), fr, t.x);
            const float2 amp2 = make_float2(amp, amp);
            const float2 UX = __fmul2_rn(X, amp2), UY = __fmul2_rn(Y, amp2);
            acc[4 * m + 0] = __ffma2_rn(UX, D1, acc[4 * m + 0]);
            acc[4 * m + 1] = __ffma2_rn(UY, D2, acc[4 * m + 1]);
            acc[4 * m + 2] = __ffma2_rn(UX, D2, acc[4 * m + 2]);
            acc[4 * m + 3] = __ffma2_rn(UY, D1, acc[4 * m + 3]);
        }
    };
    for (int t0 = beg; t0 < end; t0 += kThreads) {
        __syncthreads();
        int outside = 0;
#pragma unroll 1
        for (int l = tid; l < kThreads; l += kTableThreads) {
            const int idx = t0 + l;
            if (idx >= end) break;
            const float4 p = a.particles[idx];
            const double px = p.x, py = p.y, pz = p.z;
            const uint32_t qx = fixed_turns(a.m[0] * px + a.m[1] * py + a.m[2] * pz);
            const uint32_t qy = fixed_turns(a.m[3] * px + a.m[4] * py + a.m[5] * pz);
            const float h = a.radii[idx] * a.inv_ds;
            outside |= !(h >= 0.f && h * r_most <= (float)(a.table_n - 1));
            s_q[l] = make_uint4(qx, qy, __float_as_uint(p.w), __float_as_uint(h));
            const float2 rx = unit_rotation(qx), ry = unit_rotation(qy);
            s_rot[l] = make_float4(rx.x, ry.x, rx.y, ry.y);
        }
        const bool clamp = __syncthreads_or(outside) != 0;
        const int count = min(kThreads, end - t0);
#pragma unroll 1
        for (int s0 = 0; s0 < count; s0 += 32) {
            const int in = min(32, count - s0);
            __syncwarp();  // the stage before has been read
            if (lane < in) {
                const uint4 q = s_q[s0 + lane];
                const float4 R = s_rot[s0 + lane];
                const float w = __uint_as_float(q.z);
                // two steps of x at once: the squared rotations
                const float2 Rx = make_float2(fmaf(R.x, R.x, -R.z * R.z), 2.f * R.x * R.z);
                const float2 Ry = make_float2(fmaf(R.y, R.y, -R.w * R.w), 2.f * R.y * R.w);
#pragma unroll 1
                for (int sp = 0; sp < spans; ++sp) {
                    float cr, ci, er, ei;
                    const uint32_t ux = (uint32_t)(kL * (g0 + sp));
                    __sincosf(turns_to_radians(ux * q.x), &ci, &cr);
                    __sincosf(turns_to_radians(ux * q.y), &ei, &er);
                    er *= w;
                    ei *= w;
                    float4* xf = &s_x[warp][sp][lane * kXRow];
#pragma unroll
                    for (int m = 0; m < kL / 2; ++m) {
                        xf[m] = make_float4(cr, er, ci, ei);
                        const float nc = fmaf(cr, Rx.x, -ci * Rx.y), ne = fmaf(er, Ry.x, -ei * Ry.y);
                        ci = fmaf(cr, Rx.y, ci * Rx.x);
                        ei = fmaf(er, Ry.y, ei * Ry.x);
                        cr = nc;
                        er = ne;
                    }
                }
            }
            __syncwarp();
            const float4* xf = s_x[warp][g - g0];
            if (clamp) {
#pragma unroll 1
                for (int j = 0; j < in; ++j) add_particle(s0 + j, xf + j * kXRow, at_y(s0 + j), std::true_type{});
            } else {
                // the next particle's sines are taken while this one is summed
                AtY d = at_y(s0);
#pragma unroll 1
                for (int j = 0; j < in; ++j) {
                    const AtY next = at_y(min(s0 + j + 1, s0 + in - 1));
                    add_particle(s0 + j, xf + j * kXRow, d, std::false_type{});
                    d = next;
                }
            }
        }
        if (a.chunk > kThreads) {
            add_tile<4 * kL>(sums, stride, acc, t0 == beg);
            clear();
        }
    }
    if (!active) return;
    float2* out = a.partial + blockIdx.y * a.plane;
    const bool scratch = a.chunk > kThreads && beg < end;
#pragma unroll
    for (int m = 0; m < kL; ++m) {
        const int x = x0 + m;
        if (x >= c || x < y) continue;  // (y, x) has the points with x < y
        double2 A[4];
#pragma unroll
        for (int v = 0; v < 4; ++v)
            A[v] = scratch ? sums[(size_t)(m * 4 + v) * stride] : make_double2(acc[4 * m + v].x, acc[4 * m + v].y);
        auto put = [&](int px, int py, double re, double im) {
            out[(size_t)(c - 1 + px) * c + py] = make_float2((float)re, (float)im);
        };
        put(x, y, A[0].x - A[1].x, A[2].x + A[3].x);
        if (x > 0) put(-x, y, A[0].x + A[1].x, A[2].x - A[3].x);
        if (x != y) {
            put(y, x, A[0].y - A[1].y, A[3].y + A[2].y);
            if (y > 0) put(-y, x, A[0].y + A[1].y, A[3].y - A[2].y);
        }
    }
}

struct SliceFinalizeArgs {
    const float2* partial;
    int splits;
    size_t plane;
    int cx, cy, nx, row;  // row = ny / 2 + 1
    double kx, ky;
    int basis;
    int factored;   // times Phi^(|k| h)
    double h, scale;
    float2* out;
    int accumulate;
};

// One warp row of 32 elements x 16 warps: warp w sums splits w, w + 16, ... in
// FP64, warp 0 adds the sixteen sums in order, applies the factored Phi^ and the
// scale, conjugates (the kernels summed w e^{+i theta}) and writes the C2R
// layout: every element of it, the ones that are no slice sample as zeros (the
// reference's memset), unless the group is added to earlier ones.
constexpr int kFinalWarps = 16;
__global__ void __launch_bounds__(32 * kFinalWarps) slice_finalize_kernel(SliceFinalizeArgs f) {
    __shared__ double2 s_part[kFinalWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long e = (long long)blockIdx.x * 32 + lane;
    const bool inside = e < (long long)f.nx * f.row;
    const int ix = inside ? (int)(e / f.row) : 0, y = inside ? (int)(e % f.row) : 0;
    const int x = ix < f.cx ? ix : ix - f.nx;
    const bool sample = inside && y < f.cy && (ix < f.cx || ix > f.nx - f.cx);
    double sr = 0.0, si = 0.0;
    if (sample) {
        const float2* p = f.partial + (size_t)(x + f.cx - 1) * f.cy + y;
#pragma unroll 8
        for (int s = warp; s < f.splits; s += kFinalWarps) {
            const float2 v = p[(size_t)s * f.plane];
            sr += v.x;
            si += v.y;
        }
    }
    s_part[warp][lane] = make_double2(sr, si);
    __syncthreads();
    if (warp != 0 || !inside) return;
    if (!sample) {
        if (!f.accumulate) f.out[e] = make_float2(0.f, 0.f);
        return;
    }
#pragma unroll
    for (int w = 1; w < kFinalWarps; ++w) {
        sr += s_part[w][lane].x;
        si += s_part[w][lane].y;
    }
    double factor = f.scale;
    if (f.factored) {
        const double rx = f.kx * x, ry = f.ky * y;
        factor *= phi_fp64(f.basis, sqrt(rx * rx + ry * ry) * f.h);
    }
    const float re = (float)(sr * factor), im = (float)(-si * factor);
    if (f.accumulate) {
        const float2 o = f.out[e];
        f.out[e] = make_float2(o.x + re, o.y + im);
    } else {
        f.out[e] = make_float2(re, im);
    }
}

}  // namespace

int launch_slice_sum(const SumRequest& req, int nx, int ny, Workspace& ws, KernelTimer* timer) {
    const Lattice& lat = req.lat;
    const int row = ny / 2 + 1;
    if (req.basis < 0 || req.basis >= kBasisCount) return set_error(kInvalidValue, "unknown basis function id");
    if (req.n < 0) return set_error(kInvalidValue, "negative number of terms");
    if (req.n > 0 && req.particles == nullptr) return set_error(kInvalidValue, "dataset group has no device particles");
    const bool known = req.radii && req.radius_min >= 0.f && std::isfinite(req.radius_max);
    // one radius for all: a NaN among equal radii makes its particle's terms NaNs
    const bool uniform = known && !req.radius_nan && req.radius_min == req.radius_max;
    const bool factored = !req.radii || uniform;
    const bool gauss = !factored && known && (req.basis == kGaussian || req.basis == kGaussianDecaying);
    const bool table = !factored && (req.basis == kSph || req.basis == kWendland) && lat.kx == lat.ky &&
                       lat.kx > 0 && lat.nx == 2 * lat.ny - 1;
    if (lat.nx <= 0 || lat.ny <= 0 || (req.n > 0 && !factored && !gauss && !table)) {
        if (!req.accumulate) {
            const int st = check_cuda(cudaMemsetAsync(req.out, 0, sizeof(float2) * (size_t)nx * row, req.stream),
                                      "cudaMemsetAsync");
            if (st != kOk) return st;
        }
        return lat.nx <= 0 || lat.ny <= 0 ? kOk : launch_plain_sum(req, ws, timer);
    }

    SliceSumArgs a{};
    a.particles = req.particles;
    a.radii = req.radii;
    a.n = req.n;
    a.cx = (lat.nx + 1) / 2;
    a.cy = lat.ny;
    for (int i = 0; i < 6; ++i) a.m[i] = lat.m[i];
    a.gamma = req.basis == kGaussian ? kPiLog2e : -kPiLog2e;
    a.kx2 = (float)(lat.kx * lat.kx);
    a.ky2 = (float)(lat.ky * lat.ky);
    a.step = lat.kx;
    a.plane = (size_t)lat.nx * lat.ny;

    int st = kOk;
    int splits = 0;
    if (req.n > 0) {
        const bool by_table = !factored && table;
        double ds = 0.0;
        int resident = 2;  // blocks an SM
        int threads = kThreads;
        long long blocks = (long long)((a.cx + kTile - 1) / kTile) * ((a.cy + kTile - 1) / kTile);
        if (by_table) {
            ds = phi_table_cell(req.basis);
            const double rmax = lat.kx * std::sqrt(2.0) * (lat.ny - 1);
            a.table_n = phi_table_cells(req.basis, req.radius_max >= 0.f ? rmax * req.radius_max : 1e30);
            a.inv_ds = (float)(1.0 / ds);
            // Warps a block: 4, or 3 where that leaves clearly fewer warps past
            // the triangle's end (17 warps of rows at a cutoff of 64 take 20 or
            // 18: 825 us and 758 with 245,066 particles) and the smaller
            // blocks, each with a table of its own, still fill an SM.  6 are
            // as fast there, and slower at some sizes of few splits (282 us
            // against 252 with 60,000 particles).
            const int warps = (triangle_threads(a.cx) + 31) / 32;
            double most = 0.0;
            for (int w : {4, 3}) {
                const int fit = std::max(1, std::min<int>(kTableResident / w,
                                                          (int)(227 * 1024 / (table_block_smem(w) + 16 * (size_t)(a.table_n + 1)))));
                const int count = (warps + w - 1) / w;
                const double on_an_sm = (double)fit * warps / count;
                if (on_an_sm > 1.05 * most) {
                    most = on_an_sm;
                    threads = 32 * w;
                    blocks = count;
                    resident = fit;
                }
            }
        }
        if (blocks > INT32_MAX) return set_error(kInvalidValue, "slice too large");
        const size_t partial_bytes = a.plane * sizeof(float2);  // of a split
        const size_t split_sums = (size_t)(by_table ? 4 * kL : 32) * (size_t)blocks * threads * sizeof(double2);
        a.chunk = slice_chunk(req.n, kThreads, blocks, partial_bytes, split_sums, resident, device_sm_count());
        splits = (int)(((long long)req.n + a.chunk - 1) / a.chunk);
        if (splits > 65535) return set_error(kInvalidValue, "slice sum: too many splits");
        const size_t part_bytes = (splits * partial_bytes + 255) / 256 * 256;
        const size_t table_bytes = by_table ? ((size_t)(a.table_n + 1) * sizeof(float4) + 255) / 256 * 256 : 0;
        const size_t sums_bytes = a.chunk > kThreads ? splits * split_sums : 0;
        st = ws.reserve(part_bytes + table_bytes + sums_bytes);
        if (st != kOk) return st;
        char* base = static_cast<char*>(ws.ptr);
        a.partial = reinterpret_cast<float2*>(base);
        a.sums = reinterpret_cast<double2*>(base + part_bytes + table_bytes);
        const dim3 grid((unsigned)blocks, (unsigned)splits);
        void (*kernel)(SliceSumArgs) = gauss ? slice_gemm_kernel<true> : slice_gemm_kernel<false>;
        size_t smem = kGemmSmem;
        if (by_table) {
            a.table = reinterpret_cast<const float4*>(base + part_bytes);
            launch_phi_table(req.basis, ds, a.table_n, reinterpret_cast<float4*>(base + part_bytes), req.stream);
            kernel = threads == 32 * 4 ? slice_table_kernel<4> : slice_table_kernel<3>;
            smem = (size_t)(a.table_n + 1) * sizeof(float4);
        }
        // beside the static shared memory (25 KB at most; the product kernel's
        // fits), over the 48 KB a launch may take by itself
        if (by_table && smem > 20 * 1024) {
            st = allow_table_memory(reinterpret_cast<const void*>(kernel));
            if (st != kOk) return st;
        }
        timer_begin(timer, 0, req.stream);
        kernel<<<grid, threads, smem, req.stream>>>(a);
        count_launch();
        timer_end(timer, 0, req.stream);
        st = check_cuda(cudaGetLastError(), "slice sum launch");
        if (st != kOk) return st;
    }

    SliceFinalizeArgs f{};
    f.partial = a.partial;
    f.splits = splits;
    f.plane = a.plane;
    f.cx = a.cx;
    f.cy = a.cy;
    f.nx = nx;
    f.row = row;
    f.kx = lat.kx;
    f.ky = lat.ky;
    f.basis = req.basis;
    f.factored = factored ? 1 : 0;
    f.h = uniform ? (double)req.radius_max : 1.0;
    f.scale = req.scale;
    f.out = req.out;
    f.accumulate = req.accumulate ? 1 : 0;
    const long long elements = (long long)nx * row;
    slice_finalize_kernel<<<(unsigned)((elements + 31) / 32), 32 * kFinalWarps, 0, req.stream>>>(f);
    count_launch();
    return check_cuda(cudaGetLastError(), "slice_finalize_kernel launch");
}

}  // namespace mv
