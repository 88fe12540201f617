// Fourier-slice extraction from the 3D half-spectrum into the 2D C2R layout,
// batched over views.  No reference twin: the reference recomputes the direct
// sum per view (meshless_vis/fourier_transform.cu:67-141); its arrange_samples
// (meshless_vis/meshless_vis.cu:318-332) and the cudaMemset before it (:338)
// are fused here: every element of [view][nx][ny/2+1] is written exactly once.
//
// Element (ix, y) of a view holds slice sample x = ix (ix < cx) or ix - nx
// (ix > nx - cx), y < cy; all other elements (including arrange_samples's
// dropped u-Nyquist x == cx) are zero.  The sample is the trilinear
// interpolation of the spectrum at p = (step.x x u + step.y y v) / step3,
// reflected to conj(F(-p)) when p_z < 0, corners outside the stored lattice
// reading zero, times step.x * step.y.
//
// Block: a tile of 32 x by 8 y samples of one view, a warp's lanes along x, two
// lanes a sample.  The loads are scattered (a sample's neighbours along y lie a
// whole row of l apart in the usual views), so the L1's lookups, one a cache
// line of a warp's load, bound the kernel, not bytes.  The two lanes of a sample
// take the corners at l and l + 1, which lie in one line as a rule; lanes along
// x touch fewer lines than along y (x runs partly along l, where values are
// contiguous), the tile's other rows reuse them from L1, and its samples leave
// through shared memory as 64-byte pieces of the y-fast layout.  360 views of
// 384 x 384 from 384^3: 412 us with a thread an element in output order, 390
// with lanes along x (88% of the L1's lookups), SLICE_TILE_US us so.
#include "mv_internal.h"

namespace mv {

namespace {

constexpr int kTileX = 32, kTileY = 8;

struct SliceAt {
    const float2* spectrum;
    int gx, gy, lz;
    float inv_step;
    float u0, u1, u2, v0, v1, v2, step_x, step_y;
};

// The slice sample (x, y): trilinear interpolation, the corners of l offset dl by
// this lane and the others by its neighbour (dl = 1 - dl), added up in both.
__device__ __forceinline__ float2 slice_sample(const SliceAt& s, int x, int y, int dl) {
    const float fu = s.step_x * (float)x, fv = s.step_y * (float)y;
    float p0 = (fu * s.u0 + fv * s.v0) * s.inv_step;
    float p1 = (fu * s.u1 + fv * s.v1) * s.inv_step;
    float p2 = (fu * s.u2 + fv * s.v2) * s.inv_step;
    const bool conj = p2 < 0.f;
    if (conj) {
        p0 = -p0;
        p1 = -p1;
        p2 = -p2;
    }
    const float f0 = floorf(p0), f1 = floorf(p1), f2 = floorf(p2);
    const float t0 = p0 - f0, t1 = p1 - f1, t2 = p2 - f2;
    const int ii = (int)f0 + (s.gx >> 1), jj = (int)f1 + (s.gy >> 1), ll = (int)f2 + dl;
    // corner (di, dj), zero outside the stored lattice; corners of weight 0
    // (half of them or more where an axis of the view runs along the lattice
    // in its steps) are not read
    const bool k = (unsigned)ll < (unsigned)s.lz && (dl == 0 || t2 > 0.f);
    const bool i0 = k && (unsigned)ii < (unsigned)s.gx, i1 = k && (unsigned)(ii + 1) < (unsigned)s.gx && t0 > 0.f;
    const bool j0 = (unsigned)jj < (unsigned)s.gy, j1 = (unsigned)(jj + 1) < (unsigned)s.gy && t1 > 0.f;
    const float2* at = s.spectrum + ((long long)ii * s.gy + jj) * s.lz + ll;
    const long long row = (long long)s.gy * s.lz;
    const float2 zero = make_float2(0.f, 0.f);
    const float2 c00 = i0 && j0 ? __ldg(at) : zero, c10 = i1 && j0 ? __ldg(at + row) : zero;
    const float2 c01 = i0 && j1 ? __ldg(at + s.lz) : zero, c11 = i1 && j1 ? __ldg(at + row + s.lz) : zero;
    const float wl = dl ? t2 : 1.f - t2;
    const float w00 = (1.f - t0) * (1.f - t1) * wl, w10 = t0 * (1.f - t1) * wl;
    const float w01 = (1.f - t0) * t1 * wl, w11 = t0 * t1 * wl;
    float re = fmaf(w11, c11.x, fmaf(w01, c01.x, fmaf(w10, c10.x, w00 * c00.x)));
    float im = fmaf(w11, c11.y, fmaf(w01, c01.y, fmaf(w10, c10.y, w00 * c00.y)));
    re += __shfl_xor_sync(0xffffffffu, re, 1);
    im += __shfl_xor_sync(0xffffffffu, im, 1);
    const float scale = s.step_x * s.step_y;
    return make_float2(re * scale, (conj ? -im : im) * scale);
}

// Tile `tile` of a view's [nx][ny / 2 + 1] elements.
__device__ __forceinline__ void slice_tile(const SliceAt& s, int tile, int cx, int cy, int nx, int ny,
                                           float2* __restrict__ out) {
    __shared__ float2 s_tile[kTileY][kTileX + 1];
    const int h = ny / 2 + 1, tiles_y = (h + kTileY - 1) / kTileY;
    const int x0 = tile / tiles_y * kTileX, y0 = tile % tiles_y * kTileY;
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int y_row = y0 + row;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int ix = x0 + 16 * half + (lane >> 1);
        const bool sample = ix < nx && y_row < cy && (ix < cx || ix > nx - cx);
        float2 v = make_float2(0.f, 0.f);
        if (__any_sync(0xffffffffu, sample)) {
            // lanes without a sample take the origin's along
            v = slice_sample(s, sample ? (ix < cx ? ix : ix - nx) : 0, sample ? y_row : 0, lane & 1);
            if (!sample) v = make_float2(0.f, 0.f);
        }
        if ((lane & 1) == 0) s_tile[row][16 * half + (lane >> 1)] = v;
    }
    __syncthreads();
    const int ix = x0 + (int)threadIdx.x / kTileY, y = y0 + (int)threadIdx.x % kTileY;
    if (ix < nx && y < h) out[(size_t)ix * h + y] = s_tile[threadIdx.x % kTileY][threadIdx.x / kTileY];
}

__global__ void __launch_bounds__(kTileX* kTileY) slice_extract_kernel(SliceRequest r, int tiles) {
    const int view = blockIdx.x / tiles;
    const float* v = r.views + 8 * view;
    const SliceAt s = {r.spectrum, r.gx, r.gy, r.gz / 2 + 1, r.inv_step, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
    slice_tile(s, blockIdx.x - view * tiles, r.cx, r.cy, r.nx, r.ny,
               r.arranged + (size_t)view * r.nx * (r.ny / 2 + 1));
}

// Batched form: every view has its own spectrum and image size; a block finds
// its view by binary search over the views' first tiles.
__global__ void __launch_bounds__(kTileX* kTileY) slice_extract_batch_kernel(const SliceView* __restrict__ views,
                                                                             int n_views) {
    int lo = 0, hi = n_views - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (views[mid].first_tile <= (long long)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const SliceView& V = views[lo];
    const SliceAt s = {V.spectrum, V.gx, V.gy, V.gz / 2 + 1, V.inv_step, V.u[0], V.u[1], V.u[2],
                       V.v[0], V.v[1], V.v[2], V.step[0], V.step[1]};
    slice_tile(s, (int)(blockIdx.x - V.first_tile), V.cx, V.cy, V.nx, V.ny, V.arranged);
}

}  // namespace

long long slice_tiles(int nx, int ny) {
    return (long long)((nx + kTileX - 1) / kTileX) * ((ny / 2 + 1 + kTileY - 1) / kTileY);
}

int launch_slice_extract_batch(const SliceView* d_views, int number_of_views, long long total_tiles,
                               cudaStream_t stream, KernelTimer* timer) {
    if (number_of_views <= 0 || total_tiles <= 0) return kOk;
    if (total_tiles > INT32_MAX) return set_error(kInvalidValue, "too many slice samples");
    timer_begin(timer, 1, stream);
    slice_extract_batch_kernel<<<(unsigned)total_tiles, kTileX * kTileY, 0, stream>>>(d_views, number_of_views);
    count_launch();
    timer_end(timer, 1, stream);
    return check_cuda(cudaGetLastError(), "slice_extract_batch_kernel launch");
}

int launch_slice_extract(const SliceRequest& req, KernelTimer* timer) {
    const long long tiles = slice_tiles(req.nx, req.ny);
    if (tiles * req.number_of_views <= 0) return kOk;
    if (tiles * req.number_of_views > INT32_MAX) return set_error(kInvalidValue, "too many slice samples");
    timer_begin(timer, 1, req.stream);
    slice_extract_kernel<<<(unsigned)(tiles * req.number_of_views), kTileX * kTileY, 0, req.stream>>>(req, (int)tiles);
    count_launch();
    timer_end(timer, 1, req.stream);
    return check_cuda(cudaGetLastError(), "slice_extract_kernel launch");
}

}  // namespace mv
