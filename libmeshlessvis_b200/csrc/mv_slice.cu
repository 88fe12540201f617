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
// Block: a tile of 64 x by 8 y samples of one view, a warp's lanes along x.  The
// loads are scattered (a sample's neighbours along y lie a whole row of l apart
// in the usual views), so the L1's lookups, one a cache line of a warp's load,
// and the instructions of the interpolation bound the kernel, not bytes.  Lanes
// along x touch fewer lines than along y (x runs partly along l, where values
// are contiguous), corners of weight 0 are not read (half of them or more where
// an axis of the view runs along the lattice in its steps), the same tile of all
// views runs together (they cut the same ring of the lattice), and samples leave
// through shared memory as 64-byte pieces of the y-fast layout.  360 views of
// 384 x 384 from 384^3, turning about y: 412 us with a thread an element in
// output order and every corner read, 302 with two lanes a sample (the corners
// at l and at l + 1; fewer lookups, more instructions), 242 us so.  Turning about
// y half of the corners have weight 0; about a tilted axis it was 405 us and is
// 338, at random attitudes 395 and 366.
#include <algorithm>

#include "mv_internal.h"

namespace mv {

namespace {

constexpr int kTileX = 64, kTileY = 8, kThreads = 32 * kTileY;

struct SliceAt {
    const float2* spectrum;
    int gx, gy, lz;
    float inv_step;
    float u0, u1, u2, v0, v1, v2, step_x, step_y;
};

// The slice sample (x, y): trilinear interpolation.
__device__ __forceinline__ float2 slice_sample(const SliceAt& s, int x, int y) {
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
    const int ii = (int)f0 + (s.gx >> 1), jj = (int)f1 + (s.gy >> 1), l0 = (int)f2;
    // corner (di, dj, dl), zero outside the stored lattice and where its weight
    // is (a spectrum has at most 2^31 elements: 32-bit indexes)
    const bool i0 = (unsigned)ii < (unsigned)s.gx, i1 = (unsigned)(ii + 1) < (unsigned)s.gx && t0 > 0.f;
    const bool j0 = (unsigned)jj < (unsigned)s.gy, j1 = (unsigned)(jj + 1) < (unsigned)s.gy && t1 > 0.f;
    const bool k0 = (unsigned)l0 < (unsigned)s.lz, k1 = (unsigned)(l0 + 1) < (unsigned)s.lz && t2 > 0.f;
    const int row = s.gy * s.lz;
    const float2* at = s.spectrum + (ii * row + jj * s.lz + l0);
    float2 c[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int di = e & 1, dj = (e >> 1) & 1, dl = (e >> 2) & 1;
        const bool in = (di ? i1 : i0) && (dj ? j1 : j0) && (dl ? k1 : k0);
        c[e] = in ? __ldg(at + (di * row + dj * s.lz + dl)) : make_float2(0.f, 0.f);
    }
    float re = 0.f, im = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int di = e & 1, dj = (e >> 1) & 1, dl = (e >> 2) & 1;
        const float w = (di ? t0 : 1.f - t0) * (dj ? t1 : 1.f - t1) * (dl ? t2 : 1.f - t2);
        re = fmaf(w, c[e].x, re);
        im = fmaf(w, c[e].y, im);
    }
    const float scale = s.step_x * s.step_y;
    return make_float2(re * scale, (conj ? -im : im) * scale);
}

// One tile of a view's [nx][ny / 2 + 1] elements.
__device__ __forceinline__ void slice_tile(const SliceAt& s, int tile_x, int tile_y, int cx, int cy, int nx, int ny,
                                           float2* __restrict__ out) {
    __shared__ float2 s_tile[kTileY][kTileX + 1];
    const int h = ny / 2 + 1;
    const int x0 = tile_x * kTileX, y0 = tile_y * kTileY;
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int y_row = y0 + row;
#pragma unroll
    for (int xs = lane; xs < kTileX; xs += 32) {
        const int ix = x0 + xs;
        float2 v = make_float2(0.f, 0.f);
        if (ix < nx && y_row < cy && (ix < cx || ix > nx - cx)) v = slice_sample(s, ix < cx ? ix : ix - nx, y_row);
        s_tile[row][xs] = v;
    }
    __syncthreads();
    const int ty = threadIdx.x % kTileY;
#pragma unroll
    for (int tx = threadIdx.x / kTileY; tx < kTileX; tx += kThreads / kTileY)
        if (x0 + tx < nx && y0 + ty < h) out[(size_t)(x0 + tx) * h + y0 + ty] = s_tile[ty][tx];
}

// Tiles from (first_x, first_y) on.
__global__ void __launch_bounds__(kThreads) slice_extract_kernel(SliceRequest r, int first_x, int first_y) {
    const int view = blockIdx.x;
    const float* v = r.views + 8 * view;
    const SliceAt s = {r.spectrum, r.gx, r.gy, r.gz / 2 + 1, r.inv_step, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
    slice_tile(s, first_x + blockIdx.z, first_y + blockIdx.y, r.cx, r.cy, r.nx, r.ny,
               r.arranged + (size_t)view * r.nx * (r.ny / 2 + 1));
}

// Batched form: every view has its own spectrum and image size; a block finds
// its view by binary search over the views' first tiles.
__global__ void __launch_bounds__(kThreads) slice_extract_batch_kernel(const SliceView* __restrict__ views,
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
    const int tile = (int)(blockIdx.x - V.first_tile), tiles_y = (V.ny / 2 + 1 + kTileY - 1) / kTileY;
    slice_tile(s, tile / tiles_y, tile % tiles_y, V.cx, V.cy, V.nx, V.ny, V.arranged);
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
    slice_extract_batch_kernel<<<(unsigned)total_tiles, kThreads, 0, stream>>>(d_views, number_of_views);
    count_launch();
    timer_end(timer, 1, stream);
    return check_cuda(cudaGetLastError(), "slice_extract_batch_kernel launch");
}

int launch_slice_extract(const SliceRequest& req, KernelTimer* timer) {
    const int tiles_x = (req.nx + kTileX - 1) / kTileX, tiles_y = (req.ny / 2 + 1 + kTileY - 1) / kTileY;
    if (req.number_of_views <= 0 || tiles_x <= 0 || tiles_y <= 0) return kOk;
    if ((long long)req.nx * (req.ny / 2 + 1) * req.number_of_views > (1LL << 40))
        return set_error(kInvalidValue, "too many slice samples");
    timer_begin(timer, 1, req.stream);
    // one launch; images of more tiles than a grid's y or z holds take several
    constexpr int kMost = 65535;
    for (int x = 0; x < tiles_x; x += kMost)
        for (int y = 0; y < tiles_y; y += kMost) {
            const dim3 grid((unsigned)req.number_of_views, std::min(kMost, tiles_y - y), std::min(kMost, tiles_x - x));
            slice_extract_kernel<<<grid, kThreads, 0, req.stream>>>(req, x, y);
            count_launch();
        }
    timer_end(timer, 1, req.stream);
    return check_cuda(cudaGetLastError(), "slice_extract_kernel launch");
}

}  // namespace mv
