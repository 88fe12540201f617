// Headless image post-processing after the C2R: the reference's display and
// file-output steps, restated as CUDA kernels over batches of images.
//
//   vis_images_normalize_to_rgb  vis_noninteractive/main.cpp:70-84: per image,
//       m = max over the raw samples (starting from sample 0), negatives
//       clamped to 0, grey RGB = sample / m.
//   vis_images_colormap          vis_wx/local_glsl.h:28-87 (fragment shader of
//       the interactive viewer): a = max(0, (a - min) / (max - min)); with log
//       scale a = (log(alpha a + eps) - log(eps)) / (log(alpha + eps) - log(eps)),
//       eps = 1e-3, alpha = 0.01; then a piecewise-linear colour map with 5
//       knots (maps 1 "fire", 2 "rainbow", 3 "ice"; above the last knot the
//       last colour).
//   vis_shift_registered_dataset shift_meshless_dataset (meshless.cpp:68-84) on
//       the registered device copy, so a frame loop need not re-register.
//   vis_write_ppm                binary PPM (P6) writer on the host, in place of
//       the reference's Magick++ JPEG writer (no image library on the target);
//       rows are written top row first after the same vertical flip the
//       reference applies (main.cpp:31).
// All image batches are float[images][Nx][Ny] with x slow, as vis_copy_to_host
// returns them; RGB outputs are float[images][Nx][Ny][3].
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <type_traits>
#include <vector>

#include "meshless_vis_b200.h"
#include "mv_divide.h"
#include "mv_internal.h"

namespace mv {
namespace {

// Order-preserving map of a float to an unsigned int (for atomicMax).
__device__ __forceinline__ unsigned int ordered(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unordered(unsigned int u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// One image per blockIdx.y, 16 bytes a load between its unaligned ends; fmaxf
// passes over NaNs, from the first sample, as the reference's scan does.  A block
// that has none but NaNs (the first sample where it has no pixels of its own) adds
// nothing; an image of NaNs keeps the start value, which is one.
__global__ void __launch_bounds__(256) image_max_kernel(const float* __restrict__ img, long long per_image,
                                                        unsigned int* out_max) {
    const float* p = img + (size_t)blockIdx.y * per_image;
    float m = p[0];
    const long long head = min(per_image, (long long)((16u - ((size_t)p & 15u)) & 15u) / 4);
    const long long quads = (per_image - head) / 4;
    const float4* q = reinterpret_cast<const float4*>(p + head);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, n = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
    for (long long i = t; i < quads; i += n) {
        const float4 v = q[i];
        m = fmaxf(m, fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
    }
    for (long long i = t; i < head; i += n) m = fmaxf(m, p[i]);
    for (long long i = head + 4 * quads + t; i < per_image; i += n) m = fmaxf(m, p[i]);
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float wm[32];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        float v = threadIdx.x < (blockDim.x >> 5) ? wm[threadIdx.x] : p[0];
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (threadIdx.x == 0 && v == v) atomicMax(out_max + blockIdx.y, ordered(v));
    }
}

// Pixels to RGB: a block takes kRgbPixels consecutive pixels, four a thread (one
// 16-byte load where the images are aligned), and writes their 3 kRgbPixels
// floats from shared memory, 16 bytes a thread and store.  Bound: HBM (4 bytes
// read, 12 written a pixel).
constexpr int kRgbThreads = 256, kRgbPixels = 4 * kRgbThreads;

template <typename Rgb>
__device__ __forceinline__ void pixels_to_rgb(const float* __restrict__ img, long long count, float* __restrict__ rgb,
                                              float4* s_out, Rgb to_rgb) {
    const long long first = (long long)blockIdx.x * kRgbPixels;
    const int in = (int)min((long long)kRgbPixels, count - first);
    const int l = 4 * threadIdx.x;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (l + 4 <= in && ((size_t)img & 15u) == 0) {
        const float4 q = __ldcs(reinterpret_cast<const float4*>(img + first + l));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (l + i < in) v[i] = __ldcs(img + first + l + i);
    }
    float c[12];
#pragma unroll
    for (int i = 0; i < 4; ++i) to_rgb(first, min(l + i, in - 1), v[i], c + 3 * i);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        s_out[3 * threadIdx.x + i] = make_float4(c[4 * i], c[4 * i + 1], c[4 * i + 2], c[4 * i + 3]);
    __syncthreads();
    float* out = rgb + 3 * first;
    if (in == kRgbPixels && ((size_t)rgb & 15u) == 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
            __stcs(reinterpret_cast<float4*>(out) + i * kRgbThreads + threadIdx.x, s_out[i * kRgbThreads + threadIdx.x]);
    } else {
        const float* s = reinterpret_cast<const float*>(s_out);
        for (int i = threadIdx.x; i < 3 * in; i += kRgbThreads) __stcs(out + i, s[i]);
    }
}

__global__ void __launch_bounds__(kRgbThreads) normalize_rgb_kernel(const float* __restrict__ img, long long per_image,
                                                                    long long count,
                                                                    const unsigned int* __restrict__ maxes,
                                                                    float* __restrict__ rgb) {
    __shared__ float4 s_out[3 * kRgbThreads];
    // the block's first image and its first pixel's place in it; most blocks
    // lie in one image
    const long long first = (long long)blockIdx.x * kRgbPixels;
    const long long image = first / per_image, at = first - image * per_image;
    const bool one = at + kRgbPixels <= per_image;
    const float m0 = unordered(__ldg(maxes + image));
    pixels_to_rgb(img, count, rgb, s_out, [&](long long, int l, float a, float* c) {
        const float m = one ? m0 : unordered(__ldg(maxes + image + (at + l) / per_image));
        if (a < 0.f) a = 0.f;
        c[0] = c[1] = c[2] = a / m;
    });
}

struct Knots {
    float x[5];
    float c[5][3];
};

__host__ __device__ inline Knots color_knots(int map) {
    if (map == 2) return Knots{{0.f, 0.25f, 0.5f, 0.75f, 1.f},
                               {{0, 0, 1}, {0, 1, 1}, {0, 1, 0}, {1, 1, 0}, {1, 0, 0}}};
    if (map == 3) return Knots{{0.f, 0.475f, 0.694f, 0.745f, 1.f},
                               {{0, 0, 0}, {0.f, 0.004f, 0.686f}, {0.f, 0.42f, 1.f}, {0.f, 0.518f, 1.f}, {1, 1, 1}}};
    return Knots{{0.f, 0.475f, 0.694f, 0.745f, 1.f},
                 {{0, 0, 0}, {0.686f, 0.004f, 0.f}, {1.f, 0.42f, 0.f}, {1.f, 0.518f, 0.f}, {1, 1, 1}}};
}

// The colour map's segments and colours come from shared memory (indexed by
// a thread's own segment, kernel parameters went through local memory: 1.90 ms
// for 360 images of 384 x 384, where their bytes take 0.13).  The divisors are
// the same for all pixels, their reciprocals are taken once a thread: with four
// full divisions a pixel the instructions bounded the kernel: 413 us with the
// normalisation of the same images, 380 so (the colour map alone 203).  Pixels
// too near the range's start for that are divided: 208 us, at 8 blocks an SM (225
// at the 40 registers that it would take without the bound; a factor on all
// numbers in place of the test, 209, or 197 without the logarithm, where the test
// takes 192).
__global__ void __launch_bounds__(kRgbThreads, 8) colormap_kernel(const float* __restrict__ img, long long count,
                                                                  float imin, float imax, int log_scale, Knots k,
                                                                  float* __restrict__ rgb) {
    __shared__ float4 s_out[3 * kRgbThreads];
    __shared__ float4 s_x[8];     // segment up to knot i: its ends, length, 1 / length
    __shared__ float4 s_c[8];     // colours of the knots
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const float x0 = k.x[i > 0 ? i - 1 : 0], d = k.x[i] - x0;
            s_x[i] = make_float4(x0, k.x[i], d, 1.f / d);
            s_c[i] = make_float4(k.c[i][0], k.c[i][1], k.c[i][2], 0.f);
        }
    }
    __syncthreads();
    const float eps = 1e-3f, alpha = 0.01f;
    const float log_eps = logf(eps), log_range = logf(alpha + eps) - logf(eps), log_r = 1.f / log_range;
    const float range = imax - imin, range_r = 1.f / range;
    // pixels up to here above imin (as bits, +0 the last of all) are divided; all
    // of them where the range is none that divide_by takes
    const bool shared = range > 1e-30f && range < 1e30f;
    const uint32_t small = shared ? __float_as_uint(divide_by_least(range)) - 2u : ~0u;
    auto color = [&](float above, float* c, auto by_reciprocal) {
        constexpr bool kShared = decltype(by_reciprocal)::value;
        float a = fmaxf(0.f, kShared ? divide_by(above, range, range_r) : above / range);
        if (log_scale) a = divide_by(-log_eps + logf(alpha * a + eps), log_range, log_r);
        // the first knot at or past a; past the last (or for NaNs) its colour
        const int i = a <= k.x[1] ? 1 : a <= k.x[2] ? 2 : a <= k.x[3] ? 3 : 4;
        const float4 x = s_x[i], c1 = s_c[i], c0 = s_c[i - 1];
        auto weight = [&](float l) { return kShared ? divide_finite(l, x.z, x.w) : l / x.z; };
        const bool inside = a <= x.y;
        const float wi = inside ? weight(a - x.x) : 1.f, wl = inside ? weight(x.y - a) : 0.f;
        c[0] = wi * c1.x + wl * c0.x;
        c[1] = wi * c1.y + wl * c0.y;
        c[2] = wi * c1.z + wl * c0.z;
    };
    pixels_to_rgb(img, count, rgb, s_out, [&](long long, int, float v, float* c) {
        const float above = v - imin;
        if (__float_as_uint(above) - 1u <= small) color(above, c, std::false_type{});
        else color(above, c, std::true_type{});
    });
}

__global__ void shift_kernel(float4* p, int n, float dx, float dy, float dz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 v = p[i];
    v.x += dx;
    v.y += dy;
    v.z += dz;
    p[i] = v;
}

}  // namespace

int config_stream_and_scratch(VisConfig* c, cudaStream_t* stream, void** scratch, size_t bytes);  // mv_api.cu

}  // namespace mv

using namespace mv;

extern "C" {

int vis_images_normalize_to_rgb(VisConfig* vis_config, const float* d_images, int number_of_images,
                                int2 number_of_samples, float* d_rgb) {
    const long long per_image = (long long)number_of_samples.x * number_of_samples.y;
    if (!d_images || !d_rgb || number_of_images < 0 || per_image <= 0)
        return set_error(kInvalidValue, "vis_images_normalize_to_rgb: bad arguments");
    if (number_of_images == 0) return kOk;
    cudaStream_t stream;
    void* scratch = nullptr;
    int rc = config_stream_and_scratch(vis_config, &stream, &scratch, sizeof(unsigned int) * number_of_images);
    if (rc != kOk) return rc;
    unsigned int* maxes = static_cast<unsigned int*>(scratch);
    rc = check_cuda(cudaMemsetAsync(maxes, 0, sizeof(unsigned int) * number_of_images, stream),  // below every ordered float
                    "cudaMemsetAsync");
    if (rc != kOk) return rc;
    // as many images at a time as the L2 keeps between the two passes
    const long long group = std::min<long long>(32768, std::max<long long>(1, ((long long)48 << 20) / 4 / per_image));
    for (long long g = 0; g < number_of_images; g += group) {
        const long long images = std::min<long long>(group, number_of_images - g), count = images * per_image;
        const float* img = d_images + g * per_image;
        const int blocks_x = (int)std::min<long long>(16, (per_image + 1023) / 1024);
        image_max_kernel<<<dim3(blocks_x, (unsigned)images), 256, 0, stream>>>(img, per_image, maxes + g);
        count_launch();
        normalize_rgb_kernel<<<(unsigned)((count + kRgbPixels - 1) / kRgbPixels), kRgbThreads, 0, stream>>>(
            img, per_image, count, maxes + g, d_rgb + 3 * g * per_image);
        count_launch();
    }
    return check_cuda(cudaGetLastError(), "vis_images_normalize_to_rgb");
}

int vis_images_colormap(VisConfig* vis_config, const float* d_images, int number_of_images, int2 number_of_samples,
                        float intensity_min, float intensity_max, int log_scale, int color_map, float* d_rgb) {
    const long long count = (long long)number_of_samples.x * number_of_samples.y * number_of_images;
    if (!d_images || !d_rgb || number_of_images < 0 || count < 0 || color_map < 1 || color_map > 3 ||
        !(intensity_max != intensity_min))
        return set_error(kInvalidValue, "vis_images_colormap: bad arguments");
    if (count == 0) return kOk;
    cudaStream_t stream;
    int rc = config_stream_and_scratch(vis_config, &stream, nullptr, 0);
    if (rc != kOk) return rc;
    colormap_kernel<<<(unsigned)((count + kRgbPixels - 1) / kRgbPixels), kRgbThreads, 0, stream>>>(
        d_images, count, intensity_min, intensity_max, log_scale, color_knots(color_map), d_rgb);
    count_launch();
    return check_cuda(cudaGetLastError(), "vis_images_colormap");
}

int vis_shift_registered_dataset(VisConfig* vis_config, MeshlessDataset* meshless_dataset, float x, float y,
                                 float z) {
    if (!meshless_dataset || (meshless_dataset->number_of_groups > 0 && !meshless_dataset->groups))
        return set_error(kInvalidValue, "vis_shift_registered_dataset: NULL dataset");
    cudaStream_t stream;
    int rc = config_stream_and_scratch(vis_config, &stream, nullptr, 0);
    if (rc != kOk) return rc;
    for (int g = 0; g < meshless_dataset->number_of_groups; ++g) {
        const Group& grp = meshless_dataset->groups[g];
        if (grp.number_of_terms <= 0) continue;
        if (!grp.d_constraints)
            return set_error(kNotRegistered, "vis_shift_registered_dataset: group not registered");
        shift_kernel<<<(grp.number_of_terms + 255) / 256, 256, 0, stream>>>(
            reinterpret_cast<float4*>(grp.d_constraints), grp.number_of_terms, x, y, z);
        count_launch();
    }
    return check_cuda(cudaGetLastError(), "vis_shift_registered_dataset");
}

int vis_write_ppm(const char* filename, const float* h_rgb, int2 number_of_samples) {
    const int w = number_of_samples.x, h = number_of_samples.y;
    if (!filename || !h_rgb || w < 1 || h < 1) return set_error(kInvalidValue, "vis_write_ppm: bad arguments");
    FILE* f = std::fopen(filename, "wb");
    if (!f) return set_error(kInvalidValue, std::string("vis_write_ppm: cannot open ") + filename);
    std::fprintf(f, "P6\n%d %d\n255\n", w, h);
    // The reference reads the x-slow image as rows of length Nx (Magick
    // read(width, height, ...)) and flips it vertically before writing.
    std::vector<unsigned char> row((size_t)3 * w);
    for (int r = h - 1; r >= 0; --r) {
        for (int c = 0; c < w; ++c)
            for (int k = 0; k < 3; ++k) {
                float v = h_rgb[3 * ((size_t)r * w + c) + k];
                v = v < 0.f ? 0.f : (v > 1.f ? 1.f : v);
                row[3 * c + k] = (unsigned char)std::lround(v * 255.f);
            }
        if (std::fwrite(row.data(), 1, row.size(), f) != row.size()) {
            std::fclose(f);
            return set_error(kInvalidValue, "vis_write_ppm: write failed");
        }
    }
    std::fclose(f);
    return kOk;
}

}  // extern "C"
