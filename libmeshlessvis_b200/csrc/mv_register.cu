// Statistics of a registered group, from its device copy: the largest |weight|
// and the radius extremes, and the smoothing-length histogram (HBinStats).  The
// same results as the host's serial passes (mv_api.cu, host_statistics): maxima,
// minima and counts do not depend on the order, NaNs are passed over, and a
// radius's bin is found by the same float comparisons against the same edges.
// Bound: launch latency and the copies around them (30,011 particles take 5 us a
// kernel), at large sizes HBM.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "mv_device.cuh"
#include "mv_internal.h"

namespace mv {
namespace {

// Order-preserving map of a float to an unsigned integer, never 0 for a number.
__host__ __device__ __forceinline__ uint32_t ordered_bits(uint32_t u) {
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__global__ void __launch_bounds__(256) register_extremes_kernel(const float4* __restrict__ particles,
                                                                const float* __restrict__ radii, int n,
                                                                RegisterStats* out) {
    uint32_t w = 0u, lo = 0u, hi = 0u;
    bool nan = false;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float a = fabsf(particles[i].w);
        if (a >= 0.f) w = max(w, ordered_bits(__float_as_uint(a)));
        if (radii) {
            const float r = radii[i] + 0.f;  // -0 counts as 0
            if (r == r) {
                const uint32_t o = ordered_bits(__float_as_uint(r));
                lo = max(lo, ~o);
                hi = max(hi, o);
            } else {
                nan = true;
            }
        }
    }
    w = __reduce_max_sync(0xffffffffu, w);
    lo = __reduce_max_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    nan = __any_sync(0xffffffffu, nan);
    if ((threadIdx.x & 31) == 0) {
        if (w) atomicMax(&out->weight_max, w);
        if (lo) atomicMax(&out->radius_min, lo);
        if (hi) atomicMax(&out->radius_max, hi);
        if (nan) atomicMax(&out->radius_nan, 1u);
    }
}

// Device layout of a histogram: edges, counts, largest |weight| (bits).
struct Histogram {
    float edges[kHBinFine + 1];
    int count[kHBinFine];
    uint32_t wmax[kHBinFine];
};

__global__ void __launch_bounds__(256) register_histogram_kernel(const float4* __restrict__ particles,
                                                                 const float* __restrict__ radii, int n,
                                                                 Histogram* h) {
    __shared__ float s_edges[kHBinFine + 1];
    __shared__ int s_count[kHBinFine];
    __shared__ uint32_t s_wmax[kHBinFine];
    for (int i = threadIdx.x; i <= kHBinFine; i += blockDim.x) s_edges[i] = h->edges[i];
    for (int i = threadIdx.x; i < kHBinFine; i += blockDim.x) {
        s_count[i] = 0;
        s_wmax[i] = 0u;
    }
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int f = hbin_of(s_edges, kHBinFine, radii[i]);
        const float a = fabsf(particles[i].w);
        atomicAdd(&s_count[f], 1);
        if (a > 0.f) atomicMax(&s_wmax[f], __float_as_uint(a));  // positive floats order as their bits
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kHBinFine; i += blockDim.x) {
        if (s_count[i]) atomicAdd(&h->count[i], s_count[i]);
        if (s_wmax[i]) atomicMax(&h->wmax[i], s_wmax[i]);
    }
}

int register_blocks(int n) { return std::max(1, std::min((n + 1023) / 1024, 2 * device_sm_count())); }

}  // namespace

float register_value(uint32_t o, float none) {
    if (o == 0u) return none;
    const uint32_t u = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
    float f;
    std::memcpy(&f, &u, sizeof f);
    return f;
}

int launch_register_extremes_clear(RegisterStats* d, int n, cudaStream_t stream) {
    return check_cuda(cudaMemsetAsync(d, 0, sizeof(RegisterStats) * (size_t)n, stream), "cudaMemsetAsync");
}

int launch_register_extremes(const float4* particles, const float* radii, int n, RegisterStats* out,
                             cudaStream_t stream) {
    register_extremes_kernel<<<register_blocks(n), 256, 0, stream>>>(particles, radii, n, out);
    count_launch();
    return check_cuda(cudaGetLastError(), "register_extremes_kernel launch");
}

size_t register_histogram_bytes() { return (sizeof(Histogram) + 255) / 256 * 256; }

int launch_register_histogram(const float4* particles, const float* radii, int n, const float* edges, void* out,
                              cudaStream_t stream) {
    Histogram* h = static_cast<Histogram*>(out);
    int st = check_cuda(cudaMemsetAsync(h->count, 0, sizeof(h->count) + sizeof(h->wmax), stream), "cudaMemsetAsync");
    if (st == kOk)
        st = check_cuda(cudaMemcpyAsync(h->edges, edges, sizeof(h->edges), cudaMemcpyHostToDevice, stream),
                        "registration edges H2D");
    if (st != kOk) return st;
    register_histogram_kernel<<<register_blocks(n), 256, 0, stream>>>(particles, radii, n, h);
    count_launch();
    return check_cuda(cudaGetLastError(), "register_histogram_kernel launch");
}

void read_register_histogram(const void* host, int* count, float* wmax) {
    const Histogram* h = static_cast<const Histogram*>(host);
    std::memcpy(count, h->count, sizeof(h->count));
    std::memcpy(wmax, h->wmax, sizeof(h->wmax));
}

}  // namespace mv
