// Bandwidth-bound layers of the vDNN training path for sm_100a: ReLU, max-pool, softmax,
// tensor difference, bias add / bias gradient, LRN, loss, axpy, fill.
// All kernels stream fp32 NCHW tensors with 16-byte accesses where alignment allows and size
// their grids in whole multiples of the SM count.
#include <cooperative_groups.h>
#include <math.h>

#include <mutex>
#include <vector>

#include "common.cuh"

namespace vdnn {

thread_local int g_last_cuda_error = 0;
unsigned long long g_kernel_launches = 0;

int sm_count() {
    static std::vector<int> cached;                      // indexed by device ordinal, grown on demand
    static std::mutex lock;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 148;
    std::lock_guard<std::mutex> g(lock);
    if (cached.size() <= static_cast<size_t>(dev)) cached.resize(dev + 1, 0);
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

namespace {

namespace cg = cooperative_groups;

// Times in the comments of this file, before and after: B200, calls one behind the other in a graph, large tensors taken from
// three sets that together pass L2, small ones resident in it (a launch of one value takes 1.1 us so).  A single call behind a
// flush of L2 reads about 6 us more, the launch.

constexpr int kThreads = 256;

// Blocks for a streaming kernel in which every thread handles `per_thread` items per loop trip.
inline int stream_grid(size_t items, int per_thread) {
    const size_t want = ceil_div(items, static_cast<size_t>(kThreads) * per_thread);
    const size_t cap = static_cast<size_t>(sm_count()) * 8;     // 8 x 256 threads = a full SM
    size_t g = want < cap ? want : cap;
    if (g > static_cast<size_t>(sm_count())) g = g / sm_count() * sm_count();
    return g ? static_cast<int>(g) : 1;
}

// Images (of `items` items each) whose items a 32-bit index can address: FastDiv takes dividends below 2^31.
inline int images_per_launch(int n, size_t items) {
    const size_t most = 0x7fffffffu / items;
    return most < static_cast<size_t>(n) ? static_cast<int>(most) : n;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

__device__ __forceinline__ float relu1(float v) { return v > 0.0f ? v : (v != v ? v : 0.0f); }

// ---------------------------------------------------------------- ReLU
__global__ void __launch_bounds__(kThreads) relu_fwd_kernel(size_t n4, size_t n, const float* __restrict__ x,
                                                            float* __restrict__ y) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    float4* y4 = reinterpret_cast<float4*>(y);
    for (; i + 3 * stride < n4; i += 4 * stride) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = __ldcs(x4 + i + u * stride);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            v[u].x = relu1(v[u].x); v[u].y = relu1(v[u].y); v[u].z = relu1(v[u].z); v[u].w = relu1(v[u].w);
            y4[i + u * stride] = v[u];
        }
    }
    for (; i < n4; i += stride) {
        float4 v = __ldcs(x4 + i);
        v.x = relu1(v.x); v.y = relu1(v.y); v.z = relu1(v.z); v.w = relu1(v.w);
        y4[i] = v;
    }
    // scalar tail (and the whole tensor when the pointers are not 16-byte aligned: n4 == 0)
    for (size_t j = n4 * 4 + static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < n; j += stride)
        y[j] = relu1(x[j]);
}

__global__ void __launch_bounds__(kThreads) relu_bwd_kernel(size_t n4, size_t n, const float* __restrict__ dy,
                                                            const float* __restrict__ x, float* __restrict__ dx) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const float4* d4 = reinterpret_cast<const float4*>(dy);
    float4* o4 = reinterpret_cast<float4*>(dx);
    for (; i + stride < n4; i += 2 * stride) {
        float4 a[2], g[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) { a[u] = __ldcs(x4 + i + u * stride); g[u] = __ldcs(d4 + i + u * stride); }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            float4 r;
            r.x = a[u].x > 0.0f ? g[u].x : 0.0f; r.y = a[u].y > 0.0f ? g[u].y : 0.0f;
            r.z = a[u].z > 0.0f ? g[u].z : 0.0f; r.w = a[u].w > 0.0f ? g[u].w : 0.0f;
            o4[i + u * stride] = r;
        }
    }
    for (; i < n4; i += stride) {
        float4 a = __ldcs(x4 + i), g = __ldcs(d4 + i), r;
        r.x = a.x > 0.0f ? g.x : 0.0f; r.y = a.y > 0.0f ? g.y : 0.0f;
        r.z = a.z > 0.0f ? g.z : 0.0f; r.w = a.w > 0.0f ? g.w : 0.0f;
        o4[i] = r;
    }
    for (size_t j = n4 * 4 + static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < n; j += stride)
        dx[j] = x[j] > 0.0f ? dy[j] : 0.0f;
}

// ---------------------------------------------------------------- tanh / sigmoid (mode as in vdnn_b200.h)
template <int MODE> __device__ __forceinline__ float act1(float x) {
    return MODE == VDNN_ACT_TANH ? tanhf(x) : 1.0f / (1.0f + expf(-x));
}
template <int MODE> __device__ __forceinline__ float dact1(float y, float dy) {
    return MODE == VDNN_ACT_TANH ? dy * (1.0f - y * y) : dy * y * (1.0f - y);
}

template <int MODE>
__global__ void __launch_bounds__(kThreads) act_fwd_kernel(size_t n4, size_t n, const float* __restrict__ x,
                                                           float* __restrict__ y) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    const size_t first = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    float4* y4 = reinterpret_cast<float4*>(y);
    for (size_t i = first; i < n4; i += stride) {
        float4 v = __ldcs(x4 + i);
        v.x = act1<MODE>(v.x); v.y = act1<MODE>(v.y); v.z = act1<MODE>(v.z); v.w = act1<MODE>(v.w);
        y4[i] = v;
    }
    for (size_t j = n4 * 4 + first; j < n; j += stride) y[j] = act1<MODE>(x[j]);
}

template <int MODE>
__global__ void __launch_bounds__(kThreads) act_bwd_kernel(size_t n4, size_t n, const float* __restrict__ y,
                                                           const float* __restrict__ dy, float* __restrict__ dx) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    const size_t first = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const float4* y4 = reinterpret_cast<const float4*>(y);
    const float4* d4 = reinterpret_cast<const float4*>(dy);
    float4* o4 = reinterpret_cast<float4*>(dx);
    for (size_t i = first; i < n4; i += stride) {
        const float4 a = __ldcs(y4 + i), d = __ldcs(d4 + i);
        float4 o;
        o.x = dact1<MODE>(a.x, d.x); o.y = dact1<MODE>(a.y, d.y); o.z = dact1<MODE>(a.z, d.z); o.w = dact1<MODE>(a.w, d.w);
        o4[i] = o;
    }
    for (size_t j = n4 * 4 + first; j < n; j += stride) dx[j] = dact1<MODE>(y[j], dy[j]);
}

// ---------------------------------------------------------------- out = a - b, w += alpha g, fill
// The loss's seed and the softmax kernels below end every step, a few microseconds each, and are launched early
// (tc::launch_early): the four of 64 x 1000 called one behind the other take 12.7 us instead of 20.5.  Such a kernel starts
// beside its predecessor, so it reads what that one wrote by plain loads through plain pointers: nothing may be fetched ahead,
// or through the read-only path, of the wait.
__global__ void __launch_bounds__(kThreads) sub_kernel(size_t n4, size_t n, const float* a, const float* b, float* out) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    const size_t first = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    tc::follow_up();
    tc::after_predecessor();
    const float4* a4 = reinterpret_cast<const float4*>(a);
    const float4* b4 = reinterpret_cast<const float4*>(b);
    for (size_t i = first; i < n4; i += stride) {
        const float4 u = a4[i], v = b4[i];
        reinterpret_cast<float4*>(out)[i] = make_float4(u.x - v.x, u.y - v.y, u.z - v.z, u.w - v.w);
    }
    for (size_t j = n4 * 4 + first; j < n; j += stride) out[j] = a[j] - b[j];
}

__global__ void __launch_bounds__(kThreads) axpy_kernel(size_t n4, size_t n, float alpha, const float* __restrict__ g,
                                                        float* __restrict__ w) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    const float4* g4 = reinterpret_cast<const float4*>(g);
    float4* w4 = reinterpret_cast<float4*>(w);
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += stride) {
        float4 a = g4[i], b = w4[i];
        b.x = fmaf(alpha, a.x, b.x); b.y = fmaf(alpha, a.y, b.y); b.z = fmaf(alpha, a.z, b.z); b.w = fmaf(alpha, a.w, b.w);
        w4[i] = b;
    }
    for (size_t j = n4 * 4 + static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < n; j += stride)
        w[j] = fmaf(alpha, g[j], w[j]);
}

__global__ void __launch_bounds__(kThreads) fill_kernel(size_t n, float v, float* __restrict__ dst) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = v;
}

// ---------------------------------------------------------------- bias add, bias gradient
// y[(n*K + k)*pq + i] += alpha * bias[k] over the flat tensor, `div` = pq and K (see vdnn_add_bias for the three forms):
//   BIAS_PLANE4  pq % 4 == 0: a float4 lies inside one channel's plane;   BIAS_ROW4  pq == 1, K % 4 == 0: a float4 takes
//   four channels;   BIAS_SCALAR  everything else.
// Bound by memory.  The form before this took a block per (image, channel) plane, which for a fully connected layer is one
// block for every single value: 64 x 4096 cost 63 us; flat it costs 1.8 (1 MB in, 1 MB out).
enum BiasForm { BIAS_SCALAR, BIAS_PLANE4, BIAS_ROW4 };
template <BiasForm FORM>
__global__ void __launch_bounds__(kThreads) add_bias_kernel(uint32_t items, FastDiv div_pq, FastDiv div_k, float alpha,
                                                            const float* __restrict__ bias, float* __restrict__ y) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < items; i += stride) {
        uint32_t plane, rest, ch;
        if (FORM == BIAS_ROW4) plane = i; else div_pq.divmod(i, plane, rest);
        div_k.divmod(plane, rest, ch);
        if (FORM == BIAS_SCALAR) {
            y[i] += alpha * bias[ch];
        } else {
            float4 b;
            if (FORM == BIAS_ROW4) b = __ldg(reinterpret_cast<const float4*>(bias) + ch);
            else b.x = b.y = b.z = b.w = __ldg(bias + ch);
            float4 v = reinterpret_cast<float4*>(y)[i];
            v.x += alpha * b.x; v.y += alpha * b.y; v.z += alpha * b.z; v.w += alpha * b.w;
            reinterpret_cast<float4*>(y)[i] = v;
        }
    }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum of one value per block over the blocks of a cluster; the result is valid in the first thread of rank 0.  Every
// thread of the cluster calls it.
__device__ __forceinline__ float cluster_sum(float block_value, float* slot) {
    cg::cluster_group cluster = cg::this_cluster();
    if (threadIdx.x == 0) *slot = block_value;
    cluster.sync();
    float v = 0.0f;
    if (cluster.block_rank() == 0 && threadIdx.x == 0)
        for (unsigned r = 0; r < cluster.num_blocks(); ++r) v += *cluster.map_shared_rank(slot, r);
    cluster.sync();                         // no block leaves while its slot may still be read
    return v;
}

// db[ch] = alpha * sum over (n, pq) of dy[n][ch][pq] + beta * db[ch].  A cluster of up to eight blocks takes a channel and
// adds its parts through distributed shared memory: one launch, no pre-scaling pass, no atomics, the same bits every time.
// Bound by reading dy.  The flat index over (image, pixel) keeps all threads busy whatever the plane size; VEC = planes of
// whole float4.  Measured (64 x 96 x 55 x 55, planes of odd size): 58.6 us with one strided plane after another, now 26.5
// (2.8 TB/s).
template <int VEC>
__global__ void __launch_bounds__(512) bwd_bias_kernel(uint32_t items, int k, FastDiv div_plane, float alpha, const float* __restrict__ dy,
                                                       float beta, float* __restrict__ db) {
    __shared__ float part[16];
    __shared__ float slot;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t slices = cluster.num_blocks(), rank = cluster.block_rank();
    const uint32_t ch = blockIdx.x / slices;
    const uint32_t plane = div_plane.d;                      // items per (image, channel) plane
    const uint32_t step = slices * blockDim.x;
    const uint32_t first = rank * blockDim.x + threadIdx.x;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    auto at = [&](uint32_t i) -> size_t {
        uint32_t in, off;
        div_plane.divmod(i, in, off);
        return (static_cast<size_t>(in) * k + ch) * plane + off;
    };
    auto load = [&](uint32_t i) -> float {
        if (VEC == 4) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(dy) + at(i));
            return (v.x + v.y) + (v.z + v.w);
        }
        return __ldg(dy + at(i));
    };
    uint32_t i = first;
    for (; i + 3 * static_cast<size_t>(step) < items; i += 4 * step)
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] += load(i + u * step);
    for (; i < items; i += step) acc[0] += load(i);
    float v = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) v = warp_sum(threadIdx.x < (blockDim.x >> 5) ? part[threadIdx.x] : 0.0f);
    v = cluster_sum(v, &slot);
    if (rank == 0 && threadIdx.x == 0) db[ch] = beta == 0.0f ? alpha * v : fmaf(alpha, v, beta * db[ch]);
}

// The same for planes of fewer than 32 values (a fully connected layer has planes of one): dy is then read along its rows,
// a block taking 32 / pq whole channels = up to 32 adjacent columns, eight rows at a time; blocks of a cluster share the
// rows.  Per-plane reading cost 90 us for 64 x 4096 (a block of 256 threads per channel, one value per row each); this
// form 3.2.
__global__ void __launch_bounds__(256) bwd_bias_narrow_kernel(int n, int k, int pq, float alpha, const float* __restrict__ dy, float beta,
                                                              float* __restrict__ db) {
    __shared__ float part[8][33];
    cg::cluster_group cluster = cg::this_cluster();
    const int lane = threadIdx.x & 31, row_lane = threadIdx.x >> 5;
    const int per_block = 32 / pq;                           // channels of this block
    const int slices = cluster.num_blocks(), rank = cluster.block_rank();
    const int ch0 = blockIdx.x / slices * per_block;
    const int cols = min(per_block, k - ch0) * pq;
    const size_t pitch = static_cast<size_t>(k) * pq;
    const float* col = dy + static_cast<size_t>(ch0) * pq + lane;
    const int step = 8 * slices;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (lane < cols) {
        int r = rank * 8 + row_lane;
        for (; r + 3 * step < n; r += 4 * step)
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[u] += __ldg(col + (static_cast<size_t>(r) + u * step) * pitch);
        for (; r < n; r += step) acc[0] += __ldg(col + static_cast<size_t>(r) * pitch);
    }
    part[row_lane][lane] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
    __syncthreads();
    if (row_lane == 0) {
        float v = 0.0f;
#pragma unroll
        for (int r = 0; r < 8; ++r) v += part[r][lane];
        part[0][lane] = v;
    }
    cluster.sync();
    if (rank == 0 && static_cast<int>(threadIdx.x) < per_block && ch0 + static_cast<int>(threadIdx.x) < k) {
        float v = 0.0f;
        for (unsigned b = 0; b < cluster.num_blocks(); ++b) {
            const float* row = cluster.map_shared_rank(&part[0][0], b);
            for (int j = 0; j < pq; ++j) v += row[threadIdx.x * pq + j];
        }
        const int ch = ch0 + threadIdx.x;
        db[ch] = beta == 0.0f ? alpha * v : fmaf(alpha, v, beta * db[ch]);
    }
    cluster.sync();
}

// ---------------------------------------------------------------- max pooling
// One thread per output; the flat index is taken apart with multiplications (a 64-bit division per output was a third of the
// time of this kernel).  WIN > 0: square window of that size, unrolled, so its loads are in flight together; 0: any window.
// Bound by L1 (a stride-2 row touches every line twice): 64 x 96 x 55 x 55, 3 x 3 / 2: 42.0 us before, 22.2 now (4.2 TB/s).
template <int WIN>
__global__ void __launch_bounds__(kThreads) maxpool_fwd_generic(uint32_t total, int h, int w, FastDiv div_p, FastDiv div_q, int wh, int ww,
                                                                int sh, int sw, const float* __restrict__ x,
                                                                float* __restrict__ y) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        uint32_t t, q, plane, p;
        div_q.divmod(idx, t, q);
        div_p.divmod(t, plane, p);
        const float* xp = x + static_cast<size_t>(plane) * h * w + static_cast<size_t>(p * sh) * w + q * sw;
        float m = -INFINITY;
        if (WIN > 0) {
            float v[WIN > 0 ? WIN * WIN : 1];
#pragma unroll
            for (int i = 0; i < WIN; ++i)
#pragma unroll
                for (int j = 0; j < WIN; ++j) v[i * WIN + j] = __ldg(xp + i * w + j);
#pragma unroll
            for (int i = 0; i < WIN * WIN; ++i) if (v[i] > m) m = v[i];
        } else {
            for (int i = 0; i < wh; ++i)
                for (int j = 0; j < ww; ++j) {
                    const float v = xp[i * w + j];
                    if (v > m) m = v;
                }
        }
        y[idx] = m;
    }
}

// 2x2 window, stride 2, even H and W, W % 4 == 0: each thread reads two float4 rows and writes
// two outputs (float2).
__global__ void __launch_bounds__(kThreads) maxpool_fwd_2x2(size_t pairs, int w, int Qh /* Q/2 */,
                                                            const float* __restrict__ x, float* __restrict__ y) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < pairs; idx += stride) {
        const size_t row = idx / Qh;                 // (plane * P + p)
        const int qp = static_cast<int>(idx - row * Qh);
        const float* xr = x + row * 2 * w + qp * 4;
        const float4 a = __ldcs(reinterpret_cast<const float4*>(xr));
        const float4 b = __ldcs(reinterpret_cast<const float4*>(xr + w));
        float m0 = -INFINITY, m1 = -INFINITY;
        if (a.x > m0) m0 = a.x; if (a.y > m0) m0 = a.y; if (b.x > m0) m0 = b.x; if (b.y > m0) m0 = b.y;
        if (a.z > m1) m1 = a.z; if (a.w > m1) m1 = a.w; if (b.z > m1) m1 = b.z; if (b.w > m1) m1 = b.w;
        reinterpret_cast<float2*>(y)[idx] = make_float2(m0, m1);
    }
}

// Windows of 2 x 2 or 3 x 3 at stride 2.  A lane owns two columns of dx (a window's first two) and walks down a band of
// window rows: it finds each window's first maximum in registers -- the last row of a 3 x 3 window is the first of the next --
// and hands place and dy to its right neighbour by shuffle, so that no shared memory and no barrier is involved and four
// windows' loads are in flight.  The columns of all planes form one list: small planes share a warp; of a 3 x 3 warp's 32
// columns the first is there for its neighbour only.  Sums are in scan order, the same every time.
// With the windows in shared memory (two barriers, three times the instructions) 64 x 96 x 55 x 55, 3 x 3, took 78 us in a single
// call behind a flush of L2 (now 49 so, and 41.6 at 4.0 TB/s one behind the other), 128 x 256 x 13 x 13 57 (23), 64 x 512 x 14 x
// 14, 2 x 2, 57 (21).
template <int WIN>
__global__ void __launch_bounds__(kThreads, 4) maxpool_bwd_columns(int total, int h, int w, FastDiv div_items, int P, int Q, int band_rows, bool pairs,
                                                                   const float* __restrict__ dy, const float* __restrict__ x, float* __restrict__ dx) {
    constexpr int NEW = WIN == 3 ? 31 : 32, UNROLL = 4;
    const int lane = threadIdx.x & 31;
    const long long first = (static_cast<long long>(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5)) * NEW;
    if (first >= total) return;                                  // a whole warp
    const long long item = first + lane - (WIN == 3 ? 1 : 0);
    const bool valid = item >= 0 && item < total, out = valid && (WIN == 2 || lane > 0);
    uint32_t plane = 0, q = 0;
    if (valid) div_items.divmod(static_cast<uint32_t>(item), plane, q);
    const bool has = valid && static_cast<int>(q) < Q;           // there is a window in these columns
    const float* xp = x + static_cast<size_t>(plane) * h * w + 2 * q;
    const float* gp = dy + static_cast<size_t>(plane) * P * Q + q;
    float* op = dx + static_cast<size_t>(plane) * h * w + 2 * q;
    const bool second = 2 * static_cast<int>(q) + 1 < w;
    const int rows = (h + 1) / 2, p_beg = blockIdx.y * band_rows, p_end = min(rows, p_beg + band_rows);

    auto row_max = [](const float* v, float* m, int* b) {
        *m = -INFINITY; *b = 0;
#pragma unroll
        for (int j = 0; j < WIN; ++j) if (v[j] > *m) { *m = v[j]; *b = j; }
    };
    float carry_m = -INFINITY, up_g = 0.0f, up_left_g = 0.0f;    // the window above, and the one to its left
    int carry_b = 0, up_k = -1, up_left_k = -1;
    if (WIN == 3) {
        // the window above the band, whose last row begins the band
        if (has && p_beg > 0 && p_beg - 1 < P) {
            const float* r = xp + static_cast<size_t>(2 * p_beg - 2) * w;
            float v[3][3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) v[a][b] = __ldg(r + a * w + b);
            up_g = __ldg(gp + static_cast<size_t>(p_beg - 1) * Q);
            float m, mm;
            int b;
            row_max(v[0], &m, &up_k);
            row_max(v[1], &mm, &b);
            if (mm > m) { m = mm; up_k = 3 + b; }
            row_max(v[2], &carry_m, &carry_b);
            if (carry_m > m) up_k = 6 + carry_b;
        } else if (has && p_beg == 0) {
            const float v[3] = {__ldg(xp), __ldg(xp + 1), __ldg(xp + 2)};
            row_max(v, &carry_m, &carry_b);
        }
        up_left_k = __shfl_up_sync(0xffffffffu, up_k, 1);
        up_left_g = __shfl_up_sync(0xffffffffu, up_g, 1);
        if (q == 0) up_left_k = -1;
    }
    for (int p0 = p_beg; p0 < p_end; p0 += UNROLL) {
        float v[UNROLL][2][WIN], g[UNROLL];                      // rows 2 p + 1, 2 p + 2 (3 x 3) or 2 p, 2 p + 1 of window row p
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int p = p0 + u;
            const bool live = has && p < P && p < p_end;
            const float* r = xp + static_cast<size_t>(2 * p + (WIN == 3 ? 1 : 0)) * w;
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < WIN; ++b) v[u][a][b] = live ? __ldg(r + a * w + b) : 0.0f;
            g[u] = live ? __ldg(gp + static_cast<size_t>(p) * Q) : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int p = p0 + u;
            if (p >= p_end) break;
            float m, mm;
            int k, b;
            if (WIN == 3) {
                m = carry_m; k = carry_b;
                row_max(v[u][0], &mm, &b);
                if (mm > m) { m = mm; k = 3 + b; }
                row_max(v[u][1], &carry_m, &carry_b);
                if (carry_m > m) k = 6 + carry_b;
            } else {
                row_max(v[u][0], &m, &k);
                row_max(v[u][1], &mm, &b);
                if (mm > m) k = 2 + b;
            }
            if (!has || p >= P) k = -1;
            float o00 = 0.0f, o01 = 0.0f, o10 = 0.0f, o11 = 0.0f;
            if (WIN == 3) {
                int left_k = __shfl_up_sync(0xffffffffu, k, 1);
                const float left_g = __shfl_up_sync(0xffffffffu, g[u], 1);
                if (q == 0) left_k = -1;
                if (up_left_k == 8) o00 += up_left_g;
                if (up_k == 6) o00 += up_g;
                if (up_k == 7) o01 += up_g;
                if (left_k == 2) o00 += left_g;
                if (left_k == 5) o10 += left_g;
                up_k = k; up_g = g[u];
                up_left_k = left_k; up_left_g = left_g;
            }
            if (k == 0) o00 += g[u];
            if (k == 1) o01 += g[u];
            if (k == WIN) o10 += g[u];
            if (k == WIN + 1) o11 += g[u];
            if (out) {
                float* o = op + static_cast<size_t>(2 * p) * w;
                const bool below = 2 * p + 1 < h;
                if (pairs) {
                    *reinterpret_cast<float2*>(o) = make_float2(o00, o01);
                    if (below) *reinterpret_cast<float2*>(o + w) = make_float2(o10, o11);
                } else {
                    o[0] = o00;
                    if (second) o[1] = o01;
                    if (below) {
                        o[w] = o10;
                        if (second) o[w + 1] = o11;
                    }
                }
            }
        }
    }
}

// Any window.  A block takes a band of dx rows of one plane: the x rows that the band's windows cover go to shared memory,
// one thread per window finds the window's first maximum there and leaves its place and dy, and one thread per input
// element adds up the few windows around it that point to it, in scan order.  x and dy are read and dx is written once, in full
// rows, with no atomics and no pre-zeroed dx; the sums come out the same every time.
__global__ void __launch_bounds__(kThreads) maxpool_bwd_band(int bands, int band_rows, int h, FastDiv div_w, int P, FastDiv div_q, int wh, int ww,
                                                             int sh, int sw, const float* __restrict__ dy,
                                                             const float* __restrict__ x, float* __restrict__ dx) {
    extern __shared__ float smem[];
    const int w = div_w.d, Q = div_q.d;
    const unsigned plane = blockIdx.x / bands, band = blockIdx.x - plane * bands;
    const int r0 = band * band_rows, r1 = min(h, r0 + band_rows);
    // windows that reach rows r0 .. r1 - 1, and the rows they cover
    const int p0 = r0 < wh ? 0 : (r0 - wh) / sh + 1, p1 = min(P, (r1 - 1) / sh + 1);
    const int np = max(0, p1 - p0);
    const int x0 = p0 * sh, xrows = np > 0 ? (np - 1) * sh + wh : 0;
    const float* xp = x + static_cast<size_t>(plane) * h * w;
    const float* dyp = dy + static_cast<size_t>(plane) * P * Q;
    float* dxp = dx + static_cast<size_t>(plane) * h * w;
    float* xs = smem;                                           // [xrows][w]
    const int rows_max = band_rows / sh + (wh + sh - 1) / sh + 1;        // windows rows of any band
    float2* win = reinterpret_cast<float2*>(xs + (((rows_max - 1) * sh + wh) * w + 1) / 2 * 2);    // [np][Q] dy, place of the maximum
    // dy first: its loads are in flight together with those of x
#pragma unroll 2
    for (int i = threadIdx.x; i < np * Q; i += kThreads) win[i].x = __ldg(dyp + p0 * Q + i);
#pragma unroll 8
    for (int i = threadIdx.x; i < xrows * w; i += kThreads) xs[i] = __ldg(xp + x0 * w + i);
    __syncthreads();
    for (int i = threadIdx.x; i < np * Q; i += blockDim.x) {
        uint32_t p, q;
        div_q.divmod(i, p, q);
        const int o = p * sh * w + q * sw;
        float m = -INFINITY;
        int best = 0;                                           // position inside the window: row * ww + column
        for (int a = 0; a < wh; ++a)
            for (int b = 0; b < ww; ++b) {
                const float v = xs[o + a * w + b];
                if (v > m) { m = v; best = a * ww + b; }
            }
        win[i].y = __int_as_float(best);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < (r1 - r0) * w; i += blockDim.x) {
        uint32_t row, col;
        div_w.divmod(i, row, col);
        const int iw = col, ih = r0 + row;
        const int pl = max(p0, ih < wh ? 0 : (ih - wh) / sh + 1), ph = min(p1 - 1, ih / sh);
        const int ql = iw < ww ? 0 : (iw - ww) / sw + 1, qh = min(Q - 1, iw / sw);
        float g = 0.0f;
        for (int p = pl; p <= ph; ++p)
            for (int q = ql; q <= qh; ++q) {
                const float2 v = win[(p - p0) * Q + q];
                if (__float_as_int(v.y) == (ih - p * sh) * ww + iw - q * sw) g += v.x;
            }
        dxp[r0 * w + i] = g;
    }
}

// Windows too large for a band in shared memory: one thread per window finds its first maximum and adds dy there; dx is
// zeroed beforehand.  An input element's contributions are added in arbitrary order.
__global__ void __launch_bounds__(kThreads) maxpool_bwd_scatter(int planes, int h, int w, int P, int Q, int wh, int ww,
                                                                int sh, int sw, const float* __restrict__ dy,
                                                                const float* __restrict__ x, float* __restrict__ dx) {
    const size_t total = static_cast<size_t>(planes) * P * Q;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const int q = static_cast<int>(idx % Q);
        const size_t t = idx / Q;
        const int p = static_cast<int>(t % P);
        const size_t plane = t / P;
        const size_t origin = plane * h * w + static_cast<size_t>(p * sh) * w + q * sw;
        float m = -INFINITY;
        int best = 0;
        for (int i = 0; i < wh; ++i)
            for (int j = 0; j < ww; ++j) {
                const float v = x[origin + i * w + j];
                if (v > m) { m = v; best = i * w + j; }
            }
        atomicAdd(dx + origin + best, dy[idx]);
    }
}

__global__ void __launch_bounds__(kThreads) maxpool_bwd_2x2(size_t pairs, int w, int Qh, const float* __restrict__ dy,
                                                            const float* __restrict__ x, float* __restrict__ dx) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < pairs; idx += stride) {
        const size_t row = idx / Qh;
        const int qp = static_cast<int>(idx - row * Qh);
        const size_t off = row * 2 * w + qp * 4;
        const float4 a = __ldcs(reinterpret_cast<const float4*>(x + off));
        const float4 b = __ldcs(reinterpret_cast<const float4*>(x + off + w));
        const float2 g = __ldcs(reinterpret_cast<const float2*>(dy) + idx);
        // first maximum in scan order (row 0: x,y ; row 1: x,y) of each 2x2 window
        int s0 = 0; float m0 = -INFINITY;
        if (a.x > m0) { m0 = a.x; s0 = 0; } if (a.y > m0) { m0 = a.y; s0 = 1; }
        if (b.x > m0) { m0 = b.x; s0 = 2; } if (b.y > m0) { m0 = b.y; s0 = 3; }
        int s1 = 0; float m1 = -INFINITY;
        if (a.z > m1) { m1 = a.z; s1 = 0; } if (a.w > m1) { m1 = a.w; s1 = 1; }
        if (b.z > m1) { m1 = b.z; s1 = 2; } if (b.w > m1) { m1 = b.w; s1 = 3; }
        float4 ra, rb;
        ra.x = s0 == 0 ? g.x : 0.0f; ra.y = s0 == 1 ? g.x : 0.0f; rb.x = s0 == 2 ? g.x : 0.0f; rb.y = s0 == 3 ? g.x : 0.0f;
        ra.z = s1 == 0 ? g.y : 0.0f; ra.w = s1 == 1 ? g.y : 0.0f; rb.z = s1 == 2 ? g.y : 0.0f; rb.w = s1 == 3 ? g.y : 0.0f;
        *reinterpret_cast<float4*>(dx + off) = ra;
        *reinterpret_cast<float4*>(dx + off + w) = rb;
    }
}

// ---------------------------------------------------------------- softmax (one warp per row)
__device__ __forceinline__ double warp_sum_f64(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the block of one double per thread, in every thread; `part` holds one per warp.
__device__ __forceinline__ double block_sum_f64(double v, double* part) {
    v = warp_sum_f64(v);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.0;
    for (unsigned w = 0; w < blockDim.x >> 5; ++w) v += part[w];
    return v;
}

// The row sums are carried in double: with saturated outputs (y close to one-hot) the backward
// expression dy - sum(dy*y) cancels almost completely, and a float sum would leave only a few
// correct bits.  The tensors stay fp32; the extra cost on N x 1000 elements is nil.
//
// A block per row, the row in registers (rows of up to 8 * 1024 values; longer ones are read again in every pass: with
// 256 threads at most, 256 rows of 4000 took 5.2 us forward and 4.2 backward; now 3.6 and 3.2).  These calls are bound by
// latency: with one warp per row and a dependent loop per pass, 64 rows of 1000 took 7.2 us forward and 5.2 backward; now 2.1
// and 1.8.  The followers are let in late, when the row is summed: let in at the start, their blocks take slots beside rows
// that still load (256 x 4000 with 256 threads: 7.5 us forward instead of 5.2).
constexpr int ROW_VALUES = 8, ROW_THREADS = 1024;

// f(j, p[j], q[j]) for this thread's columns behind the register pass, ROW_VALUES loads in flight at a time: through plain
// pointers the compiler would not fetch ahead of the stores that f may do.
template <class F>
__device__ __forceinline__ void beyond_registers(int cols, const float* p, const float* q, F f) {
    const int t = threadIdx.x, nt = blockDim.x;
    for (int j0 = t + ROW_VALUES * nt; j0 < cols; j0 += ROW_VALUES * nt) {
        float a[ROW_VALUES], b[ROW_VALUES];
#pragma unroll
        for (int u = 0; u < ROW_VALUES; ++u) {
            const int j = j0 + u * nt;
            a[u] = j < cols ? p[j] : 0.0f;
            b[u] = j < cols && q != p ? q[j] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < ROW_VALUES; ++u)
            if (j0 + u * nt < cols) f(j0 + u * nt, a[u], b[u]);
    }
}

__global__ void __launch_bounds__(ROW_THREADS) softmax_fwd_kernel(int cols, const float* x, float* y) {
    __shared__ float part_m[ROW_THREADS / 32];
    __shared__ double part_s[ROW_THREADS / 32];
    tc::after_predecessor();
    const float* xr = x + static_cast<size_t>(blockIdx.x) * cols;
    float* yr = y + static_cast<size_t>(blockIdx.x) * cols;
    const int t = threadIdx.x, nt = blockDim.x;
    float v[ROW_VALUES];
    float m = -INFINITY;
#pragma unroll
    for (int u = 0; u < ROW_VALUES; ++u) { v[u] = t + u * nt < cols ? xr[t + u * nt] : -INFINITY; }
#pragma unroll
    for (int u = 0; u < ROW_VALUES; ++u) m = fmaxf(m, v[u]);
    beyond_registers(cols, xr, xr, [&](int, float a, float) { m = fmaxf(m, a); });
    m = warp_max(m);
    if ((t & 31) == 0) part_m[t >> 5] = m;
    __syncthreads();
    m = part_m[0];
    for (int w = 1; w < nt >> 5; ++w) m = fmaxf(m, part_m[w]);
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < ROW_VALUES; ++u)
        if (t + u * nt < cols) { v[u] = expf(v[u] - m); s += static_cast<double>(v[u]); }
    beyond_registers(cols, xr, xr, [&](int, float a, float) { s += static_cast<double>(expf(a - m)); });
    const double inv = 1.0 / block_sum_f64(s, part_s);
    tc::follow_up();
#pragma unroll
    for (int u = 0; u < ROW_VALUES; ++u)
        if (t + u * nt < cols) yr[t + u * nt] = static_cast<float>(static_cast<double>(v[u]) * inv);
    beyond_registers(cols, xr, xr, [&](int j, float a, float) { yr[j] = static_cast<float>(static_cast<double>(expf(a - m)) * inv); });
}

__global__ void __launch_bounds__(ROW_THREADS) softmax_bwd_kernel(int cols, const float* y, const float* dy, float* dx) {
    __shared__ double part_s[ROW_THREADS / 32];
    tc::after_predecessor();
    const size_t row = static_cast<size_t>(blockIdx.x) * cols;
    const int t = threadIdx.x, nt = blockDim.x;
    float a[ROW_VALUES], g[ROW_VALUES];
    double dot = 0.0;
#pragma unroll
    for (int u = 0; u < ROW_VALUES; ++u) {
        const int j = t + u * nt;
        a[u] = j < cols ? y[row + j] : 0.0f;
        g[u] = j < cols ? dy[row + j] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < ROW_VALUES; ++u)
        if (t + u * nt < cols) dot += static_cast<double>(a[u]) * static_cast<double>(g[u]);
    beyond_registers(cols, y + row, dy + row, [&](int, float p, float q) { dot += static_cast<double>(p) * static_cast<double>(q); });
    dot = block_sum_f64(dot, part_s);
    tc::follow_up();
#pragma unroll
    for (int u = 0; u < ROW_VALUES; ++u)
        if (t + u * nt < cols) dx[row + t + u * nt] = static_cast<float>(static_cast<double>(a[u]) * (static_cast<double>(g[u]) - dot));
    beyond_registers(cols, y + row, dy + row, [&](int j, float p, float q) {
        dx[row + j] = static_cast<float>(static_cast<double>(p) * (static_cast<double>(q) - dot));
    });
}

// ---------------------------------------------------------------- loss (one cluster)
// A warp per row, the rows dealt to the warps of up to eight blocks; the blocks' sums meet through distributed shared
// memory in rank order.  One block of 32 warps took 11.1 us for 64 x 1000 (two rows after another per warp, 32 dependent
// trips each), 8 x 512 threads 4.2.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) loss_kernel(int rows, int cols, const float* y, const float* label, double* out2) {
    __shared__ double s_sq[THREADS / 32], s_ce[THREADS / 32];
    __shared__ double block[2];
    tc::follow_up();
    tc::after_predecessor();
    cg::cluster_group cluster = cg::this_cluster();
    double sq = 0.0, ce = 0.0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    for (int r = blockIdx.x + gridDim.x * warp; r < rows; r += gridDim.x * nwarps) {
        const float* yr = y + static_cast<size_t>(r) * cols;
        const float* tr = label + static_cast<size_t>(r) * cols;
        float best = -INFINITY; int arg = 0x7fffffff;
        for (int j0 = lane; j0 < cols; j0 += 32 * ROW_VALUES) {
            float a[ROW_VALUES], b[ROW_VALUES];
#pragma unroll
            for (int u = 0; u < ROW_VALUES; ++u) {
                const int j = j0 + 32 * u;
                a[u] = j < cols ? yr[j] : 0.0f;
                b[u] = j < cols ? tr[j] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < ROW_VALUES; ++u) {
                const double d = static_cast<double>(a[u]) - static_cast<double>(b[u]);
                sq += d * d;                                   // out of range: 0 - 0
                if (j0 + 32 * u < cols && b[u] > best) { best = b[u]; arg = j0 + 32 * u; }
            }
        }
        // first index of the maximum label across the warp
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
            if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
        }
        if (lane == 0) {
            const double p = arg < cols ? yr[arg] : 0.0;       // no maximum: a row of NaN labels
            ce += -log(p > 1e-30 ? p : 1e-30);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
        ce += __shfl_xor_sync(0xffffffffu, ce, o);
    }
    if (lane == 0) { s_sq[warp] = sq; s_ce[warp] = ce; }
    __syncthreads();
    if (threadIdx.x < 2) {
        const double* s = threadIdx.x == 0 ? s_sq : s_ce;
        double a = 0.0;
        for (int i = 0; i < nwarps; ++i) a += s[i];
        block[threadIdx.x] = a;
    }
    cluster.sync();
    if (cluster.block_rank() == 0 && threadIdx.x < 2) {
        double a = 0.0;
        for (unsigned r = 0; r < cluster.num_blocks(); ++r) a += *cluster.map_shared_rank(&block[threadIdx.x], r);
        out2[threadIdx.x] = (threadIdx.x == 0 ? 0.5 * a : a) / rows;
    }
    cluster.sync();
}

// ---------------------------------------------------------------- cross-channel LRN
// One thread per (n, spatial position); the channel loop keeps a sliding window of squares so
// every x is read once from DRAM (neighbouring threads read neighbouring positions).
__global__ void __launch_bounds__(kThreads) lrn_fwd_kernel(int n, int c, int hw, int win, float alpha_over_n, float beta,
                                                           float k, const float* __restrict__ x, float* __restrict__ y) {
    const size_t total = static_cast<size_t>(n) * hw;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    const int half = win / 2;
    for (size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const size_t in = idx / hw;
        const size_t base = in * c * hw + (idx - in * hw);
        float ss = 0.0f;
        for (int j = 0; j < half && j < c; ++j) { const float v = x[base + static_cast<size_t>(j) * hw]; ss = fmaf(v, v, ss); }
        for (int ic = 0; ic < c; ++ic) {
            if (ic + half < c) { const float v = x[base + static_cast<size_t>(ic + half) * hw]; ss = fmaf(v, v, ss); }
            if (ic - half - 1 >= 0) { const float v = x[base + static_cast<size_t>(ic - half - 1) * hw]; ss = fmaf(-v, v, ss); }
            const float scale = fmaf(alpha_over_n, fmaxf(ss, 0.0f), k);
            y[base + static_cast<size_t>(ic) * hw] = x[base + static_cast<size_t>(ic) * hw] * powf(scale, -beta);
        }
    }
}

__global__ void __launch_bounds__(kThreads) lrn_bwd_kernel(int n, int c, int hw, int win, float alpha_over_n, float beta,
                                                           float k, const float* __restrict__ x, const float* __restrict__ y,
                                                           const float* __restrict__ dy, float* __restrict__ dx) {
    const size_t total = static_cast<size_t>(n) * hw;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    const int half = win / 2;
    for (size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const size_t in = idx / hw;
        const size_t base = in * c * hw + (idx - in * hw);
        // dx_i = dy_i * s_i^-beta - 2*alpha*beta/n * x_i * sum_{j: |i-j|<=half} dy_j*y_j/s_j
        for (int ic = 0; ic < c; ++ic) {
            const int lo = ic - half < 0 ? 0 : ic - half, hi = ic + half >= c ? c - 1 : ic + half;
            float t = 0.0f, s_i = k;
            for (int j = lo; j <= hi; ++j) {
                const int l2 = j - half < 0 ? 0 : j - half, h2 = j + half >= c ? c - 1 : j + half;
                float ss = 0.0f;
                for (int m = l2; m <= h2; ++m) { const float v = x[base + static_cast<size_t>(m) * hw]; ss = fmaf(v, v, ss); }
                const float sj = fmaf(alpha_over_n, ss, k);
                if (j == ic) s_i = sj;
                t += dy[base + static_cast<size_t>(j) * hw] * y[base + static_cast<size_t>(j) * hw] / sj;
            }
            const size_t o = base + static_cast<size_t>(ic) * hw;
            dx[o] = dy[o] * powf(s_i, -beta) - 2.0f * alpha_over_n * beta * x[o] * t;
        }
    }
}

// s^-beta and, where asked for, 1 / s, for the scale s >= k > 0 of a position.  beta = 0.75 (AlexNet's, and the default of
// the callers) takes two square roots instead of powf: r = s^-1/2, s^-3/4 = r * sqrt(r), 1 / s = r * r, each within a few
// units in the last place like powf itself.
template <bool BETA34>
__device__ __forceinline__ float lrn_pow(float s, float beta, float* inv_s) {
    if (BETA34) {
        const float r = rsqrtf(s);
        if (inv_s) *inv_s = r * r;
        return r * sqrtf(r);
    }
    if (inv_s) *inv_s = 1.0f / s;
    return powf(s, -beta);
}

// Window of 5 (the AlexNet setting).  Bound by memory: forward reads x and writes y, backward reads x and dy and writes dx.
// A thread takes LRN_CH channels of one position; their x (with two neighbours on either side, for backward four) is loaded
// at once, so the loads of a thread are in flight together and there are c / LRN_CH times as many threads as positions;
// adjacent chunks of a block of positions sit in one block, so the overlap is read from L1.  One thread per position,
// walking all channels with one load in flight and a powf per channel, took 136.8 us forward and 242.7 backward for
// 64 x 96 x 55 x 55 (1.09 and 0.92 TB/s); now 35.4 and 57.3 (4.2 and 3.9 TB/s).
constexpr int LRN_CH = 16, LRN_POS = 64, LRN_CHUNKS = 4;
template <bool BETA34>
__global__ void __launch_bounds__(LRN_POS * LRN_CHUNKS) lrn_fwd_win5_kernel(int c, int hw, float alpha_over_n, float beta, float k,
                                                                            const float* __restrict__ x, float* __restrict__ y) {
    const int pos = blockIdx.x * LRN_POS + threadIdx.x, c0 = (blockIdx.y * LRN_CHUNKS + threadIdx.y) * LRN_CH;
    if (pos >= hw || c0 >= c) return;
    const size_t base = static_cast<size_t>(blockIdx.z) * c * hw + pos;
    float v[LRN_CH + 4];
#pragma unroll
    for (int j = 0; j < LRN_CH + 4; ++j) {
        const int ch = c0 + j - 2;
        v[j] = ch >= 0 && ch < c ? __ldg(x + base + static_cast<size_t>(ch) * hw) : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < LRN_CH; ++j) {
        if (c0 + j >= c) break;
        const float ss = (v[j] * v[j] + v[j + 1] * v[j + 1]) + (v[j + 2] * v[j + 2] + v[j + 3] * v[j + 3]) + v[j + 4] * v[j + 4];
        y[base + static_cast<size_t>(c0 + j) * hw] = v[j + 2] * lrn_pow<BETA34>(fmaf(alpha_over_n, ss, k), beta, nullptr);
    }
}

// dx_i = dy_i * s_i^-beta - 2*alpha*beta/n * x_i * sum_{|j-i|<=2} t_j with t_j = dy_j * y_j / s_j.  y_j = x_j * s_j^-beta is
// formed again from x, which is read anyway: one tensor less to read.
template <bool BETA34>
__global__ void __launch_bounds__(LRN_POS * LRN_CHUNKS) lrn_bwd_win5_kernel(int c, int hw, float alpha_over_n, float beta, float k,
                                                                            const float* __restrict__ x, const float* __restrict__ dy,
                                                                            float* __restrict__ dx) {
    const int pos = blockIdx.x * LRN_POS + threadIdx.x, c0 = (blockIdx.y * LRN_CHUNKS + threadIdx.y) * LRN_CH;
    if (pos >= hw || c0 >= c) return;
    const size_t base = static_cast<size_t>(blockIdx.z) * c * hw + pos;
    float v[LRN_CH + 8], g[LRN_CH + 4];
#pragma unroll
    for (int j = 0; j < LRN_CH + 8; ++j) {
        const int ch = c0 + j - 4;
        v[j] = ch >= 0 && ch < c ? __ldg(x + base + static_cast<size_t>(ch) * hw) : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < LRN_CH + 4; ++j) {
        const int ch = c0 + j - 2;
        g[j] = ch >= 0 && ch < c ? __ldg(dy + base + static_cast<size_t>(ch) * hw) : 0.0f;
    }
    const float f = 2.0f * alpha_over_n * beta;
    float t[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, pw[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < LRN_CH + 4; ++j) {                      // channel c0 + j - 2: x at v[j + 2], dy at g[j]
        const float ss = (v[j] * v[j] + v[j + 1] * v[j + 1]) + (v[j + 2] * v[j + 2] + v[j + 3] * v[j + 3]) + v[j + 4] * v[j + 4];
        float inv;
        pw[0] = pw[1]; pw[1] = pw[2];
        pw[2] = lrn_pow<BETA34>(fmaf(alpha_over_n, ss, k), beta, &inv);
        t[0] = t[1]; t[1] = t[2]; t[2] = t[3]; t[3] = t[4];
        t[4] = g[j] * (v[j + 2] * pw[2]) * inv;                 // 0 outside the tensor: dy is
        if (j >= 4 && c0 + j - 4 < c)                           // channel i = c0 + j - 4
            dx[base + static_cast<size_t>(c0 + j - 4) * hw] = g[j - 2] * pw[0] - f * v[j] * (((t[0] + t[1]) + (t[2] + t[3])) + t[4]);
    }
}

}  // namespace
}  // namespace vdnn

using namespace vdnn;

extern "C" {

int vdnn_relu_fwd(size_t count, const float* x, float* y, void* stream) {
    if (!x || !y) return VDNN_ERR_BAD_ARG;
    if (count == 0) return VDNN_OK;
    const size_t n4 = (aligned16(x) && aligned16(y)) ? count / 4 : 0;
    relu_fwd_kernel<<<stream_grid(n4 ? n4 : count, 4), kThreads, 0, as_stream(stream)>>>(n4, count, x, y);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_relu_bwd(size_t count, const float* y, const float* dy, const float* x, float* dx, void* stream) {
    (void)y;
    if (!dy || !x || !dx) return VDNN_ERR_BAD_ARG;
    if (count == 0) return VDNN_OK;
    const size_t n4 = (aligned16(x) && aligned16(dy) && aligned16(dx)) ? count / 4 : 0;
    relu_bwd_kernel<<<stream_grid(n4 ? n4 : count, 2), kThreads, 0, as_stream(stream)>>>(n4, count, dy, x, dx);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_activation_fwd(int mode, size_t count, const float* x, float* y, void* stream) {
    if (mode == VDNN_ACT_RELU) return vdnn_relu_fwd(count, x, y, stream);
    if (mode != VDNN_ACT_TANH && mode != VDNN_ACT_SIGMOID) return VDNN_ERR_UNSUPPORTED;
    if (!x || !y) return VDNN_ERR_BAD_ARG;
    if (count == 0) return VDNN_OK;
    const size_t n4 = (aligned16(x) && aligned16(y)) ? count / 4 : 0;
    const int grid = stream_grid(n4 ? n4 : count, 1);
    if (mode == VDNN_ACT_TANH) act_fwd_kernel<VDNN_ACT_TANH><<<grid, kThreads, 0, as_stream(stream)>>>(n4, count, x, y);
    else act_fwd_kernel<VDNN_ACT_SIGMOID><<<grid, kThreads, 0, as_stream(stream)>>>(n4, count, x, y);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_activation_bwd(int mode, size_t count, const float* y, const float* dy, const float* x, float* dx, void* stream) {
    if (mode == VDNN_ACT_RELU) return vdnn_relu_bwd(count, y, dy, x, dx, stream);
    if (mode != VDNN_ACT_TANH && mode != VDNN_ACT_SIGMOID) return VDNN_ERR_UNSUPPORTED;
    if (!y || !dy || !dx) return VDNN_ERR_BAD_ARG;
    if (count == 0) return VDNN_OK;
    const size_t n4 = (aligned16(y) && aligned16(dy) && aligned16(dx)) ? count / 4 : 0;
    const int grid = stream_grid(n4 ? n4 : count, 1);
    if (mode == VDNN_ACT_TANH) act_bwd_kernel<VDNN_ACT_TANH><<<grid, kThreads, 0, as_stream(stream)>>>(n4, count, y, dy, dx);
    else act_bwd_kernel<VDNN_ACT_SIGMOID><<<grid, kThreads, 0, as_stream(stream)>>>(n4, count, y, dy, dx);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_sub(size_t count, const float* a, const float* b, float* out, void* stream) {
    if (!a || !b || !out) return VDNN_ERR_BAD_ARG;
    if (count == 0) return VDNN_OK;
    const size_t n4 = (aligned16(a) && aligned16(b) && aligned16(out)) ? count / 4 : 0;
    VDNN_CUDA(tc::launch_early(sub_kernel, dim3(stream_grid(n4 ? n4 : count, 1)), kThreads, 0, as_stream(stream), n4, count, a, b, out));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_axpy(size_t count, float alpha, const float* g, float* w, void* stream) {
    if (!g || !w) return VDNN_ERR_BAD_ARG;
    if (count == 0) return VDNN_OK;
    const size_t n4 = (aligned16(g) && aligned16(w)) ? count / 4 : 0;
    axpy_kernel<<<stream_grid(n4 ? n4 : count, 1), kThreads, 0, as_stream(stream)>>>(n4, count, alpha, g, w);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_fill(size_t count, float value, float* dst, void* stream) {
    if (!dst) return VDNN_ERR_BAD_ARG;
    if (count == 0) return VDNN_OK;
    fill_kernel<<<stream_grid(count, 1), kThreads, 0, as_stream(stream)>>>(count, value, dst);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_add_bias(int n, int k, int pq, float alpha, const float* bias, float* y, void* stream) {
    if (!bias || !y || n <= 0 || k <= 0 || pq <= 0) return VDNN_ERR_BAD_ARG;
    const size_t image = static_cast<size_t>(k) * pq;
    const int per_launch = images_per_launch(n, image);      // 32-bit item indexes inside a launch
    if (per_launch < 1) {                                    // an image of 2^31 values or more: plane by plane
        for (size_t plane = 0; plane < static_cast<size_t>(n) * k; ++plane) {
            const int st = vdnn_add_bias(1, 1, pq, alpha, bias + plane % k, y + plane * pq, stream);
            if (st != VDNN_OK) return st;
        }
        return VDNN_OK;
    }
    for (int n0 = 0; n0 < n; n0 += per_launch) {
        const size_t total = static_cast<size_t>(n - n0 < per_launch ? n - n0 : per_launch) * image;
        float* yp = y + static_cast<size_t>(n0) * image;
        cudaStream_t s = as_stream(stream);
        if (pq % 4 == 0 && aligned16(yp)) {
            const uint32_t items = static_cast<uint32_t>(total / 4);
            add_bias_kernel<BIAS_PLANE4><<<stream_grid(items, 1), kThreads, 0, s>>>(items, FastDiv(pq / 4), FastDiv(k), alpha, bias, yp);
        } else if (pq == 1 && k % 4 == 0 && aligned16(yp) && aligned16(bias)) {
            const uint32_t items = static_cast<uint32_t>(total / 4);
            add_bias_kernel<BIAS_ROW4><<<stream_grid(items, 1), kThreads, 0, s>>>(items, FastDiv(1), FastDiv(k / 4), alpha, bias, yp);
        } else {
            add_bias_kernel<BIAS_SCALAR><<<stream_grid(total, 1), kThreads, 0, s>>>(static_cast<uint32_t>(total), FastDiv(pq), FastDiv(k), alpha, bias, yp);
        }
        VDNN_LAUNCHED();
    }
    return VDNN_OK;
}

int vdnn_conv_bwd_bias(int n, int k, int pq, float alpha, const float* dy, float beta, float* db, void* stream) {
    if (!dy || !db || n <= 0 || k <= 0 || pq <= 0) return VDNN_ERR_BAD_ARG;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    cfg.stream = as_stream(stream);
    // blocks per channel (group): enough to occupy every SM twice over, but no block with less than four loads a thread
    auto blocks_of = [&](int groups, size_t items, int threads) {
        int s = 1;
        while (s < 8 && static_cast<long long>(groups) * s < 2LL * sm_count() && items / (2 * s) >= static_cast<size_t>(4 * threads)) s *= 2;
        return s;
    };
    if (pq < 32) {
        const int groups = ceil_div(k, 32 / pq);
        const int slices = blocks_of(groups, static_cast<size_t>(n) * 32, 256);
        cfg.gridDim = dim3(static_cast<unsigned>(slices) * groups); cfg.blockDim = dim3(256);
        attr[0].val.clusterDim.x = slices;
        VDNN_CUDA(cudaLaunchKernelEx(&cfg, bwd_bias_narrow_kernel, n, k, pq, alpha, dy, beta, db));
        VDNN_LAUNCHED();
        return VDNN_OK;
    }
    const bool vec = pq % 4 == 0 && aligned16(dy);
    const uint32_t plane = static_cast<uint32_t>(vec ? pq / 4 : pq);
    const int per_launch = images_per_launch(n, plane);
    for (int n0 = 0; n0 < n; n0 += per_launch) {
        const uint32_t items = static_cast<uint32_t>(n - n0 < per_launch ? n - n0 : per_launch) * plane;
        const int threads = items >= 2048 ? 512 : 128;
        const int slices = blocks_of(k, items, threads);
        cfg.gridDim = dim3(static_cast<unsigned>(slices) * k); cfg.blockDim = dim3(threads);
        attr[0].val.clusterDim.x = slices;
        const float* src = dy + static_cast<size_t>(n0) * k * pq;
        const float b = n0 == 0 ? beta : 1.0f;
        if (vec) VDNN_CUDA(cudaLaunchKernelEx(&cfg, bwd_bias_kernel<4>, items, k, FastDiv(plane), alpha, src, b, db));
        else VDNN_CUDA(cudaLaunchKernelEx(&cfg, bwd_bias_kernel<1>, items, k, FastDiv(plane), alpha, src, b, db));
        VDNN_LAUNCHED();
    }
    return VDNN_OK;
}

int vdnn_pool_out_dims(int h, int w, int win_h, int win_w, int stride_h, int stride_w, int* p, int* q) {
    if (!p || !q || win_h <= 0 || win_w <= 0 || stride_h <= 0 || stride_w <= 0 || h < win_h || w < win_w)
        return VDNN_ERR_BAD_ARG;
    *p = (h - win_h) / stride_h + 1;
    *q = (w - win_w) / stride_w + 1;
    return VDNN_OK;
}

static bool pool_fast_2x2(int h, int w, int wh, int ww, int sh, int sw, const void* a, const void* b, const void* c) {
    return wh == 2 && ww == 2 && sh == 2 && sw == 2 && h % 2 == 0 && w % 4 == 0 && aligned16(a) && aligned16(b) &&
           (c == nullptr || aligned16(c));
}

int vdnn_maxpool_fwd(int n, int c, int h, int w, int win_h, int win_w, int stride_h, int stride_w,
                     const float* x, float* y, void* stream) {
    int P, Q;
    if (!x || !y || n <= 0 || c <= 0) return VDNN_ERR_BAD_ARG;
    if (vdnn_pool_out_dims(h, w, win_h, win_w, stride_h, stride_w, &P, &Q) != VDNN_OK) return VDNN_ERR_BAD_ARG;
    const int planes = n * c;
    if (pool_fast_2x2(h, w, win_h, win_w, stride_h, stride_w, x, y, nullptr)) {
        const size_t pairs = static_cast<size_t>(planes) * P * (Q / 2);
        maxpool_fwd_2x2<<<stream_grid(pairs, 1), kThreads, 0, as_stream(stream)>>>(pairs, w, Q / 2, x, y);
        VDNN_LAUNCHED();
        return VDNN_OK;
    }
    const size_t out_plane = static_cast<size_t>(P) * Q, in_plane = static_cast<size_t>(h) * w;
    const int per_launch = images_per_launch(planes, out_plane);          // 32-bit indexes inside a launch
    if (per_launch < 1) return VDNN_ERR_UNSUPPORTED;
    const FastDiv dp(P), dq(Q);
    for (int p0 = 0; p0 < planes; p0 += per_launch) {
        const uint32_t total = static_cast<uint32_t>((planes - p0 < per_launch ? planes - p0 : per_launch) * out_plane);
        const float* xs = x + p0 * in_plane;
        float* ys = y + p0 * out_plane;
        const int grid = stream_grid(total, 1);
        const int win = win_h == win_w ? win_h : 0;
        if (win == 2) maxpool_fwd_generic<2><<<grid, kThreads, 0, as_stream(stream)>>>(total, h, w, dp, dq, 2, 2, stride_h, stride_w, xs, ys);
        else if (win == 3) maxpool_fwd_generic<3><<<grid, kThreads, 0, as_stream(stream)>>>(total, h, w, dp, dq, 3, 3, stride_h, stride_w, xs, ys);
        else maxpool_fwd_generic<0><<<grid, kThreads, 0, as_stream(stream)>>>(total, h, w, dp, dq, win_h, win_w, stride_h, stride_w, xs, ys);
        VDNN_LAUNCHED();
    }
    return VDNN_OK;
}

int vdnn_maxpool_bwd(int n, int c, int h, int w, int win_h, int win_w, int stride_h, int stride_w,
                     const float* y, const float* dy, const float* x, float* dx, void* stream) {
    (void)y;
    int P, Q;
    if (!dy || !x || !dx || n <= 0 || c <= 0) return VDNN_ERR_BAD_ARG;
    if (vdnn_pool_out_dims(h, w, win_h, win_w, stride_h, stride_w, &P, &Q) != VDNN_OK) return VDNN_ERR_BAD_ARG;
    const int planes = n * c;
    if (pool_fast_2x2(h, w, win_h, win_w, stride_h, stride_w, x, dx, dy)) {
        const size_t pairs = static_cast<size_t>(planes) * P * (Q / 2);
        maxpool_bwd_2x2<<<stream_grid(pairs, 1), kThreads, 0, as_stream(stream)>>>(pairs, w, Q / 2, dy, x, dx);
        VDNN_LAUNCHED();
        return VDNN_OK;
    }
    const int items = (w + 1) / 2, window_rows = (h + 1) / 2;
    if (win_h == win_w && (win_h == 2 || win_h == 3) && stride_h == 2 && stride_w == 2 && static_cast<long long>(planes) * items < 0x7fffffffLL) {
        const int total = planes * items, per_block = (kThreads / 32) * (win_h == 3 ? 31 : 32), blocks = ceil_div(total, per_block);
        // bands of window rows: three waves of blocks, but not less than four rows, of which a band reads one twice
        const int want = ceil_div(3 * 4 * sm_count(), blocks), most = window_rows / 4 > 1 ? window_rows / 4 : 1;
        const int band = ceil_div(window_rows, want < most ? want : most);
        const bool pairs = w % 2 == 0 && (reinterpret_cast<uintptr_t>(dx) & 7u) == 0;
        const dim3 grid(blocks, ceil_div(window_rows, band));
        if (win_h == 3) maxpool_bwd_columns<3><<<grid, kThreads, 0, as_stream(stream)>>>(total, h, w, FastDiv(items), P, Q, band, pairs, dy, x, dx);
        else maxpool_bwd_columns<2><<<grid, kThreads, 0, as_stream(stream)>>>(total, h, w, FastDiv(items), P, Q, band, pairs, dy, x, dx);
        VDNN_LAUNCHED();
        return VDNN_OK;
    }
    // rows of a band: about 16 KB of shared memory, so that a full set of blocks stays resident, but at least two rows
    auto smem_of = [&](int rows) {
        const size_t np = rows / stride_h + (win_h + stride_h - 1) / stride_h + 1;
        return ((((np - 1) * stride_h + win_h) * w + 1) / 2 * 2 + 2 * np * Q) * sizeof(float);
    };
    int band = h;
    while (band > 2 && smem_of(band) > 16 * 1024) band = (band + 1) / 2;
    const size_t smem = smem_of(band);
    const long long blocks = static_cast<long long>(planes) * ceil_div(h, band);
    // a window so large that not even one row's share fits is outside what any network here has
    if (smem <= 200 * 1024 && blocks <= 0x7fffffffLL) {
        const int bands = ceil_div(h, band);
        if (smem > 48 * 1024) VDNN_CUDA(cudaFuncSetAttribute(maxpool_bwd_band, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        maxpool_bwd_band<<<static_cast<unsigned>(blocks), kThreads, smem, as_stream(stream)>>>(bands, band, h, FastDiv(w), P, FastDiv(Q), win_h, win_w, stride_h, stride_w,
                                                                                  dy, x, dx);
    } else {
        VDNN_CUDA(cudaMemsetAsync(dx, 0, static_cast<size_t>(planes) * h * w * sizeof(float), as_stream(stream)));
        const size_t total = static_cast<size_t>(planes) * P * Q;
        maxpool_bwd_scatter<<<stream_grid(total, 1), kThreads, 0, as_stream(stream)>>>(planes, h, w, P, Q, win_h, win_w,
                                                                                       stride_h, stride_w, dy, x, dx);
    }
    VDNN_LAUNCHED();
    return VDNN_OK;
}

// Threads of a softmax block: four values each up to 256 threads, then up to ROW_VALUES each and more threads.
static int softmax_threads(int cols) {
    int t = 32;
    while (t < 256 && t * 4 < cols) t *= 2;
    while (t < ROW_THREADS && t * ROW_VALUES < cols) t *= 2;
    return t;
}

int vdnn_softmax_fwd(int rows, int cols, const float* x, float* y, void* stream) {
    if (!x || !y || rows <= 0 || cols <= 0) return VDNN_ERR_BAD_ARG;
    VDNN_CUDA(tc::launch_early(softmax_fwd_kernel, dim3(rows), softmax_threads(cols), 0, as_stream(stream), cols, x, y));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_softmax_bwd(int rows, int cols, const float* y, const float* dy, float* dx, void* stream) {
    if (!y || !dy || !dx || rows <= 0 || cols <= 0) return VDNN_ERR_BAD_ARG;
    VDNN_CUDA(tc::launch_early(softmax_bwd_kernel, dim3(rows), softmax_threads(cols), 0, as_stream(stream), cols, y, dy, dx));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_loss(int rows, int cols, const float* y, const float* label, double* out2, void* stream) {
    if (!y || !label || !out2 || rows <= 0 || cols <= 0) return VDNN_ERR_BAD_ARG;
    // A warp per row up to 8 * 32 rows.  Fewer warps have more registers for loads in flight and meet sooner, so up to 8 * 16 rows
    // take 512 threads (128 x 1000: 4.6 us, with 1024 5.0; 256 x 1000: 7.5 and 6.6).
    const bool wide = rows > 8 * 16;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = rows >= 8 ? 8 : 1;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    cfg.gridDim = dim3(attr[0].val.clusterDim.x); cfg.blockDim = dim3(wide ? 1024 : 512);
    cfg.stream = as_stream(stream);
    if (wide) VDNN_CUDA(cudaLaunchKernelEx(&cfg, loss_kernel<1024>, rows, cols, y, label, out2));
    else VDNN_CUDA(cudaLaunchKernelEx(&cfg, loss_kernel<512>, rows, cols, y, label, out2));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

// The chunked kernels of the 5-wide window: grid.z carries the images (longer batches go in several launches).
static dim3 lrn_grid(int c, int hw) { return dim3(ceil_div(hw, LRN_POS), ceil_div(c, LRN_CH * LRN_CHUNKS), 1); }
static bool lrn_chunked(int c, int win) { return win == 5 && ceil_div(c, LRN_CH * LRN_CHUNKS) <= 65535; }

int vdnn_lrn_fwd(int n, int c, int hw, int win, float alpha, float beta, float k, const float* x, float* y,
                 void* stream) {
    if (!x || !y || n <= 0 || c <= 0 || hw <= 0 || win <= 0 || win % 2 == 0) return VDNN_ERR_BAD_ARG;
    if (!lrn_chunked(c, win)) {
        lrn_fwd_kernel<<<stream_grid(static_cast<size_t>(n) * hw, 1), kThreads, 0, as_stream(stream)>>>(
            n, c, hw, win, alpha / win, beta, k, x, y);
        VDNN_LAUNCHED();
        return VDNN_OK;
    }
    dim3 grid = lrn_grid(c, hw);
    for (int n0 = 0; n0 < n; n0 += 65535) {
        grid.z = n - n0 < 65535 ? n - n0 : 65535;
        const size_t off = static_cast<size_t>(n0) * c * hw;
        auto kern = beta == 0.75f ? lrn_fwd_win5_kernel<true> : lrn_fwd_win5_kernel<false>;
        kern<<<grid, dim3(LRN_POS, LRN_CHUNKS), 0, as_stream(stream)>>>(c, hw, alpha / win, beta, k, x + off, y + off);
        VDNN_LAUNCHED();
    }
    return VDNN_OK;
}

int vdnn_lrn_bwd(int n, int c, int hw, int win, float alpha, float beta, float k, const float* x, const float* y,
                 const float* dy, float* dx, void* stream) {
    if (!x || !y || !dy || !dx || n <= 0 || c <= 0 || hw <= 0 || win <= 0 || win % 2 == 0) return VDNN_ERR_BAD_ARG;
    if (!lrn_chunked(c, win)) {
        lrn_bwd_kernel<<<stream_grid(static_cast<size_t>(n) * hw, 1), kThreads, 0, as_stream(stream)>>>(
            n, c, hw, win, alpha / win, beta, k, x, y, dy, dx);
        VDNN_LAUNCHED();
        return VDNN_OK;
    }
    dim3 grid = lrn_grid(c, hw);
    for (int n0 = 0; n0 < n; n0 += 65535) {
        grid.z = n - n0 < 65535 ? n - n0 : 65535;
        const size_t off = static_cast<size_t>(n0) * c * hw;
        auto kern = beta == 0.75f ? lrn_bwd_win5_kernel<true> : lrn_bwd_win5_kernel<false>;
        kern<<<grid, dim3(LRN_POS, LRN_CHUNKS), 0, as_stream(stream)>>>(c, hw, alpha / win, beta, k, x + off, dy + off, dx + off);
        VDNN_LAUNCHED();
    }
    return VDNN_OK;
}

int vdnn_offload(void* dst_pinned_h, const void* src, size_t bytes, void* ready_event, void* done_event,
                 void* copy_stream) {
    if (!dst_pinned_h || !src) return VDNN_ERR_BAD_ARG;
    cudaStream_t s = as_stream(copy_stream);
    if (ready_event) VDNN_CUDA(cudaStreamWaitEvent(s, static_cast<cudaEvent_t>(ready_event), 0));
    VDNN_CUDA(cudaMemcpyAsync(dst_pinned_h, src, bytes, cudaMemcpyDeviceToHost, s));
    if (done_event) VDNN_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(done_event), s));
    return VDNN_OK;
}

int vdnn_prefetch(void* dst, const void* src_pinned_h, size_t bytes, void* ready_event, void* done_event,
                  void* copy_stream) {
    if (!dst || !src_pinned_h) return VDNN_ERR_BAD_ARG;
    cudaStream_t s = as_stream(copy_stream);
    if (ready_event) VDNN_CUDA(cudaStreamWaitEvent(s, static_cast<cudaEvent_t>(ready_event), 0));
    VDNN_CUDA(cudaMemcpyAsync(dst, src_pinned_h, bytes, cudaMemcpyHostToDevice, s));
    if (done_event) VDNN_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(done_event), s));
    return VDNN_OK;
}

const char* vdnn_status_string(int status) {
    switch (status) {
    case VDNN_OK: return "VDNN_OK";
    case VDNN_ERR_BAD_ARG: return "VDNN_ERR_BAD_ARG";
    case VDNN_ERR_CUDA: return "VDNN_ERR_CUDA";
    case VDNN_ERR_WORKSPACE: return "VDNN_ERR_WORKSPACE";
    case VDNN_ERR_UNSUPPORTED: return "VDNN_ERR_UNSUPPORTED";
    case VDNN_ERR_OUT_OF_MEMORY: return "VDNN_ERR_OUT_OF_MEMORY";
    case VDNN_ERR_TIMEOUT: return "VDNN_ERR_TIMEOUT";
    case VDNN_ERR_STATE: return "VDNN_ERR_STATE";
    case VDNN_ERR_SCRATCH_LIMIT: return "VDNN_ERR_SCRATCH_LIMIT";
    default: return "VDNN_ERR_UNKNOWN";
    }
}

int vdnn_last_cuda_error(void) { return g_last_cuda_error; }

const char* vdnn_build_info(void) { return "vdnn_b200 0.1 (sm_100a)"; }

}  // extern "C"
