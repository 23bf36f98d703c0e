// C-ABI entry points for the contraction-shaped layers (CONV forward / data gradient / filter
// gradient and SGEMM).  Each call builds the operand views of gemm_operands.cuh over the caller's
// NCHW / KCRS tensors, plans a split along K when the output has too few tiles to fill the GPU,
// and runs the selected engine.  Split results are combined either with fp32 atomics straight
// into the output (MEMORY_OPT: no workspace) or through per-split partial tiles in the caller's
// workspace followed by a fixed-order reduction (PERF_OPT: deterministic).
#include <cuda_pipeline.h>
#include <math.h>
#include <string.h>

#include <type_traits>

#include "common.cuh"
#include "gemm_ffma.cuh"
#include "gemm_tc.cuh"
#include "gemm_dense.cuh"
#include "conv_split16.cuh"
#include "conv_halo.cuh"
#include "dgrad_window.cuh"

namespace vdnn {
namespace {

int g_engine = VDNN_ENGINE_AUTO;
// VDNN_NO_TMA=1 in the environment keeps PERF_OPT forward / data gradient on the gather-fed kernel (A/B measurements).
const bool g_no_tma = []() { const char* v = getenv("VDNN_NO_TMA"); return v && *v && *v != '0'; }();
// VDNN_TMA_WGRAD=0: the PERF_OPT filter gradient stays on the gather-fed kernel (default: TMA-fed where the shape allows).
const bool g_tma_wgrad = []() { const char* v = getenv("VDNN_TMA_WGRAD"); return !(v && *v == '0'); }();

struct SplitPlan { int splits; int k_chunk; };

// Split K so that the grid is as close to two full waves of output tiles as it can get without exceeding them
// (a third, nearly empty wave would cost as much as a full one), keeping at least 64 k per split.
SplitPlan plan_split(int M, int N, int K) {
    const int bn = g_engine == VDNN_ENGINE_FFMA ? 128 : tc::tile_n(N);
    const long tiles = static_cast<long>(ceil_div(M, 128)) * ceil_div(N, bn);
    const int sms = sm_count();
    int splits = 1;
    if (tiles < sms) {
        splits = static_cast<int>((2L * sms) / tiles);
        const int max_by_k = K / 64 > 0 ? K / 64 : 1;
        if (splits > max_by_k) splits = max_by_k;
        if (splits > 1024) splits = 1024;
        if (splits < 1) splits = 1;
    }
    int k_chunk = ceil_div(ceil_div(K, splits), 32) * 32;      // multiple of both engines' k tile
    if (k_chunk < 32) k_chunk = 32;
    SplitPlan p;
    p.k_chunk = k_chunk;
    p.splits = ceil_div(K, k_chunk);
    return p;
}

__global__ void __launch_bounds__(256) scale_dense_kernel(size_t n, float beta, float* __restrict__ out) {
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        out[i] = beta == 0.0f ? 0.0f : beta * out[i];
}

__global__ void __launch_bounds__(256) scale_matrix_kernel(int rows, int cols, int ld, float beta, float* __restrict__ out) {
    for (int j = blockIdx.y; j < cols; j += gridDim.y)
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
            float* p = out + static_cast<size_t>(j) * ld + i;
            *p = beta == 0.0f ? 0.0f : beta * *p;
        }
}

// out[i] = alpha * sum_s partial[s][i] + beta * out[i] in a fixed order.  A block takes 256 / lanes groups of VEC adjacent
// sums; its lanes share a group's splits (lane l adds splits l, l + lanes, ... with four loads in flight) and their parts
// are added in lane order.  With one thread per sum, a layer of few weights and many splits (an image's first filters: 864
// sums of 150 parts) walked its splits one load after another on a handful of SMs: 10 us in a single call; now 4.2, and 2.7
// in a row of calls.
template <int VEC>
__global__ void __launch_bounds__(256) reduce_partials_kernel(size_t n, int splits, int lanes, float alpha, float beta,
                                                              const float* __restrict__ partial, float* __restrict__ out, const int* skip) {
    __shared__ float part[256 * VEC];
    tc::follow_up();
    tc::after_predecessor();
    if (skip && *skip) return;
    const int per_block = 256 / lanes, g = threadIdx.x % per_block, l = threadIdx.x / per_block;
    const size_t i = (static_cast<size_t>(blockIdx.x) * per_block + g) * VEC;
    float acc[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) acc[v] = 0.0f;
    if (i < n) {
        auto add = [&](int s) {
            if (VEC == 4) {
                const float4 p = __ldcs(reinterpret_cast<const float4*>(partial + static_cast<size_t>(s) * n + i));
                acc[0] += p.x; acc[1 % VEC] += p.y; acc[2 % VEC] += p.z; acc[3 % VEC] += p.w;
            } else {
                acc[0] += __ldcs(partial + static_cast<size_t>(s) * n + i);
            }
        };
#pragma unroll 4
        for (int s = l; s < splits; s += lanes) add(s);
    }
    if (lanes > 1) {
#pragma unroll
        for (int v = 0; v < VEC; ++v) part[threadIdx.x * VEC + v] = acc[v];
        __syncthreads();
        if (l == 0)
            for (int k = 1; k < lanes; ++k)
#pragma unroll
                for (int v = 0; v < VEC; ++v) acc[v] += part[(k * per_block + g) * VEC + v];
    }
    if (l == 0 && i < n) {
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
            float r = alpha * acc[v];
            if (beta != 0.0f) r = fmaf(beta, out[i + v], r);
            out[i + v] = r;
        }
    }
}

// skip (may be null): a word on the device that says that there are no partial results.
int reduce_partials(size_t n, int splits, float alpha, float beta, const float* partial, float* out, cudaStream_t stream, const int* skip = nullptr) {
    const bool vec = n % 4 == 0 && ((reinterpret_cast<uintptr_t>(partial) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    const size_t groups = vec ? n / 4 : n;
    // lanes per sum: as many as leave each one two splits, while the grid is below two blocks per SM
    int lanes = 1;
    while (lanes < 32 && 4 * lanes <= splits && ceil_div<size_t>(groups * lanes, 256) < static_cast<size_t>(2 * sm_count())) lanes *= 2;
    const size_t blocks = ceil_div<size_t>(groups * lanes, 256);
    if (blocks > 0x7fffffffu) return VDNN_ERR_UNSUPPORTED;
    if (vec) VDNN_CUDA(tc::launch_early(reduce_partials_kernel<4>, dim3(static_cast<unsigned>(blocks)), 256, 0, stream, n, splits, lanes, alpha, beta, partial, out, skip));
    else VDNN_CUDA(tc::launch_early(reduce_partials_kernel<1>, dim3(static_cast<unsigned>(blocks)), 256, 0, stream, n, splits, lanes, alpha, beta, partial, out, skip));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

// Data gradient for layers with very few input channels (the first layer: C = 3).  As a contraction it has
// N = C columns, which would leave a 128 x 64 tensor-core tile almost empty; here one thread owns one input pixel
// and all its channels, the filter bank sits in shared memory, and dy is read with unit stride across a warp.
constexpr int SMALL_C_MAX = 4;
constexpr size_t SMALL_C_SMEM_MAX = 200 * 1024;
__global__ void __launch_bounds__(256) dgrad_small_c_kernel(int N, int C, int H, int W, int K, int R, int S, int P, int Q,
                                                            int pad_h, int pad_w, int stride_h, int stride_w, float alpha,
                                                            float beta, const float* __restrict__ w,
                                                            const float* __restrict__ dy, float* __restrict__ dx) {
    extern __shared__ float w_s[];                       // [K][C][R*S], as stored
    const int wcount = K * C * R * S;
    for (int i = threadIdx.x; i < wcount; i += blockDim.x) w_s[i] = w[i];
    __syncthreads();
    const int hw = H * W, pq = P * Q, rs = R * S;
    const long long total = static_cast<long long>(N) * hw;
    for (long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
         idx += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int n = static_cast<int>(idx / hw), rem = static_cast<int>(idx - static_cast<long long>(n) * hw);
        const int h = rem / W, x = rem - h * W;
        float acc[SMALL_C_MAX] = {0.f, 0.f, 0.f, 0.f};
        const float* dyn = dy + static_cast<size_t>(n) * K * pq;
        // taps that connect this input pixel to an output pixel: (h + pad - r) divisible by the stride and in range
        for (int r = (h + pad_h) % stride_h; r < R; r += stride_h) {
            const int p = (h + pad_h - r) / stride_h;
            if (h + pad_h - r < 0 || p >= P) continue;
            for (int s = (x + pad_w) % stride_w; s < S; s += stride_w) {
                const int q = (x + pad_w - s) / stride_w;
                if (x + pad_w - s < 0 || q >= Q) continue;
                const float* dp = dyn + p * Q + q;
                const float* wp = w_s + r * S + s;
                for (int k = 0; k < K; ++k) {
                    const float g = __ldg(dp + static_cast<size_t>(k) * pq);
#pragma unroll
                    for (int c = 0; c < SMALL_C_MAX; ++c)
                        if (c < C) acc[c] = fmaf(g, wp[(k * C + c) * rs], acc[c]);
                }
            }
        }
        for (int c = 0; c < C; ++c) {
            float* o = dx + (static_cast<size_t>(n) * C + c) * hw + rem;
            float v = alpha * acc[c];
            if (beta != 0.0f) v = fmaf(beta, *o, v);
            *o = v;
        }
    }
}

// The same with dy staged through shared memory, for filters of at most 3 taps per stride step in each direction
// (R <= 3*stride: the first layers of VGG16, 3 x 3 / 1, and of AlexNet and OverFeat, 11 x 11 / 4).  With stride st the
// input pixels fall into st*st phase classes ((h + pad) mod st, (x + pad) mod st); inside a class, pixel (i, j) of the
// class, input (st*i + a - pad, st*j + b - pad), is a stride-1 correlation of dy with the sub-filter
// w[a + st*u][b + st*v], u, v < 3 (zero where that leaves the filter):  dx = sum_{u,v} dy[i - u][j - v] * w[a+st*u][b+st*v].
// A CTA of TW threads owns an 8 x TW tile of one class of one image; dy arrives 8 filters at a time as the tile plus
// its halo; every thread owns one column of the tile and keeps the 10 staged values of a column in registers, so each
// shared-memory load feeds up to 8 rows x 3 taps x C channels.  The sub-filters sit in shared memory as one float4
// (channels 0..3) per filter and tap.
constexpr int S1_TH = 8, S1_KC = 8;
template <int TW, int CC>
__global__ void __launch_bounds__(TW) dgrad_small_c_phase_kernel(int C, int H, int W, int K, int R, int S, int P, int Q, int pad_h,
                                                                 int pad_w, int st, float alpha, float beta,
                                                                 const float* __restrict__ w, const float* __restrict__ dy,
                                                                 float* __restrict__ dx) {
    extern __shared__ float4 s1_smem[];
    constexpr int ROWS = S1_TH + 2, PITCH = TW + 2;
    float4* w_s = s1_smem;                                            // [K][3*3]
    float* dy_s = reinterpret_cast<float*>(s1_smem + K * 9);           // [S1_KC][ROWS][PITCH]
    const int tx = threadIdx.x;
    const int cls = blockIdx.z % (st * st), n = blockIdx.z / (st * st), pa = cls / st, pb = cls - pa * st;
    const int i0 = blockIdx.y * S1_TH, j0 = blockIdx.x * TW;          // tile origin in class coordinates
    const int rs = R * S;
    for (int i = tx; i < K * 9; i += TW) {
        const int k = i / 9, t = i - k * 9, u = t / 3, v = t - u * 3;
        const int r = pa + st * u, sx = pb + st * v;
        float wv[4] = {0.f, 0.f, 0.f, 0.f};
        if (r < R && sx < S)
            for (int c = 0; c < C; ++c) wv[c] = w[(k * C + c) * rs + r * S + sx];
        w_s[i] = make_float4(wv[0], wv[1], wv[2], wv[3]);
    }
    float acc[S1_TH][CC];
#pragma unroll
    for (int i = 0; i < S1_TH; ++i)
#pragma unroll
        for (int c = 0; c < CC; ++c) acc[i][c] = 0.0f;
    // tile row tr holds dy row p0 + tr, tile column tc holds dy column q0 + tc
    const int p0 = i0 - 2, q0 = j0 - 2;
    const float* dyn = dy + static_cast<size_t>(n) * K * P * Q;
    const int q_a = q0 + tx, col_b = TW + tx, q_b = q0 + col_b;
    const bool ok_a = static_cast<unsigned>(q_a) < static_cast<unsigned>(Q);
    const bool has_b = col_b < PITCH, ok_b = has_b && static_cast<unsigned>(q_b) < static_cast<unsigned>(Q);
    for (int k0 = 0; k0 < K; k0 += S1_KC) {
        const int kc = min(S1_KC, K - k0);
        __syncthreads();                                   // the previous chunk has been consumed (first pass: w_s is complete)
        // asynchronous 4-byte copies straight into shared memory (zero-filled outside dy): all of a chunk's loads are
        // in flight at once.  Thread tx copies tile column tx of every row (the first two threads also the halo
        // columns on the right), so the column tests and offsets are computed once.
        for (int kk = 0; kk < kc; ++kk) {
            const float* src = dyn + static_cast<size_t>(k0 + kk) * P * Q;
            float* dst = dy_s + kk * ROWS * PITCH;
#pragma unroll
            for (int tr = 0; tr < ROWS; ++tr) {
                const int p = p0 + tr;
                const bool row_ok = static_cast<unsigned>(p) < static_cast<unsigned>(P);
                const float* rowp = src + (row_ok ? p : 0) * Q;
                const bool a = row_ok && ok_a;
                __pipeline_memcpy_async(dst + tr * PITCH + tx, rowp + (a ? q_a : 0), sizeof(float), a ? 0 : sizeof(float));
                if (has_b) {
                    const bool b2 = row_ok && ok_b;
                    __pipeline_memcpy_async(dst + tr * PITCH + col_b, rowp + (b2 ? q_b : 0), sizeof(float), b2 ? 0 : sizeof(float));
                }
            }
        }
        __pipeline_commit();
        __pipeline_wait_prior(0);
        __syncthreads();
        for (int kk = 0; kk < kc; ++kk) {
            const float* tile = dy_s + kk * ROWS * PITCH;
            const float4* wk = w_s + (k0 + kk) * 9;
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                float colv[ROWS];
#pragma unroll
                for (int tr = 0; tr < ROWS; ++tr) colv[tr] = tile[tr * PITCH + tx + (2 - v)];
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    const float4 w4 = wk[u * 3 + v];
                    const float wc[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int i = 0; i < S1_TH; ++i) {
                        const float g = colv[i + 2 - u];
#pragma unroll
                        for (int c = 0; c < CC; ++c) acc[i][c] = fmaf(g, wc[c], acc[i][c]);
                    }
                }
            }
        }
    }
    const int x = st * (j0 + tx) + pb - pad_w;
    if (x < 0 || x >= W) return;
#pragma unroll
    for (int i = 0; i < S1_TH; ++i) {
        const int h = st * (i0 + i) + pa - pad_h;
        if (h < 0 || h >= H) continue;
#pragma unroll
        for (int c = 0; c < CC; ++c) {
            if (c >= C) break;
            float* o = dx + ((static_cast<size_t>(n) * C + c) * H + h) * W + x;
            float v = alpha * acc[i][c];
            if (beta != 0.0f) v = fmaf(beta, *o, v);
            *o = v;
        }
    }
}

// Without tensors (dx null) it only answers whether it would launch.
template <int TW, int CC>
int launch_dgrad_small_c_phase(const vdnn_conv_desc* d, int P, int Q, float alpha, float beta, const float* w, const float* dy,
                               float* dx, cudaStream_t stream) {
    const int st = d->stride_h;
    const size_t smem = static_cast<size_t>(d->k) * 9 * sizeof(float4) +
                        static_cast<size_t>(S1_KC) * (S1_TH + 2) * (TW + 2) * sizeof(float);
    const long long slices = static_cast<long long>(d->n) * st * st;
    if (smem > 96 * 1024 || slices > 65535) return VDNN_ERR_UNSUPPORTED;
    if (!dx) return VDNN_OK;
    auto kern = dgrad_small_c_phase_kernel<TW, CC>;
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
    VDNN_ALLOW_SHARED(dev, kern, 96 * 1024);
    // class coordinates run over every i with 0 <= st*i + a - pad < H for some phase a: 0 .. (H - 1 + pad) / st
    const int hv = (d->h - 1 + d->pad_h) / st + 1, wv = (d->w - 1 + d->pad_w) / st + 1;
    dim3 grid(ceil_div(wv, TW), ceil_div(hv, S1_TH), static_cast<unsigned>(slices));
    kern<<<grid, TW, smem, stream>>>(d->c, d->h, d->w, d->k, d->r, d->s, P, Q, d->pad_h, d->pad_w, st, alpha, beta, w, dy, dx);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

// Data gradient of a first layer (at most four input channels), or VDNN_ERR_UNSUPPORTED where only the contraction can take
// it.  None of these kernels uses workspace.  Without tensors (dx null) it only answers whether one of them would run.
int dgrad_few_channels(const vdnn_conv_desc* d, int P, int Q, float alpha, const float* w, const float* dy, float beta, float* dx,
                       cudaStream_t stream) {
    if (d->c > SMALL_C_MAX) return VDNN_ERR_UNSUPPORTED;
    int st = window::launch(d, P, Q, alpha, beta, w, dy, dx, stream);
    if (st != VDNN_ERR_UNSUPPORTED) return st;
    if (d->stride_h == d->stride_w && d->r <= 3 * d->stride_h && d->s <= 3 * d->stride_w) {
        const bool narrow = (d->w - 1 + d->pad_w) / d->stride_w + 1 <= 64;      // class coordinates fit a 64-wide tile
        if (d->c == 3) st = narrow ? launch_dgrad_small_c_phase<64, 3>(d, P, Q, alpha, beta, w, dy, dx, stream)
                                   : launch_dgrad_small_c_phase<128, 3>(d, P, Q, alpha, beta, w, dy, dx, stream);
        else st = narrow ? launch_dgrad_small_c_phase<64, 4>(d, P, Q, alpha, beta, w, dy, dx, stream)
                         : launch_dgrad_small_c_phase<128, 4>(d, P, Q, alpha, beta, w, dy, dx, stream);
        if (st != VDNN_ERR_UNSUPPORTED) return st;
    }
    const size_t small_smem = static_cast<size_t>(d->k) * d->c * d->r * d->s * sizeof(float);
    if (small_smem > SMALL_C_SMEM_MAX) return VDNN_ERR_UNSUPPORTED;
    if (!dx) return VDNN_OK;
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
    VDNN_ALLOW_SHARED(dev, dgrad_small_c_kernel, static_cast<int>(SMALL_C_SMEM_MAX));
    const long long total = static_cast<long long>(d->n) * d->h * d->w;
    long long blocks = (total + 255) / 256;
    const long long cap = static_cast<long long>(sm_count()) * (small_smem > 100 * 1024 ? 1 : 2) * 2;
    if (blocks > cap) blocks = cap;
    dgrad_small_c_kernel<<<static_cast<int>(blocks), 256, small_smem, stream>>>(
        d->n, d->c, d->h, d->w, d->k, d->r, d->s, P, Q, d->pad_h, d->pad_w, d->stride_h, d->stride_w, alpha, beta, w, dy, dx);
    VDNN_LAUNCHED();
    return VDNN_OK;
}


// A convolution whose filter covers the whole (unpadded) input produces one output pixel per image: it is a fully
// connected layer, y[n][k] = sum_j w[k][j] x[n][j] with j running over (c, r, s) -- both operands contiguous in j.
bool is_full_extent(const vdnn_conv_desc* d) {
    return d->pad_h == 0 && d->pad_w == 0 && d->h == d->r && d->w == d->s;
}

// PERF_OPT scratch for the weight operand of forward (N = K filters) and data gradient (N = C channels): images of
// its shared-memory tiles, split into tf32 hi / lo halves, that the kernel fetches with bulk copies.
size_t packed_weight_bytes(const vdnn_conv_desc* d, int op) {
    const int red = (op == VDNN_CONV_FWD ? d->c : d->k) * d->r * d->s;
    return tc::bulk_bytes(op == VDNN_CONV_FWD ? d->k : d->c, red);
}

// PERF_OPT scratch for the dy operand of the filter gradient (N = K filters as tile columns, reduction over the
// N*P*Q pixels): the same tile images.  Only where dy fills at least 128 columns: with fewer, the columns are the
// small part of the producers' work and the images (twice the bytes of dy) would not pay for themselves.
size_t packed_dy_bytes(const vdnn_conv_desc* d, int P, int Q) {
    return d->k >= 128 ? tc::bulk_bytes(d->k, d->n * P * Q) : 0;
}

bool valid_desc(const vdnn_conv_desc* d, int* P, int* Q) {
    if (!d || d->n <= 0 || d->c <= 0 || d->h <= 0 || d->w <= 0 || d->k <= 0 || d->r <= 0 || d->s <= 0 ||
        d->pad_h < 0 || d->pad_w < 0 || d->stride_h <= 0 || d->stride_w <= 0)
        return false;
    if (d->h + 2 * d->pad_h < d->r || d->w + 2 * d->pad_w < d->s) return false;
    *P = (d->h + 2 * d->pad_h - d->r) / d->stride_h + 1;
    *Q = (d->w + 2 * d->pad_w - d->s) / d->stride_w + 1;
    return true;
}

// Offsets are 32-bit inside the kernels: every tensor must stay below 2^31 elements.
bool fits_int32(const vdnn_conv_desc* d, int P, int Q) {
    const long long lim = 0x7fffffffLL;
    return 1LL * d->n * d->c * d->h * d->w < lim && 1LL * d->n * d->k * P * Q < lim &&
           1LL * d->k * d->c * d->r * d->s < lim;
}

// Stride-1 convolutions run on the TMA-fed kernels in PERF_OPT (conv_split16.cuh): the gathered tensors are rewritten once into
// lists of positions in workspace and the kernels fetch their operand tiles by tensor copies.
// Layers of stride 2 .. 4 do so in folded form (split16.cuh).
bool split16_layer(const vdnn_conv_desc* d) {
    return g_engine != VDNN_ENGINE_FFMA && !g_no_tma && d->stride_h == d->stride_w && d->stride_h <= split16::FOLD_MAX && !is_full_extent(d);
}

// Lists of at most this many bytes are kept in workspace at a time; layers that need more are walked in slabs of whole images,
// so the workspace stays at the budget whatever the batch size.
constexpr size_t LIST_BUDGET = static_cast<size_t>(512) << 20;
int slab_images(int n, size_t bytes_per_image) {
    if (bytes_per_image * n <= LIST_BUDGET) return n;
    const size_t fit = LIST_BUDGET / bytes_per_image;
    return fit > 1 ? static_cast<int>(fit) : 1;
}

// A layer as the kernels see it: folded where it is strided, with the list geometry of its grid.
struct ListLayer { int c, h, w, R, S, pad_h, pad_w, wp, lp; split16::Fold fold; };
ListLayer list_layer(const vdnn_conv_desc* d, int P, int Q) {
    const int s = d->stride_h;
    ListLayer l{d->c, d->h, d->w, d->r, d->s, d->pad_h, d->pad_w, 0, 0, split16::Fold{s, d->c, d->h, d->w, d->pad_h, d->pad_w, d->r, d->s}};
    if (s > 1) {
        l.c = d->c * s * s; l.R = ceil_div(d->r, s); l.S = ceil_div(d->s, s); l.pad_h = l.pad_w = 0;
        // all that the taps reach, and every pixel of x: the data gradient writes the ones that no tap reaches as well
        l.h = max(P + l.R - 1, ceil_div(d->h + d->pad_h, s)); l.w = max(Q + l.S - 1, ceil_div(d->w + d->pad_w, s));
    }
    const split16::ListGeom g = split16::list_geometry(l.h, l.w, P, Q, l.pad_h, l.pad_w);
    l.wp = g.wp; l.lp = g.wp * g.hp;
    return l;
}

split16::Problem split16_problem(const vdnn_conv_desc* d, int op, int P, int Q) {
    const ListLayer l = list_layer(d, P, Q);
    if (op == VDNN_CONV_FWD) return split16::Problem{d->n, l.c, l.h, l.w, P, Q, d->k, l.R, l.S, 1, -l.pad_h, -l.pad_w, l.wp, l.lp, l.fold};
    // dx[h][w] = sum over taps of dy[h + pad - r][w + pad - s] (stride 1)
    return split16::Problem{d->n, d->k, P, Q, l.h, l.w, l.c, l.R, l.S, -1, l.pad_h, l.pad_w, l.wp, l.lp, l.fold};
}

split16::WgradProblem split16_wgrad_problem(const vdnn_conv_desc* d, int P, int Q) {
    const ListLayer l = list_layer(d, P, Q);
    return split16::WgradProblem{d->n, l.c, l.h, l.w, d->k, P, Q, l.R, l.S, l.pad_h, l.pad_w, l.wp, l.lp, l.fold};
}

// The lists of n images of x from image n0 on.
int write_x_lists(const vdnn_conv_desc* d, int P, int Q, const float* x, int n0, int n, char* lists, const split16::ScaleParts& sp, bool fresh, cudaStream_t s) {
    const ListLayer l = list_layer(d, P, Q);
    const float* src = x + static_cast<size_t>(n0) * d->c * d->h * d->w;
    if (l.fold.s > 1) return split16::write_folded_lists(src, lists, n, l.fold, l.h, l.w, sp, fresh, s);
    return split16::write_lists(src, lists, n, d->c, d->h, d->w, l.wp, l.lp, sp, split16::OP_X, fresh, s);
}
int pack_layer(const vdnn_conv_desc* d, int P, int Q, bool data_gradient, const float* w, char* tiles, const split16::ScaleParts& sp, cudaStream_t s) {
    const ListLayer l = list_layer(d, P, Q);
    if (l.fold.s > 1) return split16::pack_folded(data_gradient, w, d->k, l.fold, l.R, l.S, tiles, sp, s);
    return split16::pack_filters(data_gradient, w, d->k, d->c, d->r, d->s, tiles, sp, s);
}

// What forward or the data gradient keeps in workspace: the scale record, the packed filters, the lists of a slab of images, the
// parts of a split reduction.
struct StripPlan { int slab, splits, group_chunk; size_t pack, lists, partial, total; };

StripPlan strip_plan(const vdnn_conv_desc* d, int op, int P, int Q) {
    const split16::Problem q = split16_problem(d, op, P, Q);
    StripPlan plan;
    plan.slab = slab_images(q.n, split16::list_bytes(1, q.cin, q.lp));
    plan.pack = split16::packed_bytes(q.n_cols, q.cin, q.R * q.S);
    plan.lists = split16::list_bytes(plan.slab, q.cin, q.lp);
    // the reduction is split between groups where the tiles fill less than half of the GPU
    const int groups = split16::strip_groups(q);
    const long long tiles = split16::strip_tiles(q), slots = split16::strip_slots(q.n_cols);
    int splits = 1;
    if (plan.slab == q.n && 2 * tiles <= slots) splits = static_cast<int>(min(static_cast<long long>(groups), slots / tiles));
    plan.group_chunk = ceil_div(groups, splits);
    plan.splits = ceil_div(groups, plan.group_chunk);
    plan.partial = plan.splits > 1 ? static_cast<size_t>(plan.splits) * d->n * (op == VDNN_CONV_FWD ? d->k * P * Q : d->c * d->h * d->w) * sizeof(float) : 0;
    plan.total = split16::SCALE_BYTES + plan.pack + plan.lists + plan.partial;
    return plan;
}

// The filter gradient's: the scale record, the lists of x and dy of a slab, the parts.
struct WgradSpace { int slab; size_t x_lists, dy_lists, partial, total; };

WgradSpace wgrad_space(const vdnn_conv_desc* d, int P, int Q, size_t limit = SIZE_MAX) {
    split16::WgradProblem q = split16_wgrad_problem(d, P, Q);
    WgradSpace w;
    w.slab = slab_images(q.n, split16::list_bytes(1, q.c, q.lp) + split16::list_bytes(1, q.k, q.lp));
    for (;; w.slab = (w.slab + 1) / 2) {
        q.n = w.slab;
        w.x_lists = split16::list_bytes(w.slab, q.c, q.lp);
        w.dy_lists = split16::list_bytes(w.slab, q.k, q.lp);
        w.partial = split16::wgrad_partial_bytes(q);
        w.total = split16::SCALE_BYTES + w.x_lists + w.dy_lists + w.partial;
        if (w.total <= limit || w.slab == 1) return w;
    }
}

// Times in us of the two ways a product can take in PERF_OPT, fitted to 120 drawn layers of 32 .. 512 channels, 1x1 .. 5x5 (B200,
// calls back to back; a tenth off on average, the gathered filter gradient a fifth).  On lists: launches, blocks of the
// reduction in the waves of tiles, passes over the operands and the result (millions of elements), parts of a split
// reduction.  Gathered: blocks and waves likewise.  Choosing by them costs 0.3 % (forward), 0.8 % (data gradient) and 2 % (filter
// gradient) against the faster of the two for every layer, at worst 15, 28 and 48 %; lists everywhere or nowhere lose up to
// 3.3 and 7 times.
struct GatherRate { double block, wave; };
double gathered_us(int M, int N, int K, bool may_split, bool strided) {
    const int bn = tc::tile_n(N), blocks = ceil_div(K, 32), size = bn == 64 ? 0 : (bn == 128 ? 1 : 2);
    const long long tiles = static_cast<long long>(ceil_div(M, 128)) * ceil_div(N, bn);
    int splits = 1;
    if (may_split && tiles < sm_count()) splits = max(1, min(static_cast<int>(2 * sm_count() / tiles), K / 64));
    const double waves = static_cast<double>(ceil_div<long long>(tiles * splits, bn == 64 ? 2 * sm_count() : sm_count()));
    static const GatherRate plain[3] = {{1.4, 1.5}, {0.8, 4.9}, {1.18, 7.7}}, fwd[3] = {{2.4, 4.0}, {0.89, 7.8}, {1.33, 9.1}}, data[3] = {{1.2, 0.0}, {0.69, 0.0}, {1.24, 0.0}};       // data gradients below 40 us start at 11
    GatherRate rate = !strided ? plain[size] : (may_split ? data[size] : fwd[size]);
    if (strided && !may_split && bn == 64 && tiles <= sm_count()) rate.block *= 0.5;      // a CTA has its SM to itself
    return (strided && may_split ? 14.0 : (may_split ? 7.0 : 3.0)) + waves * (rate.block * ceil_div(blocks, splits) + rate.wave);
}

// Folded channels that fill most of their blocks of 64: a first layer of stride 4, or 16 channels and more.
// Small images cost the folding pass up to three times as much per element: its blocks take positions of one image.
double small_images(const vdnn_conv_desc* d) { return 1.0 + 2.0 * min(1.0, 100.0 / (static_cast<double>(d->h) * d->w)); }
bool useful_channels(int c) { return 10 * c >= 7 * split16::padded_channels(c); }

// Forward and data gradient.  With the engine forced to VDNN_ENGINE_TCGEN05 every eligible shape runs on lists (small shapes in the
// tests).
bool choose_strips(const vdnn_conv_desc* d, int op) {
    if (!split16_layer(d) || (op != VDNN_CONV_FWD && op != VDNN_CONV_BWD_DATA)) return false;
    const bool fwd = op == VDNN_CONV_FWD;
    int P, Q;
    const bool first = d->c <= SMALL_C_MAX;          // those of stride 1 have their own kernels
    if ((first && d->stride_h == 1) || (fwd ? d->c * d->stride_h * d->stride_w : d->k) < 8) return false;
    if (!valid_desc(d, &P, &Q) || !fits_int32(d, P, Q)) return false;
    const split16::Problem q = split16_problem(d, op, P, Q);
    if (static_cast<long long>(q.n) * q.lp >= 0x7fffff00LL) return false;
    if (g_engine == VDNN_ENGINE_TCGEN05) return true;
    if (q.n * q.out_h * q.out_w < split16::BM) return false;         // less than a tile: nothing was fitted there
    const StripPlan plan = strip_plan(d, op, P, Q);
    const double src = 0.5e-6 * (static_cast<double>(q.n) * q.cin * q.in_h * q.in_w + static_cast<double>(q.n) * q.lp * split16::padded_channels(q.cin));
    const double out = 1e-6 * q.n * q.n_cols * q.out_h * q.out_w, weights = 1e-6 * q.cin * q.n_cols * q.R * q.S;
    const double waves = static_cast<double>(ceil_div<long long>(split16::strip_tiles(q) * plan.splits, split16::strip_slots(q.n_cols)));
    const double blocks = waves * plan.group_chunk * split16::taps_per_strip(q.S), parts = plan.splits > 1 ? 1 + 2 * plan.splits : 1;
    const int M = fwd ? d->n * P * Q : d->n * d->h * d->w, N = fwd ? d->k : d->c, K = (fwd ? d->c : d->k) * d->r * d->s;
    if (d->stride_h > 1) {
        // Folded layers, fitted to 100 of stride 2 and 4 and corrected by 100 small ones (150 .. 30000 outputs), which lost up to
        // 2.5 times as the data gradient and twice as forward before.  The data gradient gains most, 2 times and more from 1 GFLOP up: the
        // gather tests every tap of every pixel and multiplies zeros, the first layers' kernels do 33 TFLOP/s of multiply-adds.
        // Forward is bound by its passes, and taken where it is surely the faster.
        if (fwd) return useful_channels(q.cin) && 1.1 * (25.0 + 0.4 * blocks + 5.5 * small_images(d) * src + 2.2 * out * parts + 5.0 * weights) < gathered_us(M, N, K, false, true);
        const double lists = 26.0 + 0.77 * blocks + 1.2 * src + 2.0 * out * parts + 5.1 * weights;
        return lists < (first ? 10.0 + 78e-9 * d->n * P * Q * d->k * d->c * d->r * d->s : gathered_us(M, N, K, true, true));
    }
    const double lists = (fwd ? 25.0 : 20.0) + 0.8 * blocks + 1.8 * src + 1.1 * out * parts + 7.7 * weights;
    return lists < gathered_us(M, N, K, !fwd, false) + 0.5 * (src + out);
}

bool choose_wgrad(const vdnn_conv_desc* d) {
    if (!g_tma_wgrad || !split16_layer(d) || d->c * d->stride_h * d->stride_w < 8 || (d->c <= SMALL_C_MAX && d->stride_h == 1)) return false;
    int P, Q;
    if (!valid_desc(d, &P, &Q) || !fits_int32(d, P, Q)) return false;
    const split16::WgradProblem q = split16_wgrad_problem(d, P, Q);
    if (static_cast<long long>(q.n) * q.lp >= 0x7fffff00LL) return false;
    if (g_engine == VDNN_ENGINE_TCGEN05) return true;
    if (d->n * P * Q < split16::BM) return false;
    const split16::WgradPlan w = split16::wgrad_plan(q);
    const double dw = 1e-6 * d->k * d->c * d->r * d->s, dy = 1e-6 * d->n * d->k * P * Q;
    // where the data gradient runs on lists (in the same call: vdnn_conv_bwd_data_filter_bias), dy's are there already
    const bool shared = choose_strips(d, VDNN_CONV_BWD_DATA);
    const double spared = shared ? 0.3 * (dy + 1e-6 * q.n * q.lp * split16::padded_channels(d->k)) : 0.0, launches = shared ? 10.0 : 0.0;
    const double both = 0.5 * (1e-6 * d->n * d->c * d->h * d->w + dy + 1e-6 * q.n * q.lp * (split16::padded_channels(q.c) + split16::padded_channels(d->k)));
    const double waves = static_cast<double>(ceil_div(ceil_div(w.groups, w.chunk) * w.ctas * ceil_div(d->k, w.bn) * w.splits, sm_count()));
    double lists = 27.0 - launches + waves * ((w.bn == 64 ? 2.46 : (w.bn == 128 ? 1.32 : 1.23)) * w.kb_chunk + 3.9) + 2.0 * (both - spared) + 4.5 * w.splits * dw;
    const int M = d->c * d->r * d->s, bn = tc::tile_n(d->k);
    const SplitPlan split = plan_split(M, d->k, d->n * P * Q);
    const double gwaves = static_cast<double>(ceil_div(ceil_div(M, 128) * ceil_div(d->k, bn) * split.splits, sm_count()));
    const double gathered = 10.0 + gwaves * ((bn == 64 ? 1.16 : (bn == 128 ? 1.2 : 1.5)) * (split.k_chunk / 32) + 3.3) + 1.4 * (split.splits > 1 ? split.splits : 0) * dw +
                            (d->k >= 128 ? 3.25 : 0.0) * dy + 1.2 * dw;
    if (d->stride_h > 1) {      // folded: bound by the passes over x; taken where surely faster
        lists = 41.0 - launches + waves * ((w.bn == 64 ? 0.0 : 0.45) * w.kb_chunk + 6.2) + 4.4 * small_images(d) * (both - spared) + 4.6 * w.splits * dw;
        return useful_channels(q.c) && (shared ? 1.2 : 1.6) * lists < 1.3 * gathered;
    }
    return lists < 1.3 * gathered;          // the gather's time is the less certain one, and errs upwards
}

// The choices of a layer are functions of its description (and of the engine), but take a microsecond or two, and a call asks
// several times: each thread remembers those of the layers it met last.
struct Choices { vdnn_conv_desc d; int engine; bool known, fwd, data, filter; };
const Choices& choices(const vdnn_conv_desc* d) {
    static thread_local Choices memo[64];
    const unsigned h = ((d->n * 31u + d->c) * 31u + d->h) * 31u + d->k * 7u + d->r + d->stride_h;
    Choices& m = memo[(h ^ (h >> 6) ^ (h >> 12)) & 63u];
    if (!m.known || m.engine != g_engine || memcmp(&m.d, d, sizeof(*d)) != 0) {
        m.known = false;
        m.fwd = choose_strips(d, VDNN_CONV_FWD); m.data = choose_strips(d, VDNN_CONV_BWD_DATA); m.filter = choose_wgrad(d);
        m.d = *d; m.engine = g_engine; m.known = true;
    }
    return m;
}
bool split16_shape(const vdnn_conv_desc* d, int op) {
    return op == VDNN_CONV_FWD ? choices(d).fwd : (op == VDNN_CONV_BWD_DATA && choices(d).data);
}
bool split16_wgrad_shape(const vdnn_conv_desc* d) { return choices(d).filter; }

int stream_blocks(size_t n) {
    size_t want = ceil_div<size_t>(n, 256);
    const size_t cap = static_cast<size_t>(sm_count()) * 8;
    if (want > cap) want = cap;
    return want ? static_cast<int>(want) : 1;
}

template <class OpA, class OpB, bool AKC, bool BKC>
int run_engine(const OpA& a, const OpB& b, const Epilogue& epi, int M, int N, int K, int splits, int k_chunk,
               cudaStream_t stream, char* b_tiles = nullptr) {
    if (g_engine != VDNN_ENGINE_FFMA && tc::supported<OpA, OpB>(M, N, K)) {
        return tc::launch<OpA, OpB, AKC, BKC>(a, b, epi, M, N, K, splits, k_chunk, stream, b_tiles);
    }
    if (g_engine == VDNN_ENGINE_TCGEN05) return VDNN_ERR_UNSUPPORTED;
    return ffma::launch<OpA, OpB, AKC, BKC>(a, b, epi, M, N, K, splits, k_chunk, stream);
}

// Zero-workspace split reductions: out = beta * out first, then every split adds alpha * its part atomically.
int scale_output(float* out, float beta, int M, int N, size_t dense_elems, int ld_rows, cudaStream_t stream) {
    if (beta == 1.0f) return VDNN_OK;
    if (dense_elems > 0 && beta == 0.0f) {
        VDNN_CUDA(cudaMemsetAsync(out, 0, dense_elems * sizeof(float), stream));
    } else if (dense_elems > 0) {
        scale_dense_kernel<<<stream_blocks(dense_elems), 256, 0, stream>>>(dense_elems, beta, out);
        VDNN_LAUNCHED();
    } else {
        scale_matrix_kernel<<<dim3(ceil_div(M, 256), N < 65535 ? N : 65535), 256, 0, stream>>>(M, N, ld_rows, beta, out);
        VDNN_LAUNCHED();
    }
    return VDNN_OK;
}

// `epi` arrives configured for a direct store (out, alpha, beta, bias, addressing).
// dense_elems > 0 says the output is one dense block of that many floats (needed for PARTIAL).  parts_optional: without room
// for the parts in `ws` the reduction runs unsplit; else that is an error.
template <class OpA, class OpB, bool AKC, bool BKC>
int contract(const OpA& a, const OpB& b, Epilogue epi, int M, int N, int K, size_t dense_elems, int ld_rows,
             int algo_mode, void* ws, size_t ws_bytes, cudaStream_t stream, char* b_tiles = nullptr, bool parts_optional = false) {
    SplitPlan plan = plan_split(M, N, K);
    const size_t need = static_cast<size_t>(plan.splits) * dense_elems * sizeof(float);
    const bool whole = parts_optional && algo_mode == VDNN_ALGO_PERF_OPT && (!ws || ws_bytes < need);
    if (epi.bias || whole) { plan.splits = 1; plan.k_chunk = ceil_div(K, 32) * 32; }
    if (plan.splits == 1) {
        epi.mode = EPI_DIRECT;
        return run_engine<OpA, OpB, AKC, BKC>(a, b, epi, M, N, K, 1, plan.k_chunk, stream, b_tiles);
    }
    if (algo_mode == VDNN_ALGO_PERF_OPT && dense_elems > 0) {
        if (!ws || ws_bytes < need) return VDNN_ERR_WORKSPACE;
        Epilogue part = epi;
        part.mode = EPI_PARTIAL;
        part.out = static_cast<float*>(ws);
        part.partial_stride = dense_elems;
        int st = run_engine<OpA, OpB, AKC, BKC>(a, b, part, M, N, K, plan.splits, plan.k_chunk, stream, b_tiles);
        if (st != VDNN_OK) return st;
        return reduce_partials(dense_elems, plan.splits, epi.alpha, epi.beta, static_cast<const float*>(ws), epi.out, stream);
    }
    const int st = scale_output(epi.out, epi.beta, M, N, dense_elems, ld_rows, stream);
    if (st != VDNN_OK) return st;
    epi.mode = EPI_ATOMIC;
    return run_engine<OpA, OpB, AKC, BKC>(a, b, epi, M, N, K, plan.splits, plan.k_chunk, stream, b_tiles);
}

// SGEMM on the dense kernel (gemm_dense.cuh), which needs no workspace in either mode.
int sgemm_dense(int transa, int transb, int m, int n, int k, float alpha, const float* A, int lda, const float* B, int ldb, float beta,
                float* C, int ldc, cudaStream_t stream) {
    dense::Params p{};
    p.M = m; p.N = n; p.out = C; p.ldc = ldc; p.alpha = alpha; p.beta = beta;
    if (transa && !transb) return dense::launch<true, true>(A, lda, B, ldb, p, k, stream);
    if (!transa && !transb) return dense::launch<false, true>(A, lda, B, ldb, p, k, stream);
    if (!transa && transb) return dense::launch<false, false>(A, lda, B, ldb, p, k, stream);
    return dense::launch<true, false>(A, lda, B, ldb, p, k, stream);
}

// Data gradient of a stride-1 convolution on the halo kernel (conv_halo.cuh), or VDNN_ERR_UNSUPPORTED where the gather-fed one
// is the better without workspace: where no box of the problem fits shared memory, on few columns (which leave the tensor cores
// waiting for operands on either), on small filters (whose elements it does not use often enough), and where its waves of
// tiles cost more.  A wave is one tile on every SM.  Fitted to 568 shapes (B200, flushed L2; 65 .. 512 columns, reductions over
// 4 .. 512 filters, maps of 3 x 4 .. 180 x 180), in us: a wave of the halo kernel takes 1.55 per 32 elements of the reduction
// with 9 taps, 1.25 from 25 taps on, and 2 besides, its start 5; a wave of the gather takes 1.4 and 1.95 on 128 columns (it
// reads dy once per tap), 2.7 and 4.2 on 256, and 5 per 128 columns besides, but it splits the reduction where a wave is not
// full.  Time lost against the better kernel of each shape, on average and at worst: 3x3 0.5 and 11 %, more taps 0.1 and 7 %,
// calls of 10 .. 30 us 0.9 and 30 %.  Going by the share of useful work in the tiles lost 2.6 and 39 %, 1.5 and 59 % (first two).
int dgrad_halo(const vdnn_conv_desc* d, int P, int Q, const float* dy, const float* w, float alpha, float beta, float* dx, cudaStream_t stream) {
    // dx[h][w] = sum over taps of dy[h + pad - r][w + pad - s]: the taps walked from the last to the first
    const halo::Problem q{d->n, d->k, P, Q, d->c, d->h, d->w, d->r, d->s, d->pad_h - (d->r - 1), d->pad_w - (d->s - 1)};
    halo::Params p{};
    const int bn = halo::tile_n(q.n_cols), taps = d->r * d->s;
    if (bn == 0 || taps < 9) return VDNN_ERR_UNSUPPORTED;
    const int M = d->n * d->h * d->w, K = d->k * taps, sms = sm_count();
    const double more = (min(taps, 25) - 9) / 16.0;
    const SplitPlan split = plan_split(M, d->c, K);
    const int columns = tc::tile_n(d->c) / 128;
    const double gather_wave = (columns == 2 ? 2.7 + 1.5 * more : 1.4 + 0.55 * more) * (split.k_chunk / 32) + 5.0 * columns;
    const long long gather_tiles = static_cast<long long>(ceil_div(M, halo::BM)) * ceil_div(d->c, 128 * columns) * split.splits;
    const double gather = static_cast<double>(ceil_div<long long>(gather_tiles, sms)) * gather_wave;
    auto slower = [&](long long waves) { return static_cast<double>(waves) * ((1.55 - 0.3 * more) * (K / 32.0) + 2.0) + 5.0 > gather; };
    // the fewest waves that its tiles can make: known without a plan, which costs some microseconds
    const double full = static_cast<double>(M) * d->c / (static_cast<double>(halo::BM) * bn * sms);
    if (slower(static_cast<long long>(ceil(full))) || !halo::plan(q, bn, &p) || slower(ceil_div<long long>(p.units, sms))) return VDNN_ERR_UNSUPPORTED;
    halo::complete(q, dy, w, &p);
    p.out = dx; p.alpha = alpha; p.beta = beta;
    return halo::launch(bn, p, stream);
}

__global__ void __launch_bounds__(256) scale_gated_kernel(size_t n, float beta, float* out, const int* gate) {
    tc::follow_up();
    tc::after_predecessor();
    if (*gate == 0) return;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) out[i] = beta == 0.0f ? 0.0f : beta * out[i];
}

// The contraction without workspace on the gather-fed kernel, computed only where *gate is set when its turn comes: the call's
// operands do not fit the form of split16.cuh.  The output is one dense block.
template <class OpA, class OpB, bool AKC, bool BKC>
int contract_gated(const OpA& a, const OpB& b, Epilogue epi, int M, int N, int K, const int* gate, cudaStream_t stream) {
    SplitPlan plan = plan_split(M, N, K);
    if (epi.bias) { plan.splits = 1; plan.k_chunk = ceil_div(K, 32) * 32; }
    epi.mode = EPI_DIRECT;
    if (plan.splits > 1) {
        epi.mode = EPI_ATOMIC;
        if (epi.beta != 1.0f) {
            const size_t n = static_cast<size_t>(M) * N;
            VDNN_CUDA(tc::launch_early(scale_gated_kernel, dim3(min(stream_blocks(n), 2 * sm_count())), 256, 0, stream, n, epi.beta, epi.out, gate));
            VDNN_LAUNCHED();
        }
    }
    return tc::launch_gated<OpA, OpB, AKC, BKC>(a, b, epi, M, N, K, plan.splits, plan.k_chunk, gate, stream);
}

// Filter gradient (and bias gradient) for layers with very few input channels and a 3 x 3 / stride-1 filter (VGG16's
// first layer: C = 3).  As a contraction it has 27 rows: a 128-row tensor-core tile is four fifths empty and the gather
// that feeds it costs more than the arithmetic.  Here a block walks tiles of 8 x 32 output pixels of one image; dy of
// 64 filters and the x halo lie in shared memory; thread (filter kk, row set g) keeps the sums of its filter for up to
// three (channel, filter row) pairs x three taps in registers, reading four dy values (one LDS.128) and, per pair, six x
// values (warp-uniform, broadcast) for 12 multiply-adds.  Every block leaves its sums as one partial result
// (partial_w[block][K][C][3][3], partial_b[block][K]); reduce_partials_kernel adds the blocks up in index order.
constexpr int WSC_TR = 8, WSC_TC = 32, WSC_KT = 64;
constexpr int WSC_DY_PITCH = WSC_TR * WSC_TC + 4;        // floats per filter in shared memory (+4: conflict-free LDS.128)
constexpr int WSC_X_PITCH = WSC_TC + 4;                  // 34 columns of halo, padded to a multiple of four floats

template <int C>
__global__ void __launch_bounds__(256, 3) wgrad_small_c_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                                                               float* __restrict__ partial_w, float* __restrict__ partial_b, int N, int H,
                                                               int W, int K, int P, int Q, int pad_h, int pad_w, int tiles_y,
                                                               int tiles_x) {
    extern __shared__ float wsc_smem[];
    float* dyS = wsc_smem;                                               // [WSC_KT][WSC_DY_PITCH]
    float* xS = wsc_smem + WSC_KT * WSC_DY_PITCH;                        // [C][WSC_TR + 2][WSC_X_PITCH]
    constexpr int PAIRS = C * 3;                                         // (channel, filter row)
    constexpr int MINE = (PAIRS + 3) / 4;                                // per row set
    const int t = threadIdx.x, kk = t & 63, g = t >> 6;
    const int k0 = blockIdx.y * WSC_KT;
    float acc[MINE][3];
#pragma unroll
    for (int j = 0; j < MINE; ++j) acc[j][0] = acc[j][1] = acc[j][2] = 0.0f;
    float bsum = 0.0f;
    const long long tiles = static_cast<long long>(N) * tiles_y * tiles_x;
    const size_t pq = static_cast<size_t>(P) * Q, hw = static_cast<size_t>(H) * W;
    for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int n = static_cast<int>(tile / (tiles_y * tiles_x)), rem = static_cast<int>(tile - static_cast<long long>(n) * tiles_y * tiles_x);
        const int p0 = (rem / tiles_x) * WSC_TR, q0 = (rem % tiles_x) * WSC_TC;
        __syncthreads();                                                 // the last tile has been consumed
        // dy: 64 filters x 8 rows x 32 columns, float4 along a row (Q is a multiple of 4: checked by the host)
        for (int i = t; i < WSC_KT * WSC_TR * (WSC_TC / 4); i += 256) {
            const int c4 = i % (WSC_TC / 4), row = (i / (WSC_TC / 4)) % WSC_TR, k = i / (WSC_TC / 4 * WSC_TR);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k0 + k < K && p0 + row < P && q0 + c4 * 4 < Q)
                v = __ldg(reinterpret_cast<const float4*>(dy + (static_cast<size_t>(n) * K + k0 + k) * pq + static_cast<size_t>(p0 + row) * Q + q0) + c4);
            *reinterpret_cast<float4*>(dyS + k * WSC_DY_PITCH + row * WSC_TC + c4 * 4) = v;
        }
        // x halo: rows p0 - pad_h .. + 9, columns q0 - pad_w .. + 33
        for (int i = t; i < C * (WSC_TR + 2) * (WSC_TC + 2); i += 256) {
            const int col = i % (WSC_TC + 2), row = (i / (WSC_TC + 2)) % (WSC_TR + 2), c = i / ((WSC_TC + 2) * (WSC_TR + 2));
            const int ih = p0 - pad_h + row, iw = q0 - pad_w + col;
            float v = 0.0f;
            if (static_cast<unsigned>(ih) < static_cast<unsigned>(H) && static_cast<unsigned>(iw) < static_cast<unsigned>(W))
                v = __ldg(x + (static_cast<size_t>(n) * C + c) * hw + static_cast<size_t>(ih) * W + iw);
            xS[(c * (WSC_TR + 2) + row) * WSC_X_PITCH + col] = v;
        }
        __syncthreads();
        const float* dk = dyS + kk * WSC_DY_PITCH;
#pragma unroll 2
        for (int pr = 0; pr < WSC_TR; ++pr) {
#pragma unroll
            for (int q4 = 0; q4 < WSC_TC / 4; ++q4) {
                const float4 d = *reinterpret_cast<const float4*>(dk + pr * WSC_TC + q4 * 4);
                if (g == 0) bsum += (d.x + d.y) + (d.z + d.w);
#pragma unroll
                for (int j = 0; j < MINE; ++j) {
                    const int pair = g + 4 * j;                          // warp-uniform
                    if (pair < PAIRS) {
                        const int c = pair / 3, r = pair - c * 3;
                        const float* xr = xS + (c * (WSC_TR + 2) + pr + r) * WSC_X_PITCH + q4 * 4;
                        const float4 a = *reinterpret_cast<const float4*>(xr);
                        const float2 b = *reinterpret_cast<const float2*>(xr + 4);
                        acc[j][0] = fmaf(d.x, a.x, fmaf(d.y, a.y, fmaf(d.z, a.z, fmaf(d.w, a.w, acc[j][0]))));
                        acc[j][1] = fmaf(d.x, a.y, fmaf(d.y, a.z, fmaf(d.z, a.w, fmaf(d.w, b.x, acc[j][1]))));
                        acc[j][2] = fmaf(d.x, a.z, fmaf(d.y, a.w, fmaf(d.z, b.x, fmaf(d.w, b.y, acc[j][2]))));
                    }
                }
            }
        }
    }
    if (k0 + kk < K) {
        float* o = partial_w + (static_cast<size_t>(blockIdx.x) * K + k0 + kk) * (C * 9);
#pragma unroll
        for (int j = 0; j < MINE; ++j) {
            const int pair = g + 4 * j;
            if (pair < PAIRS) { o[pair * 3 + 0] = acc[j][0]; o[pair * 3 + 1] = acc[j][1]; o[pair * 3 + 2] = acc[j][2]; }
        }
        if (g == 0) partial_b[static_cast<size_t>(blockIdx.x) * K + k0 + kk] = bsum;
    }
}

bool wgrad_small_c_shape(const vdnn_conv_desc* d, int Q) {
    return d->c <= SMALL_C_MAX && d->c >= 1 && d->r == 3 && d->s == 3 && d->stride_h == 1 && d->stride_w == 1 && Q % 4 == 0 && d->k % 4 == 0 &&
           !is_full_extent(d);
}
int wgrad_small_c_blocks() { return sm_count() * 3; }
size_t wgrad_small_c_bytes(const vdnn_conv_desc* d) {
    return static_cast<size_t>(wgrad_small_c_blocks()) * d->k * (d->c * 9 + 1) * sizeof(float);
}

// dw = alpha * (x corr dy) + beta * dw and, when db is given, db = alpha_b * sum dy + beta_b * db.
int wgrad_small_c(const vdnn_conv_desc* d, int P, int Q, const float* x, const float* dy, float alpha, float beta, float* dw, float alpha_b,
                  float beta_b, float* db, char* ws, size_t ws_bytes, cudaStream_t s) {
    if (ws_bytes < wgrad_small_c_bytes(d)) return VDNN_ERR_WORKSPACE;
    const int blocks = wgrad_small_c_blocks();
    float* partial_w = reinterpret_cast<float*>(ws);
    float* partial_b = partial_w + static_cast<size_t>(blocks) * d->k * d->c * 9;
    const int tiles_y = ceil_div(P, WSC_TR), tiles_x = ceil_div(Q, WSC_TC);
    const size_t smem = (static_cast<size_t>(WSC_KT) * WSC_DY_PITCH + static_cast<size_t>(d->c) * (WSC_TR + 2) * WSC_X_PITCH) * sizeof(float);
    dim3 grid(blocks, ceil_div(d->k, WSC_KT));
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
#define WSC_LAUNCH(CC)                                                                                                                   \
    {                                                                                                                                   \
        VDNN_ALLOW_SHARED(dev, wgrad_small_c_kernel<CC>, 80 * 1024); \
        wgrad_small_c_kernel<CC><<<grid, 256, smem, s>>>(x, dy, partial_w, partial_b, d->n, d->h, d->w, d->k, P, Q, d->pad_h, d->pad_w, tiles_y, tiles_x); \
    }
    switch (d->c) {
    case 1: WSC_LAUNCH(1) break;
    case 2: WSC_LAUNCH(2) break;
    case 3: WSC_LAUNCH(3) break;
    default: WSC_LAUNCH(4) break;
    }
#undef WSC_LAUNCH
    VDNN_LAUNCHED();
    const size_t we = static_cast<size_t>(d->k) * d->c * 9;
    const int st = reduce_partials(we, blocks, alpha, beta, partial_w, dw, s);
    if (st != VDNN_OK || !db) return st;
    return reduce_partials(static_cast<size_t>(d->k), blocks, alpha_b, beta_b, partial_b, db, s);
}

// Forward for the same few-channel 3 x 3 / stride-1 layers: y[n][k][p][q] = alpha * sum x * w + bias[k] + beta * y.  A block
// computes a tile of 8 x 32 output pixels of one image for 64 filters; the x halo and the 64 x (C * 9) weights (stored
// tap-major, filter innermost) lie in shared memory; a thread owns four neighbouring pixels of one row and 16 filters:
// 64 accumulators, per (channel, filter row) six x values and per tap 16 weights (warp-uniform LDS.128, broadcast) for 64
// multiply-adds.  The reduction has 27 terms: as a tensor-core tile it would be one k block per CTA.
template <int C>
__global__ void __launch_bounds__(256, 2) fwd_small_c_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                             const float* __restrict__ bias, float* __restrict__ y, int N, int H, int W,
                                                             int K, int P, int Q, int pad_h, int pad_w, int tiles_y, int tiles_x, float alpha,
                                                             float beta) {
    extern __shared__ float fsc_smem[];
    float* wS = fsc_smem;                                                // [C * 9][WSC_KT]
    float* xS = fsc_smem + C * 9 * WSC_KT;                               // [C][WSC_TR + 2][WSC_X_PITCH]
    const int t = threadIdx.x, quad = t & 63, kg = t >> 6;               // pixel quad of the tile, group of 16 filters
    const int pr = quad >> 3, q4 = quad & 7;
    const int k0 = blockIdx.y * WSC_KT;
    for (int i = t; i < C * 9 * WSC_KT; i += 256) {
        const int k = i % WSC_KT, tap = i / WSC_KT;                     // tap = c * 9 + r * 3 + s
        wS[i] = k0 + k < K ? __ldg(w + static_cast<size_t>(k0 + k) * (C * 9) + tap) : 0.0f;
    }
    const long long tiles = static_cast<long long>(N) * tiles_y * tiles_x;
    const size_t pq = static_cast<size_t>(P) * Q, hw = static_cast<size_t>(H) * W;
    for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int n = static_cast<int>(tile / (tiles_y * tiles_x)), rem = static_cast<int>(tile - static_cast<long long>(n) * tiles_y * tiles_x);
        const int p0 = (rem / tiles_x) * WSC_TR, q0 = (rem % tiles_x) * WSC_TC;
        __syncthreads();                                                 // the last tile's halo has been consumed (and wS is written)
        for (int i = t; i < C * (WSC_TR + 2) * (WSC_TC + 2); i += 256) {
            const int col = i % (WSC_TC + 2), row = (i / (WSC_TC + 2)) % (WSC_TR + 2), c = i / ((WSC_TC + 2) * (WSC_TR + 2));
            const int ih = p0 - pad_h + row, iw = q0 - pad_w + col;
            float v = 0.0f;
            if (static_cast<unsigned>(ih) < static_cast<unsigned>(H) && static_cast<unsigned>(iw) < static_cast<unsigned>(W))
                v = __ldg(x + (static_cast<size_t>(n) * C + c) * hw + static_cast<size_t>(ih) * W + iw);
            xS[(c * (WSC_TR + 2) + row) * WSC_X_PITCH + col] = v;
        }
        __syncthreads();
        float acc[16][4];
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                const float* xr = xS + (c * (WSC_TR + 2) + pr + r) * WSC_X_PITCH + q4 * 4;
                const float4 a = *reinterpret_cast<const float4*>(xr);
                const float2 b = *reinterpret_cast<const float2*>(xr + 4);
                const float xv[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
#pragma unroll
                for (int sx = 0; sx < 3; ++sx) {
                    const float* wk = wS + ((c * 3 + r) * 3 + sx) * WSC_KT + kg * 16;
#pragma unroll
                    for (int j4 = 0; j4 < 4; ++j4) {
                        const float4 wv = *reinterpret_cast<const float4*>(wk + j4 * 4);
                        const float ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j)
#pragma unroll
                            for (int i = 0; i < 4; ++i) acc[j4 * 4 + j][i] = fmaf(ww[j], xv[sx + i], acc[j4 * 4 + j][i]);
                    }
                }
            }
        const int p = p0 + pr, q = q0 + q4 * 4;
        if (p < P && q < Q) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int k = k0 + kg * 16 + j;
                if (k >= K) break;
                float4* o = reinterpret_cast<float4*>(y + (static_cast<size_t>(n) * K + k) * pq + static_cast<size_t>(p) * Q + q);
                const float bk = bias ? __ldg(bias + k) : 0.0f;
                float4 v = make_float4(fmaf(alpha, acc[j][0], bk), fmaf(alpha, acc[j][1], bk), fmaf(alpha, acc[j][2], bk), fmaf(alpha, acc[j][3], bk));
                if (beta != 0.0f) { const float4 old = *o; v.x = fmaf(beta, old.x, v.x); v.y = fmaf(beta, old.y, v.y); v.z = fmaf(beta, old.z, v.z); v.w = fmaf(beta, old.w, v.w); }
                *o = v;
            }
        }
    }
}

int fwd_small_c(const vdnn_conv_desc* d, int P, int Q, float alpha, const float* x, const float* w, const float* bias, float beta, float* y,
                cudaStream_t s) {
    const int tiles_y = ceil_div(P, WSC_TR), tiles_x = ceil_div(Q, WSC_TC);
    const size_t smem = (static_cast<size_t>(d->c) * 9 * WSC_KT + static_cast<size_t>(d->c) * (WSC_TR + 2) * WSC_X_PITCH) * sizeof(float);
    const long long tiles = static_cast<long long>(d->n) * tiles_y * tiles_x;
    long long blocks = static_cast<long long>(sm_count()) * 2;
    if (blocks > tiles) blocks = tiles;
    dim3 grid(static_cast<unsigned>(blocks), ceil_div(d->k, WSC_KT));
    switch (d->c) {
    case 1: fwd_small_c_kernel<1><<<grid, 256, smem, s>>>(x, w, bias, y, d->n, d->h, d->w, d->k, P, Q, d->pad_h, d->pad_w, tiles_y, tiles_x, alpha, beta); break;
    case 2: fwd_small_c_kernel<2><<<grid, 256, smem, s>>>(x, w, bias, y, d->n, d->h, d->w, d->k, P, Q, d->pad_h, d->pad_w, tiles_y, tiles_x, alpha, beta); break;
    case 3: fwd_small_c_kernel<3><<<grid, 256, smem, s>>>(x, w, bias, y, d->n, d->h, d->w, d->k, P, Q, d->pad_h, d->pad_w, tiles_y, tiles_x, alpha, beta); break;
    default: fwd_small_c_kernel<4><<<grid, 256, smem, s>>>(x, w, bias, y, d->n, d->h, d->w, d->k, P, Q, d->pad_h, d->pad_w, tiles_y, tiles_x, alpha, beta); break;
    }
    VDNN_LAUNCHED();
    return VDNN_OK;
}

XGather make_xgather(const vdnn_conv_desc* d, const float* x, int P, int Q) {
    XGather g;
    g.x = x; g.C = d->c; g.H = d->h; g.W = d->w; g.R = d->r; g.S = d->s;
    g.pad_h = d->pad_h; g.pad_w = d->pad_w; g.stride_h = d->stride_h; g.stride_w = d->stride_w;
    g.n_pix = d->n * P * Q; g.n_filt = d->c * d->r * d->s;
    g.Q = Q;
    g.div_pq = FastDiv(P * Q); g.div_q = FastDiv(Q); g.div_rs = FastDiv(d->r * d->s); g.div_s = FastDiv(d->s);
    g.div_c = FastDiv(d->c);
    g.chw = d->c * d->h * d->w; g.hw = d->h * d->w;
    return g;
}

// KCRS weights viewed as [c][(tap, ko)]: offset c*RS + tap + ko*C*RS (the B operand of the data gradient).
SplitDense dgrad_weight_view(const vdnn_conv_desc* d, const float* w) {
    const int rs = d->r * d->s;
    SplitDense B;
    B.p = w; B.rows = d->c; B.cols = d->k * rs;
    B.row_div = FastDiv(1u << 30); B.row_hi = 0;
    B.col_div = FastDiv(d->k);
    B.row_lo = rs; B.col_hi = 1; B.col_lo = d->c * rs;
    return B;
}

DyGather make_dygather(const vdnn_conv_desc* d, const float* dy, int P, int Q) {
    DyGather A;
    A.dy = dy; A.K = d->k; A.P = P; A.Q = Q; A.R = d->r; A.S = d->s;
    A.pad_h = d->pad_h; A.pad_w = d->pad_w; A.stride_h = d->stride_h; A.stride_w = d->stride_w;
    A.n_pix = d->n * d->h * d->w; A.n_cols = d->k * d->r * d->s;
    A.div_hw = FastDiv(d->h * d->w); A.div_w = FastDiv(d->w); A.div_k = FastDiv(d->k); A.div_s = FastDiv(d->s);
    A.div_sh = FastDiv(d->stride_h); A.div_sw = FastDiv(d->stride_w);
    A.kpq = d->k * P * Q; A.pq = P * Q;
    return A;
}

// dy viewed as [k][(n, pq)]: offset = k*PQ + n*K*PQ + pq
SplitDense wgrad_dy_view(const vdnn_conv_desc* d, const float* dy, int pq) {
    SplitDense B;
    B.p = dy; B.rows = d->k; B.cols = d->n * pq;
    B.row_div = FastDiv(1u << 30); B.row_hi = 0; B.row_lo = pq;
    B.col_div = FastDiv(pq); B.col_hi = d->k * pq; B.col_lo = 1;
    return B;
}

// Output addressing: rows are the pixels of `channels` planes of `plane` floats.
Epilogue plane_epilogue(float* out, const float* bias, float alpha, float beta, int channels, int plane) {
    Epilogue e{};
    e.out = out; e.bias = bias; e.alpha = alpha; e.beta = beta;
    e.row_div = FastDiv(plane); e.row_hi = channels * plane; e.row_lo = 1; e.col_stride = plane;
    return e;
}
Epilogue filter_epilogue(float* dw, float alpha, float beta, int crs) {
    Epilogue e{};
    e.out = dw; e.bias = nullptr; e.alpha = alpha; e.beta = beta;
    e.row_div = FastDiv(1u << 30); e.row_hi = 0; e.row_lo = 1; e.col_stride = crs;
    return e;
}

// The three products on the gather-fed kernel without workspace, for operands that the TMA-fed kernels leave to it.
int fwd_gated(const vdnn_conv_desc* d, int P, int Q, float alpha, const float* x, const float* w, const float* bias, float beta, float* y, const int* gate,
              cudaStream_t s) {
    const int crs = d->c * d->r * d->s;
    XGatherPixRows A; A.g = make_xgather(d, x, P, Q);
    return contract_gated<XGatherPixRows, SplitDense, false, true>(A, make_dense(w, d->k, crs, crs, 1), plane_epilogue(y, bias, alpha, beta, d->k, P * Q),
                                                                   d->n * P * Q, d->k, crs, gate, s);
}
int dgrad_gated(const vdnn_conv_desc* d, int P, int Q, float alpha, const float* w, const float* dy, float beta, float* dx, const int* gate, cudaStream_t s) {
    return contract_gated<DyGather, SplitDense, false, false>(make_dygather(d, dy, P, Q), dgrad_weight_view(d, w),
                                                              plane_epilogue(dx, nullptr, alpha, beta, d->c, d->h * d->w), d->n * d->h * d->w, d->c,
                                                              d->k * d->r * d->s, gate, s);
}
int wgrad_gated(const vdnn_conv_desc* d, int P, int Q, float alpha, const float* x, const float* dy, float beta, float* dw, const int* gate, cudaStream_t s) {
    const int crs = d->c * d->r * d->s;
    XGatherFiltRows A; A.g = make_xgather(d, x, P, Q);
    return contract_gated<XGatherFiltRows, SplitDense, true, true>(A, wgrad_dy_view(d, dy, P * Q), filter_epilogue(dw, alpha, beta, crs), crs, d->k,
                                                                   d->n * P * Q, gate, s);
}

bool aligned128(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 127u) == 0; }
size_t x_elems(const vdnn_conv_desc* d) { return static_cast<size_t>(d->n) * d->c * d->h * d->w; }
size_t w_elems(const vdnn_conv_desc* d) { return static_cast<size_t>(d->k) * d->c * d->r * d->s; }
size_t y_elems(const vdnn_conv_desc* d, int P, int Q) { return static_cast<size_t>(d->n) * d->k * P * Q; }

// Forward (src = x, out = y) or data gradient (src = dy, out = dx) on the TMA-fed kernels.
int strips_split16(const vdnn_conv_desc* d, int op, int P, int Q, float alpha, const float* src, const float* w, const float* bias, float beta, float* out,
                   char* ws, size_t ws_bytes, cudaStream_t s) {
    const StripPlan plan = strip_plan(d, op, P, Q);
    if (ws_bytes < plan.total) return VDNN_ERR_WORKSPACE;
    const bool fwd = op == VDNN_CONV_FWD;
    const split16::Problem q = split16_problem(d, op, P, Q);
    const int product = fwd ? split16::FWD : split16::DATA;
    const size_t src_elems = fwd ? x_elems(d) : y_elems(d, P, Q), out_elems = fwd ? y_elems(d, P, Q) : x_elems(d);
    const split16::ScaleParts sp = split16::scale_parts(ws, fwd ? src_elems : 0, w_elems(d), fwd ? 0 : src_elems);
    char* tiles = ws + split16::SCALE_BYTES;
    char* lists = tiles + plan.pack;
    int st = split16::find_magnitudes(sp, fwd ? src : nullptr, fwd ? src_elems : 0, w, w_elems(d), fwd ? nullptr : src, fwd ? 0 : src_elems, s);
    if (st != VDNN_OK) return st;
    if ((st = pack_layer(d, P, Q, !fwd, w, tiles, sp, s)) != VDNN_OK) return st;
    float* partial = plan.splits > 1 ? reinterpret_cast<float*>(lists + plan.lists) : nullptr;
    const int* wide = &sp.scales->wide[product];
    for (int n0 = 0; n0 < q.n; n0 += plan.slab) {
        split16::Problem part = q;
        part.n = min(plan.slab, q.n - n0);
        const size_t src_at = src_elems / q.n * n0, out_at = out_elems / q.n * n0;
        st = fwd ? write_x_lists(d, P, Q, src, n0, part.n, lists, sp, false, s)
                 : split16::write_lists(src + src_at, lists, part.n, d->k, P, Q, q.wp, q.lp, sp, split16::OP_DY, false, s);
        if (st != VDNN_OK) return st;
        if (partial) st = split16::strip_launch(part, lists, tiles, partial, nullptr, 1.0f, 0.0f, EPI_PARTIAL, out_elems, plan.splits, plan.group_chunk, sp.scales, product, s);
        else st = split16::strip_launch(part, lists, tiles, out + out_at, bias, alpha, beta, EPI_DIRECT, out_elems, 1, plan.group_chunk, sp.scales, product, s);
        if (st != VDNN_OK) return st;
    }
    if (partial) {
        if ((st = reduce_partials(out_elems, plan.splits, alpha, beta, partial, out, s, wide)) != VDNN_OK) return st;
    }
    st = fwd ? fwd_gated(d, P, Q, alpha, src, w, partial ? nullptr : bias, beta, out, wide, s) : dgrad_gated(d, P, Q, alpha, w, src, beta, out, wide, s);
    if (st != VDNN_OK || !partial || !bias) return st;
    return vdnn_add_bias(d->n, d->k, P * Q, 1.0f, bias, out, s);
}

// The bias gradient of a layer whose dy is rewritten as lists: that pass can form the sums (then *sums = db, scaled by beta_b here),
// which spares a pass over dy, but adds them by atomics, a thousand or so to an address, one after the other.  Where dy fits L2
// it is better read once more: 12 x 64 x 77 x 81 57 us with sums, 10 + 6 without.
int bias_with_lists(const vdnn_conv_desc* d, int P, int Q, float alpha_b, const float* dy, float beta_b, float* db, float** sums, cudaStream_t s) {
    if (y_elems(d, P, Q) * sizeof(float) <= (static_cast<size_t>(64) << 20) || (beta_b != 0.0f && beta_b != 1.0f))
        return vdnn_conv_bwd_bias(d->n, d->k, P * Q, alpha_b, dy, beta_b, db, s);
    *sums = db;
    if (beta_b == 0.0f) VDNN_CUDA(cudaMemsetAsync(db, 0, sizeof(float) * d->k, s));
    return VDNN_OK;
}

// Filter gradient on the TMA-fed kernels, and with `db` the bias gradient.  Every slab of images adds its share:
// dw = alpha * (sum over slabs) + beta * dw.
int wgrad_split16(const vdnn_conv_desc* d, int P, int Q, const float* x, const float* dy, char* ws, const WgradSpace& space, float* dw, float alpha, float beta,
                  float* db, float alpha_b, float beta_b, cudaStream_t s) {
    split16::WgradProblem q = split16_wgrad_problem(d, P, Q);
    const split16::ScaleParts sp = split16::scale_parts(ws, x_elems(d), 0, y_elems(d, P, Q));
    char* x_lists = ws + split16::SCALE_BYTES;
    char* dy_lists = x_lists + space.x_lists;
    float* partial = reinterpret_cast<float*>(dy_lists + space.dy_lists);
    float* sums = nullptr;
    int st = db ? bias_with_lists(d, P, Q, alpha_b, dy, beta_b, db, &sums, s) : VDNN_OK;
    if (st != VDNN_OK) return st;
    st = split16::find_magnitudes(sp, x, x_elems(d), nullptr, 0, dy, y_elems(d, P, Q), s);
    if (st != VDNN_OK) return st;
    bool fresh = split16::few_parts(sp);
    if (!fresh) {
        VDNN_CUDA(tc::launch_early(split16::scales_kernel, dim3(1), 256, 0, s, sp));
        VDNN_LAUNCHED();
    }
    const int* wide = &sp.scales->wide[split16::FILTER];
    const size_t x_img = x_elems(d) / d->n, dy_img = y_elems(d, P, Q) / d->n;
    for (int n0 = 0; n0 < d->n; n0 += space.slab) {
        q.n = min(space.slab, d->n - n0);
        const float b = n0 == 0 ? beta : 1.0f;
        if ((st = split16::write_lists(dy + n0 * dy_img, dy_lists, q.n, d->k, P, Q, q.wp, q.lp, sp, split16::OP_DY, fresh, s, sums, alpha_b)) != VDNN_OK) return st;
        if ((st = write_x_lists(d, P, Q, x, n0, q.n, x_lists, sp, false, s)) != VDNN_OK) return st;
        fresh = false;
        const split16::WgradPlan plan = split16::wgrad_plan(q);
        if ((st = split16::wgrad_launch(q, plan, x_lists, dy_lists, partial, dw, alpha, b, sp.scales, s)) != VDNN_OK) return st;
        if (plan.splits > 1 && (st = reduce_partials(w_elems(d), plan.splits, alpha, b, partial, dw, s, wide)) != VDNN_OK) return st;
    }
    return wgrad_gated(d, P, Q, alpha, x, dy, beta, dw, wide, s);
}

// ---- one pass over dy for both gradients ---------------------------------------------------------------------------
// The data gradient and the filter gradient read the same lists of dy, so where both run on the TMA-fed kernels one pass writes
// them once (and forms the bias sums), and the two kernels run slab by slab from them.
bool bwd_shared_shape(const vdnn_conv_desc* d) { return split16_shape(d, VDNN_CONV_BWD_DATA) && split16_wgrad_shape(d); }

struct BwdSharedPlan { int slab; size_t pack, dy_lists, x_lists, partial, total; };

BwdSharedPlan bwd_shared_plan(const vdnn_conv_desc* d, int P, int Q) {
    const split16::Problem q = split16_problem(d, VDNN_CONV_BWD_DATA, P, Q);
    split16::WgradProblem wq = split16_wgrad_problem(d, P, Q);
    BwdSharedPlan plan;
    plan.slab = slab_images(d->n, split16::list_bytes(1, d->k, q.lp) + split16::list_bytes(1, wq.c, q.lp));
    plan.pack = split16::packed_bytes(q.n_cols, q.cin, q.R * q.S);
    plan.dy_lists = split16::list_bytes(plan.slab, d->k, q.lp);
    plan.x_lists = split16::list_bytes(plan.slab, wq.c, q.lp);
    wq.n = plan.slab;
    plan.partial = split16::wgrad_partial_bytes(wq);
    plan.total = split16::SCALE_BYTES + plan.pack + plan.dy_lists + plan.x_lists + plan.partial;
    return plan;
}

int bwd_shared_split16(const vdnn_conv_desc* d, int P, int Q, float alpha_dx, const float* w, const float* x, const float* dy, float beta_dx, float* dx,
                       float alpha_w, float beta_w, float* dw, float alpha_b, float beta_b, float* db, char* ws, size_t ws_bytes, cudaStream_t s) {
    const BwdSharedPlan plan = bwd_shared_plan(d, P, Q);
    if (ws_bytes < plan.total) return VDNN_ERR_WORKSPACE;
    const split16::ScaleParts sp = split16::scale_parts(ws, x_elems(d), w_elems(d), y_elems(d, P, Q));
    char* tiles = ws + split16::SCALE_BYTES;
    char* dy_lists = tiles + plan.pack;
    char* x_lists = dy_lists + plan.dy_lists;
    float* partial = reinterpret_cast<float*>(x_lists + plan.x_lists);
    const split16::Problem q = split16_problem(d, VDNN_CONV_BWD_DATA, P, Q);
    split16::WgradProblem wq = split16_wgrad_problem(d, P, Q);
    float* sums = nullptr;
    int st = bias_with_lists(d, P, Q, alpha_b, dy, beta_b, db, &sums, s);
    if (st != VDNN_OK) return st;
    st = split16::find_magnitudes(sp, x, x_elems(d), w, w_elems(d), dy, y_elems(d, P, Q), s);
    if (st != VDNN_OK) return st;
    // the weights as they are now: the filter gradient below may update them in place (dw == w)
    if ((st = pack_layer(d, P, Q, true, w, tiles, sp, s)) != VDNN_OK) return st;
    if ((st = dgrad_gated(d, P, Q, alpha_dx, w, dy, beta_dx, dx, &sp.scales->wide[split16::DATA], s)) != VDNN_OK) return st;
    const int* wide = &sp.scales->wide[split16::FILTER];
    const size_t dy_img = y_elems(d, P, Q) / d->n, x_img = x_elems(d) / d->n;
    const int groups = split16::strip_groups(q);
    for (int n0 = 0; n0 < d->n; n0 += plan.slab) {
        split16::Problem part = q;
        part.n = wq.n = min(plan.slab, d->n - n0);
        const float b = n0 == 0 ? beta_w : 1.0f;
        if ((st = split16::write_lists(dy + n0 * dy_img, dy_lists, part.n, d->k, P, Q, q.wp, q.lp, sp, split16::OP_DY, false, s, sums, alpha_b)) != VDNN_OK) return st;
        if ((st = split16::strip_launch(part, dy_lists, tiles, dx + n0 * x_img, nullptr, alpha_dx, beta_dx, EPI_DIRECT, x_elems(d), 1, groups, sp.scales,
                                        split16::DATA, s)) != VDNN_OK)
            return st;
        if ((st = write_x_lists(d, P, Q, x, n0, part.n, x_lists, sp, false, s)) != VDNN_OK) return st;
        const split16::WgradPlan wplan = split16::wgrad_plan(wq);
        if ((st = split16::wgrad_launch(wq, wplan, x_lists, dy_lists, partial, dw, alpha_w, b, sp.scales, s)) != VDNN_OK) return st;
        if (wplan.splits > 1 && (st = reduce_partials(w_elems(d), wplan.splits, alpha_w, b, partial, dw, s, wide)) != VDNN_OK) return st;
    }
    return wgrad_gated(d, P, Q, alpha_w, x, dy, beta_w, dw, wide, s);
}

// vdnn_sgemm; parts_optional as in contract().
int sgemm(int transa, int transb, int m, int n, int k, float alpha, const float* A, int lda, const float* B, int ldb, float beta, float* C,
          int ldc, int algo_mode, void* workspace, size_t workspace_bytes, cudaStream_t s, bool parts_optional) {
    if (!A || !B || !C || m <= 0 || n <= 0 || k <= 0 || ldc < m) return VDNN_ERR_BAD_ARG;
    if (lda < (transa ? k : m) || ldb < (transb ? n : k)) return VDNN_ERR_BAD_ARG;
    const long long lim = 0x7fffffffLL;
    if (1LL * lda * (transa ? m : k) >= lim || 1LL * ldb * (transb ? k : n) >= lim || 1LL * ldc * n >= lim)
        return VDNN_ERR_UNSUPPORTED;
    // A'(i, kk) = op(A)[i][kk], B'(j, kk) = op(B)[kk][j]
    SplitDense a = transa ? make_dense(A, m, k, lda, 1) : make_dense(A, m, k, 1, lda);
    SplitDense b = transb ? make_dense(B, n, k, 1, ldb) : make_dense(B, n, k, ldb, 1);
    Epilogue e{};
    e.out = C; e.bias = nullptr; e.alpha = alpha; e.beta = beta;
    e.row_div = FastDiv(1u << 30); e.row_hi = 0; e.row_lo = 1; e.col_stride = ldc;
    const size_t dense = (ldc == m) ? static_cast<size_t>(m) * n : 0;
    // operands that tensor copies can fetch run on the dense kernel, the others on the gather-fed one
    if (g_engine != VDNN_ENGINE_FFMA && dense::supported(A, lda, B, ldb))
        return sgemm_dense(transa, transb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, s);
    auto run = [&](auto a_along_k, auto b_along_k) {
        return contract<SplitDense, SplitDense, decltype(a_along_k)::value, decltype(b_along_k)::value>(a, b, e, m, n, k, dense, ldc, algo_mode, workspace,
                                                                                                        workspace_bytes, s, nullptr, parts_optional);
    };
    const std::true_type yes{};
    const std::false_type no{};
    if (transa) return transb ? run(yes, no) : run(yes, yes);
    return transb ? run(no, no) : run(no, yes);
}

// A convolution of full extent is a dense product with rows of C * R * S and K floats.  Where these are whole 16 bytes, tensors
// that begin on 16-byte boundaries run on the dense kernel, and no workspace is reported.  Other tensors of such a shape, which
// the gather-fed kernel takes, run unsplit in that.
bool full_extent_dense(const vdnn_conv_desc* d, int op) {
    return g_engine != VDNN_ENGINE_FFMA && d->c * d->r * d->s % 4 == 0 && (op == VDNN_CONV_FWD || d->k % 4 == 0);
}

// vdnn_conv_bwd_filter; lists: false keeps it on the gather-fed kernel.
int bwd_filter(const vdnn_conv_desc* d, int algo_mode, float alpha, const float* x, const float* dy, float beta, float* dw, void* workspace,
               size_t workspace_bytes, void* stream, bool lists) {
    int P, Q;
    if (!x || !dy || !dw || !valid_desc(d, &P, &Q)) return VDNN_ERR_BAD_ARG;
    if (!fits_int32(d, P, Q)) return VDNN_ERR_UNSUPPORTED;
    const int crs = d->c * d->r * d->s, pq = P * Q;
    if (is_full_extent(d))      // W[k][j] = alpha * sum_n X[n][j] dY[n][k] + beta * W[k][j]   (layer.cu:736-744)
        return sgemm(0, 1, crs, d->k, d->n, alpha, x, crs, dy, d->k, beta, dw, crs, algo_mode, workspace, workspace_bytes, as_stream(stream),
                     full_extent_dense(d, VDNN_CONV_BWD_FILTER));
    if (algo_mode == VDNN_ALGO_PERF_OPT && g_engine != VDNN_ENGINE_FFMA && wgrad_small_c_shape(d, Q) && workspace &&
        (reinterpret_cast<uintptr_t>(dy) & 15u) == 0 && (reinterpret_cast<uintptr_t>(workspace) & 15u) == 0)
        return wgrad_small_c(d, P, Q, x, dy, alpha, beta, dw, 0.0f, 0.0f, nullptr, static_cast<char*>(workspace), workspace_bytes, as_stream(stream));
    // D[j][k] = sum over pixels of x(j; pixel) * dy(k; pixel), written to dw[k*CRS + j]: the expensive operand, the
    // gathered input, supplies the 128 tile rows; dy supplies up to 256 columns, so every gathered element feeds up to
    // 256 multiply-adds and layers with few filters (K = 64) still fill the tile's rows.
    XGatherFiltRows A; A.g = make_xgather(d, x, P, Q);
    const SplitDense B = wgrad_dy_view(d, dy, pq);
    const Epilogue e = filter_epilogue(dw, alpha, beta, crs);
    if (lists && algo_mode == VDNN_ALGO_PERF_OPT && split16_wgrad_shape(d)) {
        if (!workspace) return VDNN_ERR_WORKSPACE;
        if (aligned128(workspace)) {
            const WgradSpace space = wgrad_space(d, P, Q);
            if (workspace_bytes < space.total) return VDNN_ERR_WORKSPACE;
            return wgrad_split16(d, P, Q, x, dy, static_cast<char*>(workspace), space, dw, alpha, beta, nullptr, 0.0f, 0.0f, as_stream(stream));
        }
        algo_mode = VDNN_ALGO_MEMORY_OPT;
    }
    if (algo_mode == VDNN_ALGO_PERF_OPT) {
        // workspace variant: dy, which every row tile of the gathered input needs again, is split into tf32 halves and
        // laid out as tile images once; the kernel's producers then gather x only
        // (tensors off the 16-byte boundaries of a layer whose workspace is sized for wgrad_small_c: its bytes hold the parts of the
        // sums, two splits for each SM against that kernel's three blocks, but no images of dy)
        const size_t pack = wgrad_small_c_shape(d, Q) && g_engine != VDNN_ENGINE_FFMA ? 0 : packed_dy_bytes(d, P, Q);
        if (pack && (!workspace || workspace_bytes < pack)) return VDNN_ERR_WORKSPACE;
        char* tiles = (pack && g_engine != VDNN_ENGINE_FFMA && (reinterpret_cast<uintptr_t>(workspace) & 127u) == 0)
                          ? static_cast<char*>(workspace) : nullptr;
        return contract<XGatherFiltRows, SplitDense, true, true>(A, B, e, crs, d->k, d->n * pq, static_cast<size_t>(d->k) * crs, 0,
                                                                 algo_mode, static_cast<char*>(workspace) + pack,
                                                                 workspace_bytes - pack, as_stream(stream), tiles);
    }
    return contract<XGatherFiltRows, SplitDense, true, true>(A, B, e, crs, d->k, d->n * pq, static_cast<size_t>(d->k) * crs, 0,
                                                             algo_mode, workspace, workspace_bytes, as_stream(stream));
}

// Workspace of the filter gradient on the gather-fed kernel.
size_t gathered_filter_bytes(const vdnn_conv_desc* d, int P, int Q) {
    const int crs = d->c * d->r * d->s;
    const SplitPlan plan = plan_split(crs, d->k, d->n * P * Q);
    return (plan.splits > 1 ? static_cast<size_t>(plan.splits) * crs * d->k * sizeof(float) : 0) + packed_dy_bytes(d, P, Q);
}

}  // namespace
}  // namespace vdnn

using namespace vdnn;

extern "C" {

int vdnn_set_engine(int engine) {
    if (engine < VDNN_ENGINE_AUTO || engine > VDNN_ENGINE_TCGEN05) return VDNN_ERR_BAD_ARG;
    const int prev = g_engine;
    g_engine = engine;
    return prev;
}

int vdnn_get_engine(void) { return g_engine; }

int vdnn_engine_status(int* code) {
    if (!code) return VDNN_ERR_BAD_ARG;
    return tc::take_error(code);
}

int vdnn_engine_status_publish(int* dst, void* stream) {
    if (!dst) return VDNN_ERR_BAD_ARG;
    tc::publish_error_kernel<<<1, 1, 0, as_stream(stream)>>>(dst);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_engine_wait_selftest(unsigned long long limit_cycles, void* stream) {
    if (limit_cycles == 0 || limit_cycles > 2000000000ull) return VDNN_ERR_BAD_ARG;      // at most about a second
    tc::wait_probe_kernel<<<1, 32, 0, as_stream(stream)>>>(limit_cycles);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

int vdnn_engine_mma_rate_probe(int iterations, double* flops, void* stream) {
    if (iterations <= 0 || iterations > (1 << 24) || !flops) return VDNN_ERR_BAD_ARG;
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
    constexpr int smem = 200 * 1024;            // more than half an SM's shared memory: one CTA per SM
    VDNN_ALLOW_SHARED(dev, tc::mma_rate_probe_kernel, smem);
    const int ctas = sm_count();
    tc::mma_rate_probe_kernel<<<ctas, 128, smem, as_stream(stream)>>>(iterations);
    VDNN_LAUNCHED();
    *flops = 2.0 * 128 * 256 * 8 * 12 * static_cast<double>(iterations) * ctas;
    return VDNN_OK;
}

int vdnn_conv_out_dims(const vdnn_conv_desc* d, int* p, int* q) {
    int P, Q;
    if (!p || !q || !valid_desc(d, &P, &Q)) return VDNN_ERR_BAD_ARG;
    *p = P; *q = Q;
    return VDNN_OK;
}

size_t vdnn_conv_workspace_bytes(int op, int algo_mode, const vdnn_conv_desc* d) {
    int P, Q;
    if (!valid_desc(d, &P, &Q) || algo_mode != VDNN_ALGO_PERF_OPT) return 0;
    int M, N, K;
    size_t out;
    const int crs = d->c * d->r * d->s;
    if (op == VDNN_CONV_BWD_ALL) {
        if (bwd_shared_shape(d)) return bwd_shared_plan(d, P, Q).total;
        const size_t a = vdnn_conv_workspace_bytes(VDNN_CONV_BWD_DATA, algo_mode, d), b = vdnn_conv_workspace_bytes(VDNN_CONV_BWD_FILTER, algo_mode, d);
        return a > b ? a : b;
    }
    if (op == VDNN_CONV_BWD_FILTER && split16_wgrad_shape(d)) {
        size_t own = wgrad_space(d, P, Q).total;
        // a caller that sizes the filter gradient's workspace by this figure can also run all three gradients in it
        // (vdnn_conv_bwd_data_filter_bias)
        if (bwd_shared_shape(d)) { const size_t all = bwd_shared_plan(d, P, Q).total; if (all > own) own = all; }
        return own;
    }
    if (split16_shape(d, op)) return strip_plan(d, op, P, Q).total;
    if (is_full_extent(d)) {        // runs as the corresponding FC product
        if (full_extent_dense(d, op)) return 0;
        switch (op) {
        case VDNN_CONV_FWD: return vdnn_sgemm_workspace_bytes(algo_mode, d->k, d->n, crs);
        case VDNN_CONV_BWD_DATA: return vdnn_sgemm_workspace_bytes(algo_mode, crs, d->n, d->k);
        case VDNN_CONV_BWD_FILTER: return vdnn_sgemm_workspace_bytes(algo_mode, crs, d->k, d->n);
        default: return 0;
        }
    }
    // layers of few input channels: kernels without workspace
    if (op == VDNN_CONV_FWD && g_engine != VDNN_ENGINE_FFMA && wgrad_small_c_shape(d, Q)) return 0;
    if (op == VDNN_CONV_BWD_DATA && fits_int32(d, P, Q) && dgrad_few_channels(d, P, Q, 1.0f, nullptr, nullptr, 0.0f, nullptr, nullptr) == VDNN_OK) return 0;
    switch (op) {
    case VDNN_CONV_FWD: M = d->n * P * Q; N = d->k; K = crs; out = static_cast<size_t>(M) * N; break;
    case VDNN_CONV_BWD_DATA: M = d->n * d->h * d->w; N = d->c; K = d->k * d->r * d->s; out = static_cast<size_t>(M) * N; break;
    case VDNN_CONV_BWD_FILTER: M = crs; N = d->k; K = d->n * P * Q; out = static_cast<size_t>(M) * N; break;
    default: return 0;
    }
    if (op == VDNN_CONV_BWD_FILTER && wgrad_small_c_shape(d, Q)) return wgrad_small_c_bytes(d);
    const SplitPlan plan = plan_split(M, N, K);
    size_t bytes = plan.splits > 1 ? static_cast<size_t>(plan.splits) * out * sizeof(float) : 0;
    if (op == VDNN_CONV_FWD || op == VDNN_CONV_BWD_DATA) bytes += packed_weight_bytes(d, op);
    else bytes += packed_dy_bytes(d, P, Q);
    return bytes;
}

int vdnn_conv_fwd(const vdnn_conv_desc* d, int algo_mode, float alpha, const float* x, const float* w,
                  const float* bias, float beta, float* y, void* workspace, size_t workspace_bytes, void* stream) {
    int P, Q;
    if (!x || !w || !y || !valid_desc(d, &P, &Q)) return VDNN_ERR_BAD_ARG;
    if (!fits_int32(d, P, Q)) return VDNN_ERR_UNSUPPORTED;
    const int crs = d->c * d->r * d->s, pq = P * Q, rs = d->r * d->s;
    if (is_full_extent(d)) {    // Y[n][k] = sum_j W[k][j] X[n][j]   (the FC forward product, layer.cu:677-685), then the bias
        const int st = sgemm(1, 0, d->k, d->n, crs, alpha, w, crs, x, crs, beta, y, d->k, algo_mode, workspace, workspace_bytes, as_stream(stream),
                             full_extent_dense(d, VDNN_CONV_FWD));
        if (st != VDNN_OK || !bias) return st;
        return vdnn_add_bias(d->n, d->k, 1, 1.0f, bias, y, stream);
    }
    // few input channels, 3 x 3, stride 1 (the first layer of VGG16): 27 terms per output, an FFMA kernel of its own
    if (g_engine != VDNN_ENGINE_FFMA && wgrad_small_c_shape(d, Q)) {
        if ((reinterpret_cast<uintptr_t>(y) & 15u) == 0) return fwd_small_c(d, P, Q, alpha, x, w, bias, beta, y, as_stream(stream));
        // y off the 16-byte boundaries: the workspace variant below needs what the size query does not report
        if (!workspace || workspace_bytes < packed_weight_bytes(d, VDNN_CONV_FWD)) algo_mode = VDNN_ALGO_MEMORY_OPT;
    }
    const Epilogue e = plane_epilogue(y, bias, alpha, beta, d->k, pq);
    const int M = d->n * pq;
    cudaStream_t s = as_stream(stream);
    if (algo_mode == VDNN_ALGO_PERF_OPT && split16_shape(d, VDNN_CONV_FWD)) {
        if (!workspace) return VDNN_ERR_WORKSPACE;
        if (aligned128(workspace))
            return strips_split16(d, VDNN_CONV_FWD, P, Q, alpha, x, w, bias, beta, y, static_cast<char*>(workspace), workspace_bytes, s);
        algo_mode = VDNN_ALGO_MEMORY_OPT;       // workspace off the boundaries that tensor copies need
    }
    if (algo_mode == VDNN_ALGO_PERF_OPT) {
        // workspace variant: reduce tap-major (k = tap*C + c: one bounds test per run of channels); the weights, read
        // through the matching view ko*CRS + c*RS + tap, are packed once into tile images that the kernel bulk-copies
        const size_t pack = packed_weight_bytes(d, VDNN_CONV_FWD);
        if (!workspace || workspace_bytes < pack) return VDNN_ERR_WORKSPACE;
        XGatherPixRowsTap A; A.g = make_xgather(d, x, P, Q);
        SplitDense B = make_dense(w, d->k, crs, crs, 1);
        B.col_div = FastDiv(d->c); B.col_hi = 1; B.col_lo = rs;
        char* tiles = (g_engine != VDNN_ENGINE_FFMA && (reinterpret_cast<uintptr_t>(workspace) & 127u) == 0) ? static_cast<char*>(workspace) : nullptr;
        return contract<XGatherPixRowsTap, SplitDense, false, true>(A, B, e, M, d->k, crs, static_cast<size_t>(M) * d->k, 0, algo_mode,
                                                                    static_cast<char*>(workspace) + pack, workspace_bytes - pack, s, tiles);
    }
    XGatherPixRows A; A.g = make_xgather(d, x, P, Q);
    SplitDense B = make_dense(w, d->k, crs, crs, 1);
    return contract<XGatherPixRows, SplitDense, false, true>(A, B, e, M, d->k, crs, static_cast<size_t>(M) * d->k, 0,
                                                             algo_mode, workspace, workspace_bytes, s);
}

int vdnn_conv_bwd_data(const vdnn_conv_desc* d, int algo_mode, float alpha, const float* w, const float* dy,
                       float beta, float* dx, void* workspace, size_t workspace_bytes, void* stream) {
    int P, Q;
    if (!w || !dy || !dx || !valid_desc(d, &P, &Q)) return VDNN_ERR_BAD_ARG;
    if (!fits_int32(d, P, Q)) return VDNN_ERR_UNSUPPORTED;
    const int rs = d->r * d->s, hw = d->h * d->w;
    if (is_full_extent(d))      // dX[n][j] = sum_k W[k][j] dY[n][k]   (the FC data-gradient product, layer.cu:725-733)
        return sgemm(0, 0, d->c * rs, d->n, d->k, alpha, w, d->c * rs, dy, d->k, beta, dx, d->c * rs, algo_mode, workspace,
                     workspace_bytes, as_stream(stream), full_extent_dense(d, VDNN_CONV_BWD_DATA));
    if (algo_mode == VDNN_ALGO_PERF_OPT && split16_shape(d, VDNN_CONV_BWD_DATA)) {
        if (!workspace) return VDNN_ERR_WORKSPACE;
        if (aligned128(workspace))
            return strips_split16(d, VDNN_CONV_BWD_DATA, P, Q, alpha, dy, w, nullptr, beta, dx, static_cast<char*>(workspace), workspace_bytes, as_stream(stream));
        algo_mode = VDNN_ALGO_MEMORY_OPT;       // workspace off the boundaries that tensor copies need
    }
    int st = dgrad_few_channels(d, P, Q, alpha, w, dy, beta, dx, as_stream(stream));
    if (st != VDNN_ERR_UNSUPPORTED) return st;
    // Without workspace only: the gather-fed kernel with packed weights (PERF_OPT, channels or sizes that the TMA-fed kernels do
    // not take) is faster than the halo kernel on every shape measured -- 1.07 .. 2.0 times as fast at 3x3 (250 <- 500 channels,
    // 64 images of 28 x 28: 771 against 1565 us; 512 <- 256, 84 x 87: 121 against 209), 1.07 .. 2.5 at 5x5, 1.4 .. 3.0 at 7x7
    // and 9x9.
    if (algo_mode == VDNN_ALGO_MEMORY_OPT && g_engine != VDNN_ENGINE_FFMA && d->stride_h == 1 && d->stride_w == 1) {
        st = dgrad_halo(d, P, Q, dy, w, alpha, beta, dx, as_stream(stream));
        if (st != VDNN_ERR_UNSUPPORTED) return st;
    }
    const DyGather A = make_dygather(d, dy, P, Q);
    const Epilogue e = plane_epilogue(dx, nullptr, alpha, beta, d->c, hw);
    const int M = d->n * hw;
    cudaStream_t s = as_stream(stream);
    const SplitDense B = dgrad_weight_view(d, w);
    if (algo_mode == VDNN_ALGO_PERF_OPT) {
        // workspace variant: that view is packed once into tile images that the kernel bulk-copies
        const size_t pack = packed_weight_bytes(d, VDNN_CONV_BWD_DATA);
        if (!workspace || workspace_bytes < pack) return VDNN_ERR_WORKSPACE;
        char* tiles = (g_engine != VDNN_ENGINE_FFMA && (reinterpret_cast<uintptr_t>(workspace) & 127u) == 0) ? static_cast<char*>(workspace) : nullptr;
        return contract<DyGather, SplitDense, false, false>(A, B, e, M, d->c, d->k * rs, static_cast<size_t>(M) * d->c, 0, algo_mode,
                                                            static_cast<char*>(workspace) + pack, workspace_bytes - pack, s, tiles);
    }
    // zero-workspace variant: B is walked along its rows (channels, 36-byte stride) by neighbouring threads: along k it
    // would be a whole filter apart.
    return contract<DyGather, SplitDense, false, false>(A, B, e, M, d->c, d->k * rs, static_cast<size_t>(M) * d->c, 0,
                                                        algo_mode, workspace, workspace_bytes, s);
}

int vdnn_conv_bwd_filter(const vdnn_conv_desc* d, int algo_mode, float alpha, const float* x, const float* dy,
                         float beta, float* dw, void* workspace, size_t workspace_bytes, void* stream) {
    return bwd_filter(d, algo_mode, alpha, x, dy, beta, dw, workspace, workspace_bytes, stream, true);
}

// Bias gradient and filter gradient of one convolution in one call (layer.cu:631-660: cudnnConvolutionBackwardBias, then
// cudnnConvolutionBackwardFilter).  Where the filter gradient runs on the TMA-fed engine, the pass that rewrites dy into
// operand images also forms the per-channel sums of dy, so dy is read once less and one kernel launch is saved; anywhere
// else this is vdnn_conv_bwd_bias followed by vdnn_conv_bwd_filter.  
int vdnn_conv_bwd_filter_bias(const vdnn_conv_desc* d, int algo_mode, float alpha, const float* x, const float* dy, float beta,
                              float* dw, float alpha_b, float beta_b, float* db, void* workspace, size_t workspace_bytes,
                              void* stream) {
    int P, Q;
    if (!x || !dy || !dw || !db || !valid_desc(d, &P, &Q)) return VDNN_ERR_BAD_ARG;
    const bool combined = algo_mode == VDNN_ALGO_PERF_OPT && split16_wgrad_shape(d) && workspace && aligned128(workspace) &&
                          fits_int32(d, P, Q);
    if (!combined && algo_mode == VDNN_ALGO_PERF_OPT && g_engine != VDNN_ENGINE_FFMA && wgrad_small_c_shape(d, Q) && workspace && fits_int32(d, P, Q) &&
        (reinterpret_cast<uintptr_t>(dy) & 15u) == 0 && (reinterpret_cast<uintptr_t>(workspace) & 15u) == 0)
        return wgrad_small_c(d, P, Q, x, dy, alpha, beta, dw, alpha_b, beta_b, db, static_cast<char*>(workspace), workspace_bytes, as_stream(stream));
    if (!combined) {
        const int st = vdnn_conv_bwd_bias(d->n, d->k, P * Q, alpha_b, dy, beta_b, db, stream);
        return st != VDNN_OK ? st : vdnn_conv_bwd_filter(d, algo_mode, alpha, x, dy, beta, dw, workspace, workspace_bytes, stream);
    }
    const WgradSpace space = wgrad_space(d, P, Q);
    if (workspace_bytes < space.total) return VDNN_ERR_WORKSPACE;
    return wgrad_split16(d, P, Q, x, dy, static_cast<char*>(workspace), space, dw, alpha, beta, db, alpha_b, beta_b, as_stream(stream));
}

// cudnnConvolutionBackwardData, BackwardBias and BackwardFilter of one layer (layer.cu:616-660) in one call and one
// workspace (vdnn_conv_workspace_bytes(VDNN_CONV_BWD_ALL, ...), which the figure for VDNN_CONV_BWD_FILTER covers where the
// gradients share the lists of dy).  The data
// gradient uses the weights as they are on entry, also when dw == w.  Where both gradients run on the TMA-fed engine, dy
// is rewritten into operand images once for both; otherwise the three separate entry points run in the reference's order.
int vdnn_conv_bwd_data_filter_bias(const vdnn_conv_desc* d, int algo_mode, float alpha_dx, const float* w, const float* x, const float* dy,
                                   float beta_dx, float* dx, float alpha_w, float beta_w, float* dw, float alpha_b, float beta_b, float* db,
                                   void* workspace, size_t workspace_bytes, void* stream) {
    int P, Q;
    if (!w || !x || !dy || !dx || !dw || !db || !valid_desc(d, &P, &Q)) return VDNN_ERR_BAD_ARG;
    const bool shared = algo_mode == VDNN_ALGO_PERF_OPT && workspace && aligned128(workspace) && fits_int32(d, P, Q) &&
                        bwd_shared_shape(d);
    if (shared)
        return bwd_shared_split16(d, P, Q, alpha_dx, w, x, dy, beta_dx, dx, alpha_w, beta_w, dw, alpha_b, beta_b, db, static_cast<char*>(workspace),
                                  workspace_bytes, as_stream(stream));
    const int st = vdnn_conv_bwd_data(d, algo_mode, alpha_dx, w, dy, beta_dx, dx, workspace, workspace_bytes, stream);
    return st != VDNN_OK ? st
                         : vdnn_conv_bwd_filter_bias(d, algo_mode, alpha_w, x, dy, beta_w, dw, alpha_b, beta_b, db, workspace, workspace_bytes, stream);
}

// 1 where vdnn_conv_bwd_data_filter_bias shares one pass over dy between the gradients (a host that keeps the three calls
// apart loses nothing elsewhere).
int vdnn_conv_bwd_shares_dy(const vdnn_conv_desc* d, int algo_mode) {
    int P, Q;
    return (algo_mode == VDNN_ALGO_PERF_OPT && valid_desc(d, &P, &Q) && fits_int32(d, P, Q) && bwd_shared_shape(d)) ? 1 : 0;
}

}  // extern "C"

namespace {

// Scratch for vdnn_conv_bwd_filter_static.  In host code this name is only a handle for the
// symbol, not a device address: the address comes from cudaGetSymbolAddress, per device.
static __device__ __align__(256) float g_static_scratch[VDNN_STATIC_SCRATCH_BYTES / sizeof(float)];
constexpr int STATIC_SCRATCH_MAX_DEVICES = 64;
float* g_static_scratch_addr[STATIC_SCRATCH_MAX_DEVICES] = {nullptr};

// Device address of the scratch array on the current device; resolved on first use per device.  The table is not
// guarded: two host threads making their first call on one device at the same time both look the address up and
// store the same value.  Device ordinals beyond the table are refused, never silently skipped.
int static_scratch_address(float** out) {
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= STATIC_SCRATCH_MAX_DEVICES) return VDNN_ERR_UNSUPPORTED;
    if (!g_static_scratch_addr[dev]) {
        void* p = nullptr;
        VDNN_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
        g_static_scratch_addr[dev] = static_cast<float*>(p);
    }
    *out = g_static_scratch_addr[dev];
    return VDNN_OK;
}

}  // namespace

extern "C" {

int vdnn_conv_bwd_filter_static(const vdnn_conv_desc* d, float alpha, const float* x, const float* dy, float beta,
                                float* dw, void* stream) {
    int P, Q;
    if (!x || !dy || !dw || !valid_desc(d, &P, &Q)) return VDNN_ERR_BAD_ARG;
    // what this call takes and refuses: layers of whole blocks of 32 channels by 8 bytes per element besides the parts, others by the
    // figure of the gather-fed kernel
    const bool blocks = g_tma_wgrad && !g_no_tma && d->stride_h == 1 && d->stride_w == 1 && !is_full_extent(d) && d->c % 32 == 0 && d->k % 32 == 0;
    size_t need;
    if (blocks) need = 2 * sizeof(float) * (x_elems(d) + y_elems(d, P, Q)) + split16::wgrad_partial_bytes(split16_wgrad_problem(d, P, Q));
    else if (is_full_extent(d)) need = vdnn_sgemm_workspace_bytes(VDNN_ALGO_PERF_OPT, d->c * d->r * d->s, d->k, d->n);
    else need = wgrad_small_c_shape(d, Q) ? wgrad_small_c_bytes(d) : gathered_filter_bytes(d, P, Q);
    if (need > VDNN_STATIC_SCRATCH_BYTES) return VDNN_ERR_SCRATCH_LIMIT;
    float* scratch = nullptr;
    const int st = static_scratch_address(&scratch);
    if (st != VDNN_OK) return st;
    if (split16_wgrad_shape(d)) {           // as many images at a time as there is room for
        const WgradSpace space = wgrad_space(d, P, Q, VDNN_STATIC_SCRATCH_BYTES);
        if (space.total <= VDNN_STATIC_SCRATCH_BYTES)
            return wgrad_split16(d, P, Q, x, dy, reinterpret_cast<char*>(scratch), space, dw, alpha, beta, nullptr, 0.0f, 0.0f, as_stream(stream));
    }
    const bool gather_fits = is_full_extent(d) || wgrad_small_c_shape(d, Q) || gathered_filter_bytes(d, P, Q) <= VDNN_STATIC_SCRATCH_BYTES;
    // The partial sums of every split are written in full before the reduction reads them, so the
    // array's previous contents never matter.
    return bwd_filter(d, gather_fits ? VDNN_ALGO_PERF_OPT : VDNN_ALGO_MEMORY_OPT, alpha, x, dy, beta, dw, scratch, VDNN_STATIC_SCRATCH_BYTES, stream, false);
}

size_t vdnn_sgemm_workspace_bytes(int algo_mode, int m, int n, int k) {
    if (algo_mode != VDNN_ALGO_PERF_OPT || m <= 0 || n <= 0 || k <= 0) return 0;
    const int splits = plan_split(m, n, k).splits;
    return splits > 1 ? static_cast<size_t>(splits) * m * n * sizeof(float) : 0;
}

int vdnn_sgemm(int transa, int transb, int m, int n, int k, float alpha, const float* A, int lda, const float* B,
               int ldb, float beta, float* C, int ldc, int algo_mode, void* workspace, size_t workspace_bytes,
               void* stream) {
    return sgemm(transa, transb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, algo_mode, workspace, workspace_bytes, as_stream(stream), false);
}

}  // extern "C"
