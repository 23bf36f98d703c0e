// Data gradient of a first layer (at most four input channels) with a square filter and stride: FFMA, all stride phases of a
// position at once.
//
// As a contraction it has C columns, which leaves a tensor-core tile almost empty.  With stride st, input pixel
// (st * i + a - pad, st * j + b - pad) collects  sum over u, v, k of dy[k][i - u][j - v] * w[k][c][a + st * u][b + st * v]:
// the st * st phases (a, b) of a position (i, j) read the SAME window of dy.  A thread takes TI positions below each other
// with all their phases and channels (TI * st * st * CC sums in registers) and, per filter, loads the (TI + U - 1) x U window
// once (U = ceil(R / st); neighbouring threads share it through L1) against TI * R * R * CC multiply-adds; the weights of a
// filter come as float4 broadcasts from shared memory, in the order they are used.
// Walking one phase at a time, with dy staged through shared memory again for each of them, took 1233 us for 64 x 96 x 55 x 55
// (11 x 11 / 4, C = 3: 10.9 TFLOP/s); this takes 405 (calls one behind the other; 435 behind a flush of L2).  64 x 64 x 224 x 224
// (3 x 3 / 1): 634, now 366.
// What bounds it is the code of a filter, unrolled: 860 instructions for 11 x 11 / 4, and warps that wait for them.  One row
// phase per block with more positions each reads fewer weights but measured slower (452 .. 558 us), as did a loop over the
// columns of the window (624).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace vdnn {
namespace window {

template <int R, int ST, int TI, int CC> struct Shape {
    static constexpr int U = (R + ST - 1) / ST, ROWS = TI + U - 1;
    static constexpr int PER_K = (R * R * CC + 3) / 4 * 4;           // floats of a filter in shared memory
    static constexpr int THREADS = TI == 1 ? 128 : (TI * ST * ST * CC > 64 ? 384 : 256);
    // 3 x 3 / 1: little code per filter, so the next filter's window can be under way meanwhile, and warps that lie inside the
    // image take a loop without tests.
    static constexpr bool LIGHT = ST == 1 && R == 3;
};

// Where weight (r, s, c) of a filter lies: blocks (u, v) in order, inside them phase (a, b), then the channel.
template <int R, int ST, int CC>
__device__ __forceinline__ int weight_slot(int r, int s, int c) {
    const int u = r / ST, a = r - u * ST, v = s / ST, b = s - v * ST;
    const int na = min(ST, R - u * ST), nb = min(ST, R - v * ST);
    return (u * ST * R + na * v * ST + a * nb + b) * CC + c;
}

template <int R, int ST, int TI, int CC>
__device__ __forceinline__ void use_filter(float (&acc)[TI][ST * ST * CC], const float (&d)[TI + (R + ST - 1) / ST - 1][(R + ST - 1) / ST],
                                           const float4* wk) {
    constexpr int U = (R + ST - 1) / ST;
    float4 w4 = make_float4(0.f, 0.f, 0.f, 0.f);
    int at = 0;                                                 // a compile-time constant after unrolling
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int v = 0; v < U; ++v)
#pragma unroll
            for (int a = 0; a < (R - u * ST < ST ? R - u * ST : ST); ++a)
#pragma unroll
                for (int b = 0; b < (R - v * ST < ST ? R - v * ST : ST); ++b)
#pragma unroll
                    for (int c = 0; c < CC; ++c, ++at) {
                        if (at % 4 == 0) w4 = wk[at / 4];
                        const float wv = at % 4 == 0 ? w4.x : (at % 4 == 1 ? w4.y : (at % 4 == 2 ? w4.z : w4.w));
#pragma unroll
                        for (int i = 0; i < TI; ++i)
                            acc[i][(a * ST + b) * CC + c] = fmaf(d[i + U - 1 - u][U - 1 - v], wv, acc[i][(a * ST + b) * CC + c]);
                    }
}

struct Params {
    int C, H, W, K, P, Q, pad, k_chunk;
    FastDiv div_nj, div_ni;
    uint32_t total;
    float alpha, beta;
    const float* w;
    const float* dy;
    float* dx;
};

template <int R, int ST, int TI, int CC>
__global__ void __launch_bounds__(Shape<R, ST, TI, CC>::THREADS, Shape<R, ST, TI, CC>::LIGHT ? 2 : 1) dgrad_kernel(const Params p) {
    typedef Shape<R, ST, TI, CC> Sh;
    constexpr int U = Sh::U, ROWS = Sh::ROWS, WORDS = (ROWS * U + 31) / 32;
    extern __shared__ float4 w_s4[];
    float* w_s = reinterpret_cast<float*>(w_s4);
    const uint32_t idx = blockIdx.x * Sh::THREADS + threadIdx.x;
    uint32_t t, j, n, ib;
    p.div_nj.divmod(idx < p.total ? idx : p.total - 1, t, j);
    p.div_ni.divmod(t, n, ib);
    const int i0 = static_cast<int>(ib) * TI;
    // window element (x, y): dy row i0 - (U - 1) + x, column j - (U - 1) + y; zero outside dy
    unsigned mask[WORDS];
    bool inside = true;
#pragma unroll
    for (int m = 0; m < WORDS; ++m) mask[m] = 0;
#pragma unroll
    for (int x = 0; x < ROWS; ++x)
#pragma unroll
        for (int y = 0; y < U; ++y) {
            const int row = i0 - (U - 1) + x, col = static_cast<int>(j) - (U - 1) + y;
            const bool in = static_cast<unsigned>(row) < static_cast<unsigned>(p.P) && static_cast<unsigned>(col) < static_cast<unsigned>(p.Q);
            if (in) mask[(x * U + y) / 32] |= 1u << ((x * U + y) % 32);
            inside = inside && in;
        }
    inside = __all_sync(0xffffffffu, inside);
    const size_t pq = static_cast<size_t>(p.P) * p.Q;
    const int Q = p.Q;
    const float* src = p.dy + static_cast<size_t>(n) * p.K * pq + (static_cast<long long>(i0) - (U - 1)) * Q + (static_cast<int>(j) - (U - 1));
    auto load_masked = [&](float (&d)[ROWS][U], const float* q) {
#pragma unroll
        for (int x = 0; x < ROWS; ++x)
#pragma unroll
            for (int y = 0; y < U; ++y) d[x][y] = (mask[(x * U + y) / 32] >> ((x * U + y) % 32)) & 1u ? __ldg(q + x * Q + y) : 0.0f;
    };
    auto load_inside = [&](float (&d)[ROWS][U], const float* q) {
#pragma unroll
        for (int x = 0; x < ROWS; ++x)
#pragma unroll
            for (int y = 0; y < U; ++y) d[x][y] = __ldg(q + x * Q + y);
    };
    float acc[TI][ST * ST * CC];
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int e = 0; e < ST * ST * CC; ++e) acc[i][e] = 0.0f;

    for (int k0 = 0; k0 < p.K; k0 += p.k_chunk) {
        const int kc = min(p.k_chunk, p.K - k0);
        __syncthreads();
        for (int e = threadIdx.x; e < kc * (R * R * CC); e += Sh::THREADS) {
            const int k = e / (R * R * CC), rest = e - k * (R * R * CC);
            const int c = rest / (R * R), tap = rest - c * (R * R), r = tap / R, s = tap - r * R;
            w_s[k * Sh::PER_K + weight_slot<R, ST, CC>(r, s, c)] = c < p.C ? p.w[(static_cast<size_t>(k0 + k) * p.C + c) * (R * R) + tap] : 0.0f;
        }
        __syncthreads();
        const float4* wk = w_s4;
        if (Sh::LIGHT) {
            auto loop = [&](auto load) {
                float d[ROWS][U];
                load(d, src);
#pragma unroll 2
                for (int k = 0; k < kc; ++k, wk += Sh::PER_K / 4) {
                    float next[ROWS][U];
                    if (k + 1 < kc) src += pq;                  // behind the last filter of a chunk: the same again
                    load(next, src);
                    use_filter<R, ST, TI, CC>(acc, d, wk);
#pragma unroll
                    for (int x = 0; x < ROWS; ++x)
#pragma unroll
                        for (int y = 0; y < U; ++y) d[x][y] = next[x][y];
                }
                src += pq;
            };
            if (inside) loop(load_inside); else loop(load_masked);
        } else {
#pragma unroll 1
            for (int k = 0; k < kc; ++k, src += pq, wk += Sh::PER_K / 4) {
                float d[ROWS][U];
                load_masked(d, src);
                use_filter<R, ST, TI, CC>(acc, d, wk);
            }
        }
    }
    if (idx >= p.total) return;
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
        for (int a = 0; a < ST; ++a) {
            const int h = ST * (i0 + i) + a - p.pad;
            if (h < 0 || h >= p.H) continue;
#pragma unroll
            for (int b = 0; b < ST; ++b) {
                const int x = ST * static_cast<int>(j) + b - p.pad;
                if (x < 0 || x >= p.W) continue;
#pragma unroll
                for (int c = 0; c < CC; ++c) {
                    if (c >= p.C) break;
                    float* o = p.dx + ((static_cast<size_t>(n) * p.C + c) * p.H + h) * p.W + x;
                    const float v = p.alpha * acc[i][(a * ST + b) * CC + c];
                    *o = p.beta != 0.0f ? fmaf(p.beta, *o, v) : v;
                }
            }
        }
}

// Without tensors (dx null) it only answers whether it would launch.
template <int R, int ST, int TI, int CC>
int launch_shape(const vdnn_conv_desc* d, int P, int Q, float alpha, float beta, const float* w, const float* dy, float* dx, cudaStream_t stream) {
    typedef Shape<R, ST, TI, CC> Sh;
    // positions i with 0 <= ST * i + a - pad < H for some phase a
    const int hv = (d->h - 1 + d->pad_h) / ST + 1, wv = (d->w - 1 + d->pad_w) / ST + 1, ni = ceil_div(hv, TI);
    const long long total = static_cast<long long>(d->n) * ni * wv;
    if (total > 0x7ffffc00LL) return VDNN_ERR_UNSUPPORTED;
    if (!dx) return VDNN_OK;
    constexpr int LIMIT = 200 * 1024, fit = LIMIT / (Sh::PER_K * 4);
    Params p;
    p.C = d->c; p.H = d->h; p.W = d->w; p.K = d->k; p.P = P; p.Q = Q; p.pad = d->pad_h;
    p.k_chunk = d->k < fit ? d->k : fit;
    p.div_nj = FastDiv(wv); p.div_ni = FastDiv(ni); p.total = static_cast<uint32_t>(total);
    p.alpha = alpha; p.beta = beta; p.w = w; p.dy = dy; p.dx = dx;
    auto kern = dgrad_kernel<R, ST, TI, CC>;
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
    VDNN_ALLOW_SHARED(dev, kern, LIMIT);
    kern<<<static_cast<unsigned>(ceil_div<long long>(total, Sh::THREADS)), Sh::THREADS, p.k_chunk * Sh::PER_K * 4, stream>>>(p);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

// Rows of a thread: the more, the fewer weights are read per sum, as far as the registers (sums; 3 x 3 / 1 also keeps the next
// window) and the code of a filter go.  Measured at 64 filters and twice 128 registers of sums, 5 x 5 / 3 took 90 us where this
// takes 66, 7 x 7 / 3 139 and 98, 3 x 3 / 1 with four channels 86 and 49.
constexpr int rows_each(int r, int st, int cc) {
    int ti = 8;
    while (ti > 2 && (ti * st * st * cc > 96 || ti * r * r * cc > 1024 || (r == 3 && st == 1 && ti * cc > 24))) ti /= 2;
    return ti;
}

// What a thread does takes the same time however few of them there are (11 x 11 / 4: 2.4 us per filter, 5 x 5 / 1 1.6), so
// below half a block for each SM strides 1 and 2 take one row per thread: 5 x 5 / 1, 64 filters, four images of 64 x 64:
// 98 -> 44 us, 7 x 7 / 2 160 -> 109.  At strides 3 and 4 that gains little (11 x 11 / 4 229 -> 195); there the phases go to
// threads of their own below a seventh of a block for each SM (other kernels: 11 x 11 / 4, 96 filters, four images of 128 x 128
// 119 against 229 us, 16 images 252 against 225).
template <int R, int ST, int CC>
int launch_filter(const vdnn_conv_desc* d, int P, int Q, float alpha, float beta, const float* w, const float* dy, float* dx, cudaStream_t stream) {
    constexpr int TI = rows_each(R, ST, CC);
    const long long positions = static_cast<long long>(d->n) * ceil_div((d->h - 1 + d->pad_h) / ST + 1, TI) * ((d->w - 1 + d->pad_w) / ST + 1);
    const long long blocks = positions / Shape<R, ST, TI, CC>::THREADS;
    if constexpr (ST <= 2) {
        if (2 * blocks < sm_count()) return launch_shape<R, ST, 1, CC>(d, P, Q, alpha, beta, w, dy, dx, stream);
    } else {
        if (7 * blocks < sm_count()) return VDNN_ERR_UNSUPPORTED;
    }
    return launch_shape<R, ST, TI, CC>(d, P, Q, alpha, beta, w, dy, dx, stream);
}

template <int R>
int launch_side(const vdnn_conv_desc* d, int P, int Q, float alpha, float beta, const float* w, const float* dy, float* dx, cudaStream_t stream) {
    auto run = [&](auto st) {
        constexpr int ST = decltype(st)::value;
        if constexpr (ST > R) return static_cast<int>(VDNN_ERR_UNSUPPORTED);
        else return d->c <= 3 ? launch_filter<R, ST, 3>(d, P, Q, alpha, beta, w, dy, dx, stream)
                              : launch_filter<R, ST, 4>(d, P, Q, alpha, beta, w, dy, dx, stream);
    };
    switch (d->stride_h) {
    case 1: return run(std::integral_constant<int, 1>());
    case 2: return run(std::integral_constant<int, 2>());
    case 3: return run(std::integral_constant<int, 3>());
    case 4: return run(std::integral_constant<int, 4>());
    default: return VDNN_ERR_UNSUPPORTED;
    }
}

// Square filters of an odd side up to 11 at the same stride, up to 4 and to their side, both ways.  Against the kernels that take
// the others (64 filters, 16 images, output 112 x 112 at stride 1 and 2): 3x3/1 59 and 76 us, 5x5/1 106 and 262, 7x7/1 160 and
// 494, 9x9/1 293 and 809, 11x11/1 422 and 1412, 3x3/2 80 and 123, 5x5/2 131 and 191, 7x7/2 164 and 553, 9x9/2 248 and 1020,
// 11x11/2 336 and 1421; 224 x 224 images at stride 3: 51 .. 205 and 68 .. 678; at stride 4: 66 .. 158 and 111 .. 225.
// VDNN_ERR_UNSUPPORTED for all others.
inline int launch(const vdnn_conv_desc* d, int P, int Q, float alpha, float beta, const float* w, const float* dy, float* dx, cudaStream_t stream) {
    if (d->r != d->s || d->stride_h != d->stride_w || d->pad_h != d->pad_w || d->c > 4) return VDNN_ERR_UNSUPPORTED;
    switch (d->r) {
    case 3: return launch_side<3>(d, P, Q, alpha, beta, w, dy, dx, stream);
    case 5: return launch_side<5>(d, P, Q, alpha, beta, w, dy, dx, stream);
    case 7: return launch_side<7>(d, P, Q, alpha, beta, w, dy, dx, stream);
    case 9: return launch_side<9>(d, P, Q, alpha, beta, w, dy, dx, stream);
    case 11: return launch_side<11>(d, P, Q, alpha, beta, w, dy, dx, stream);
    default: return VDNN_ERR_UNSUPPORTED;
    }
}

}  // namespace window
}  // namespace vdnn
