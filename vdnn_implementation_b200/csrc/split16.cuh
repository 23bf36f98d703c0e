// Operands of the fp32 contraction as pairs of 16-bit floats, and the passes that write them.
//
// With a power of two 2^e that brings the largest magnitude of a tensor into [2^14, 2^15),
//     x 2^e = hi + lo 2^-11,      hi = f16(x 2^e),   lo = f16((x 2^e - hi) 2^11),
// both rounded to nearest, and
//     a b ~= 2^-(ea + eb) (a_hi b_hi + 2^-11 (a_hi b_lo + a_lo b_hi)).
// Two 11-bit significands carry 22 bits, as two tf32 values do (hi and the truncated lo), so three products are exact to
// 2^-22 in either form; but the tensor core multiplies f16 at twice the rate of tf32 and from half the bytes.  (Measured on
// B200 with random operands for a second: 1604 against 864 TFLOP/s in 128 x 256 MMAs, a third of that each for fp32
// products.)  The split of fp32 values over half-precision tensor cores with the scaled remainder is published: Ootomo and
// Yokota, "Recovering single precision accuracy from Tensor Cores while surpassing the FP32 theoretical peak performance",
// IJHPCA 36(4), 2022.  Error of whole calls against float64, 2-norm, nine layers of 32 .. 512 channels and 1x1 .. 5x5: 1.1e-7 to
// 2.8e-7, with pairs of tf32 values and as many chained MMAs 3.1e-7 to 4.7e-7.
//
// What f16 lacks is range.  Keeping lo scaled gives the full 22 bits to every element down to 2^-28 of the tensor's largest;
// below that the error stays at 2^-50 of the largest.  magnitude_kernel finds the largest finite magnitude of every operand
// and the smallest one of any 512 consecutive elements (zeros aside): where they are more than 2^28 apart the operand is
// "wide", the kernels of this form leave at once, and the gather-fed tf32 kernel, launched behind them with the opposite
// condition, computes the call (its launch costs about 2 us where it has nothing to do).  Infinities and NaN do not take
// part in the scale; they go through hi, with lo = 0.
//
// All kernels here are launched with tc::launch_early.  They read global memory by plain loads through plain pointers: a
// read-only load may be moved by the compiler above the wait for the predecessor's results.
#pragma once

#include <cuda_fp16.h>

#include "gemm_tc.cuh"

namespace vdnn {
namespace split16 {

enum Operand { OP_X = 0, OP_W = 1, OP_DY = 2 };
enum Product { FWD = 0, DATA = 1, FILTER = 2 };             // x w, dy w, x dy

constexpr int KB = 64;                    // elements of the reduction per block: rows of 128 bytes
constexpr int ROW_BYTES = KB * 2;
constexpr int PARTS = 1184;               // blocks of magnitude_kernel per operand
constexpr int WIDE_EXPONENTS = 28;

// In workspace, written by every call before it is read.
struct Scales { int e[3]; int wide[3]; };                   // exponents by operand; by product: does one of its operands not fit the form
constexpr size_t SCALE_BYTES = 128 + 3 * PARTS * sizeof(uint2);
static_assert(SCALE_BYTES % 128 == 0, "what follows starts on 128 bytes");

struct ScaleParts {
    Scales* scales;
    uint2* part;                          // [3][PARTS]: largest magnitude, smallest of the runs (bits)
    int blocks[3];
};

// 2^e; -126 <= e <= 127
__device__ __forceinline__ float pow2(int e) { return __int_as_float((e + 127) << 23); }

// What undoes the scales of a product, times alpha: the value of a sum is sum * c, or, where one factor could leave the range of
// fp32 though the result does not, ((sum * f) * g) * alpha.
struct Unscale {
    float c, f, g, alpha;
    bool single;
    __device__ __forceinline__ float operator()(float sum) const { return single ? sum * c : sum * f * g * alpha; }
};
__device__ __forceinline__ Unscale unscale(const Scales* s, int product, float alpha) {
    const int a = s->e[product == DATA ? OP_DY : OP_X], b = s->e[product == FILTER ? OP_DY : OP_W];
    const int t = -(a + b), h = t / 2;
    Unscale u;
    u.f = pow2(h); u.g = pow2(t - h); u.alpha = alpha;
    u.c = u.f * u.g * alpha;
    u.single = abs(t) <= 100 && fabsf(alpha) > 1e-6f && fabsf(alpha) < 1e6f;
    return u;
}

// Bound by HBM: a pass over each operand (4 bytes an element; the pass that writes the lists reads them again).  A warp takes
// runs of 512 elements with four 16-byte loads in flight per lane: 6.0 TB/s on 411 MB.  An operand is walked from its end, so
// that what the next pass reads first is still in L2.
__global__ void __launch_bounds__(256) magnitude_kernel(const float* x, size_t nx, const float* w, size_t nw,
                                                        const float* dy, size_t ndy, const ScaleParts sp) {
    tc::follow_up();
    tc::after_predecessor();
    __shared__ unsigned top[8], low[8];
    int op = 0, block = blockIdx.x;
    while (block >= sp.blocks[op]) block -= sp.blocks[op++];
    const float* p = op == OP_X ? x : (op == OP_W ? w : dy);
    const size_t n = op == OP_X ? nx : (op == OP_W ? nw : ndy);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned largest = 0u, smallest = 0xffffffffu;
    auto bits = [](float v) {
        const unsigned b = __float_as_uint(v) & 0x7fffffffu;
        return b < 0x7f800000u ? b : 0u;
    };
    auto take = [&](unsigned m) {
        m = __reduce_max_sync(0xffffffffu, m);
        largest = max(largest, m);
        if (m) smallest = min(smallest, m);
    };
    // elements before the first and after the last 16-byte boundary
    size_t head = ((16u - (reinterpret_cast<uintptr_t>(p) & 15u)) & 15u) / 4;
    if (head > n) head = n;
    const size_t nvec = (n - head) / 4, tail = head + nvec * 4;
    if (block == 0 && warp == 0) {
        unsigned m = 0u;
        if (static_cast<size_t>(lane) < head) m = bits(p[lane]);
        if (static_cast<size_t>(lane) < n - tail) m = max(m, bits(p[tail + lane]));
        take(m);
    }
    const float4* v = reinterpret_cast<const float4*>(p + head);
    const size_t runs = (nvec + 127) / 128;
    for (size_t run = static_cast<size_t>(block) * 8 + warp; run < runs; run += static_cast<size_t>(sp.blocks[op]) * 8) {
        const size_t i = (runs - 1 - run) * 128;
        float4 q[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const size_t k = i + j * 32 + lane;
            q[j] = k < nvec ? v[k] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        unsigned m = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) m = max(max(m, max(bits(q[j].x), bits(q[j].y))), max(bits(q[j].z), bits(q[j].w)));
        take(m);
    }
    if (lane == 0) { top[warp] = largest; low[warp] = smallest; }
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 1; k < 8; ++k) { largest = max(largest, top[k]); smallest = min(smallest, low[k]); }
        sp.part[op * PARTS + block] = make_uint2(largest, smallest);
    }
}

// All 256 threads of a block: exponent of an operand's scale; *wide as described above.
__device__ __forceinline__ int operand_exponent(const ScaleParts& sp, int op, int* wide) {
    __shared__ unsigned top[8], low[8];
    unsigned largest = 0u, smallest = 0xffffffffu;
    for (int i = threadIdx.x; i < sp.blocks[op]; i += 256) {
        const uint2 v = sp.part[op * PARTS + i];
        largest = max(largest, v.x); smallest = min(smallest, v.y);
    }
    largest = __reduce_max_sync(0xffffffffu, largest);
    smallest = __reduce_min_sync(0xffffffffu, smallest);
    __syncthreads();                                        // an earlier call's values have been read
    if ((threadIdx.x & 31) == 0) { top[threadIdx.x >> 5] = largest; low[threadIdx.x >> 5] = smallest; }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k) { largest = max(largest, top[k]); smallest = min(smallest, low[k]); }
    if (largest == 0u) { *wide = 0; return 0; }
    const int high = static_cast<int>(largest >> 23);      // biased exponents; subnormal numbers count as 2^-127
    *wide = high - static_cast<int>(smallest >> 23) > WIDE_EXPONENTS;
    return min(14 - (high - 127), 126);
}

// One block of 256 threads writes the record of a call.
__device__ __forceinline__ void write_scales(const ScaleParts& sp) {
    int e[3], wide[3];
#pragma unroll
    for (int op = 0; op < 3; ++op) e[op] = operand_exponent(sp, op, &wide[op]);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int op = 0; op < 3; ++op) sp.scales->e[op] = e[op];
        sp.scales->wide[FWD] = wide[OP_X] | wide[OP_W];
        sp.scales->wide[DATA] = wide[OP_DY] | wide[OP_W];
        sp.scales->wide[FILTER] = wide[OP_X] | wide[OP_DY];
    }
}
__global__ void __launch_bounds__(256) scales_kernel(const ScaleParts sp) {
    tc::follow_up();
    tc::after_predecessor();
    write_scales(sp);
}

// x0, x1 (scaled already) as packed halves
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x0, x1);
    const float2 back = __half22float2(h);
    // false for infinities and NaN as well
    const float r0 = fabsf(x0) < 65536.0f ? (x0 - back.x) * 2048.0f : 0.0f, r1 = fabsf(x1) < 65536.0f ? (x1 - back.y) * 2048.0f : 0.0f;
    const __half2 l = __floats2half2_rn(r0, r1);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void split8(const float* v, float scale, uint4& hi, uint4& lo) {
    split2(v[0] * scale, v[1] * scale, hi.x, lo.x);
    split2(v[2] * scale, v[3] * scale, hi.y, lo.y);
    split2(v[4] * scale, v[5] * scale, hi.z, lo.z);
    split2(v[6] * scale, v[7] * scale, hi.w, lo.w);
}

// The filters w[K][C][R][S] as images of the B operand's shared-memory tiles: image (column tile nt, block kb) is bn rows of
// 128 bytes of hi, then bn of lo, 16-byte chunks swizzled as tc::swz; kb = (r * S + s) * cblocks + 64-channel block.  Columns
// are filters and the reduction runs over C (forward), or columns are input channels and it runs over K (DATA = true).
// Channels and columns past the tensor are zero.  A thread writes one chunk (8 channels) for each of the S taps of a filter
// row, so that the taps, neighbours in memory, come out of the cache lines it has.
// Block 0 also writes the call's scale record: every kernel behind this one finds it there.
template <bool DATA_GRADIENT>
__global__ void __launch_bounds__(256) pack_filters_kernel(const float* w, int K, int C, int R, int S, int bn, int n_tiles, int cblocks,
                                                           char* out, const ScaleParts sp) {
    tc::follow_up();
    tc::after_predecessor();
    if (blockIdx.x == 0) write_scales(sp);
    int wide;
    const float scale = pow2(operand_exponent(sp, OP_W, &wide));
    const int cols = DATA_GRADIENT ? C : K, red = DATA_GRADIENT ? K : C, rs = R * S;
    const size_t step = DATA_GRADIENT ? static_cast<size_t>(C) * rs : rs;
    const int kblocks = rs * cblocks;
    const size_t items = static_cast<size_t>(n_tiles) * R * cblocks * bn * 8, stride = static_cast<size_t>(gridDim.x) * 256;
    for (size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; i < items; i += stride) {
        const int chunk = static_cast<int>(i & 7), row = static_cast<int>((i >> 3) % bn);
        size_t rest = (i >> 3) / bn;
        const int cb = static_cast<int>(rest % cblocks);
        rest /= cblocks;
        const int r = static_cast<int>(rest % R), nt = static_cast<int>(rest / R);
        const int col = nt * bn + row, c0 = cb * KB + chunk * 8;
        const float* src = w + (DATA_GRADIENT ? static_cast<size_t>(c0) * C + col : static_cast<size_t>(col) * C + c0) * rs + r * S;
        char* dst = out + (static_cast<size_t>(nt) * kblocks + static_cast<size_t>(r) * S * cblocks + cb) * (2 * bn * ROW_BYTES) + tc::swz(row, chunk);
        for (int s = 0; s < S; ++s) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = col < cols && c0 + j < red ? src[j * step + s] : 0.0f;
            uint4 hi, lo;
            split8(v, scale, hi, lo);
            *reinterpret_cast<uint4*>(dst) = hi;
            *reinterpret_cast<uint4*>(dst + bn * ROW_BYTES) = lo;
            dst += static_cast<size_t>(cblocks) * (2 * bn * ROW_BYTES);
        }
    }
}

// NCHW fp32 -> two lists of positions (hi, lo) with cp channels (C rounded up to whole blocks of 64, zeros past C): position
// n * lp + row * wp + column; the columns from W to wp and the rows from H on are zero.
constexpr int LIST_PIXELS = 64;
struct ListJob {
    const float* src;
    __half* hi;
    __half* lo;
    int C, cp, H, W, wp, lp;
    int tiles;                            // per block
    int op;
    float* sums;                          // receives += sum_scale * (per-channel sums): the bias gradient, where src is dy
    float sum_scale;
};

// A block takes `tiles` consecutive tiles of 64 channels x 64 pixels of one image.  A lane reads four channels of four
// neighbouring pixels (VEC: planes of whole 16 bytes on 16-byte boundaries) or eight of one pixel and of the 32nd after it,
// splits them where they are and passes them through shared memory, in chunks of eight channels, to the threads that write whole
// 128-byte rows.  Bound by HBM, 4 bytes read and 4 written per element; five blocks an SM, so that 80 KB are in flight.
// 32 x 64 x 224 x 224: 123 us (6.7 TB/s), without VEC 134; with registers for four blocks an SM only, 169.  With sums a block of
// a large tensor takes 16 tiles, for fewer atomics on one address: 156 us.
// fresh: the scale record has not been written yet; the blocks find the scale themselves, and the first one writes the record.
template <bool SUMS, bool VEC>
__global__ void __launch_bounds__(256, SUMS && !VEC ? 3 : 5) lists_kernel(const ListJob job, const ScaleParts sp, int fresh) {
    __shared__ uint4 chunk_hi[LIST_PIXELS * 8], chunk_lo[LIST_PIXELS * 8];
    tc::follow_up();
    tc::after_predecessor();
    int e;
    if (fresh) {
        int wide;
        if (blockIdx.x + blockIdx.y + blockIdx.z == 0) write_scales(sp);
        e = operand_exponent(sp, job.op, &wide);
    } else {
        e = sp.scales->e[job.op];
    }
    const float scale = pow2(e);
    const int n = blockIdx.z, c0 = blockIdx.y * KB, C = job.C, cp = job.cp, W = job.W, HW = job.H * W;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, oct = t & 7;
    const size_t base = static_cast<size_t>(n) * job.lp * cp + c0 + oct * 8;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    constexpr int PS = VEC ? 2 : 0;                                        // chunk o of pixel p lies at p * 8 + (o ^ (p >> PS & 7))
    constexpr int CHANNELS = VEC ? 4 : 8;                                  // of a lane
    const int my_c = c0 + (VEC ? (warp * 2 + (lane >> 4)) * 4 : warp * 8), mine = (lane & 15) * 4;
    float part[CHANNELS];
#pragma unroll
    for (int j = 0; j < CHANNELS; ++j) part[j] = 0.0f;
    const int tiles = SUMS ? job.tiles : 1;
    for (int it = 0; it < tiles; ++it) {
        const int p0 = (blockIdx.x * tiles + it) * LIST_PIXELS;
        if (p0 >= HW) break;
        const int npix = min(LIST_PIXELS, HW - p0);
        const float* src = job.src + (static_cast<size_t>(n) * C + my_c) * HW + p0;
        if constexpr (VEC) {
            float v[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 q = mine < npix && my_c + j < C ? *reinterpret_cast<const float4*>(src + static_cast<size_t>(j) * HW + mine)
                                                             : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                v[j][0] = q.x; v[j][1] = q.y; v[j][2] = q.z; v[j][3] = q.w;
            }
            if (SUMS && it) __syncthreads();    // the chunks of the last round have been written out
            const int quad = warp * 2 + (lane >> 4);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint2 h, l;
                split2(v[0][q] * scale, v[1][q] * scale, h.x, l.x);
                split2(v[2][q] * scale, v[3][q] * scale, h.y, l.y);
                const int pix = mine + q, at = (pix * 8 + ((quad >> 1) ^ (pix >> PS & 7))) * 2 + (quad & 1);
                reinterpret_cast<uint2*>(chunk_hi)[at] = h;
                reinterpret_cast<uint2*>(chunk_lo)[at] = l;
            }
            if (SUMS) {
#pragma unroll
                for (int j = 0; j < 4; ++j) part[j] += (v[j][0] + v[j][1]) + (v[j][2] + v[j][3]);
            }
        } else {
            float v[2][8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int pix = q * 32 + lane;
                    v[q][j] = pix < npix && my_c + j < C ? src[static_cast<size_t>(j) * HW + pix] : 0.0f;
                }
            if (SUMS && it) __syncthreads();
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int pix = q * 32 + lane;
                uint4 h, l;
                split8(v[q], scale, h, l);
                chunk_hi[pix * 8 + (warp ^ (pix & 7))] = h;
                chunk_lo[pix * 8 + (warp ^ (pix & 7))] = l;
                if (SUMS) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) part[j] += v[q][j];
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            const int pix = pass * 32 + (t >> 3);
            if (pix < npix) {
                const int pidx = p0 + pix, row = pidx / W, col = pidx - row * W;
                const size_t q = base + (static_cast<size_t>(row) * job.wp + col) * cp;
                *reinterpret_cast<uint4*>(job.hi + q) = chunk_hi[pix * 8 + (oct ^ (pix >> PS & 7))];
                *reinterpret_cast<uint4*>(job.lo + q) = chunk_lo[pix * 8 + (oct ^ (pix >> PS & 7))];
                if (col == W - 1)
                    for (int g = 1; g <= job.wp - W; ++g) {
                        *reinterpret_cast<uint4*>(job.hi + q + static_cast<size_t>(g) * cp) = zero;
                        *reinterpret_cast<uint4*>(job.lo + q + static_cast<size_t>(g) * cp) = zero;
                    }
            }
        }
    }
    if (blockIdx.x == 0)
        for (int q = job.H * job.wp + (t >> 3); q < job.lp; q += 32) {
            *reinterpret_cast<uint4*>(job.hi + base + static_cast<size_t>(q) * cp) = zero;
            *reinterpret_cast<uint4*>(job.lo + base + static_cast<size_t>(q) * cp) = zero;
        }
    if (SUMS) {
#pragma unroll
        for (int j = 0; j < CHANNELS; ++j) {
            float sum = part[j];
#pragma unroll
            for (int o = VEC ? 8 : 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if ((VEC ? lane & 15 : lane) == 0 && my_c + j < C) atomicAdd(job.sums + my_c + j, job.sum_scale * sum);
        }
    }
}

// ---- strided layers -----------------------------------------------------------------------------------------------
//
// A convolution of stride s in both directions is one of stride 1 over positions that hold s x s pixels:
//     x'[(c, a, b)][i][j] = x[c][s i + a - pad_h][s j + b - pad_w],      w'[k][(c, a, b)][u][v] = w[k][c][s u + a][s v + b],
// with ceil(R / s) x ceil(S / s) taps, no padding, and zeros outside x and past R and S.  The folded tensors exist as lists and
// packed filters only.
struct Fold { int s, c, h, w, pad_h, pad_w, R, S; };       // s = 1: not folded; the layer as it is

// As lists_kernel for x' (every position of its h2 x w2 grid is written; there are no gaps).  A block takes 64 channels of x' x 64
// positions of one row: it brings the rows of x that these need, each in one piece and all in flight at once (17 or 18 loads a
// thread), into shared memory, and every thread puts chunks of eight channels together from there.
constexpr int FOLD_MAX = 4;
template <int S>
__global__ void __launch_bounds__(256, 4) fold_lists_kernel(const float* x, __half* hi, __half* lo, const Fold f, int cp, int h2, int w2, int cblocks, const ScaleParts sp,
                                                            int fresh) {
    constexpr int ROWS = KB / S + 2, SPAN = S * 64, PITCH = SPAN + 1, LOADS = (ROWS * SPAN + 255) / 256;
    __shared__ float tile[ROWS * PITCH];
    tc::follow_up();
    tc::after_predecessor();
    int e;
    if (fresh) {
        int wide;
        if (blockIdx.x + blockIdx.y + blockIdx.z == 0) write_scales(sp);
        e = operand_exponent(sp, OP_X, &wide);
    } else {
        e = sp.scales->e[OP_X];
    }
    const float scale = pow2(e);
    const int n = blockIdx.z / cblocks, c0 = (blockIdx.z - n * cblocks) * KB, i = blockIdx.y, j0 = blockIdx.x * 64;
    const int channels = f.c * S * S, row0 = c0 / S, rows = f.c * S - row0;     // (channel, a) rows of x from row0 on
    const int t = threadIdx.x, w0 = S * j0 - f.pad_w, h0 = S * i - f.pad_h;
    const float* image = x + static_cast<size_t>(n) * f.c * f.h * f.w;
    float v[LOADS];
#pragma unroll
    for (int k = 0; k < LOADS; ++k) {
        const int at = t + 256 * k, q = at / SPAN, b = at - q * SPAN, c = (row0 + q) / S, h = h0 + (row0 + q - c * S), w = w0 + b;
        const bool there = q < ROWS && q < rows && static_cast<unsigned>(h) < static_cast<unsigned>(f.h) && static_cast<unsigned>(w) < static_cast<unsigned>(f.w);
        v[k] = there ? image[(static_cast<size_t>(c) * f.h + h) * f.w + w] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < LOADS; ++k) {
        const int at = t + 256 * k, q = at / SPAN;
        if (q < ROWS) tile[q * PITCH + at - q * SPAN] = v[k];
    }
    __syncthreads();
    const int oct = t & 7;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        const int j = pass * 32 + (t >> 3);
        if (j0 + j >= w2) continue;
        float u[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int c2 = c0 + oct * 8 + k, row = c2 / S;
            u[k] = c2 < channels ? tile[(row - row0) * PITCH + S * j + (c2 - row * S)] : 0.0f;
        }
        uint4 h, l;
        split8(u, scale, h, l);
        const size_t q = ((static_cast<size_t>(n) * h2 + i) * w2 + j0 + j) * cp + c0 + oct * 8;
        *reinterpret_cast<uint4*>(hi + q) = h;
        *reinterpret_cast<uint4*>(lo + q) = l;
    }
}

// As pack_filters_kernel for w'.
template <bool DATA_GRADIENT>
__global__ void __launch_bounds__(256) pack_folded_kernel(const float* w, int K, const Fold f, int R2, int S2, int bn, int n_tiles, int cblocks, char* out,
                                                          const ScaleParts sp) {
    tc::follow_up();
    tc::after_predecessor();
    if (blockIdx.x == 0) write_scales(sp);
    int wide;
    const float scale = pow2(operand_exponent(sp, OP_W, &wide));
    const int s = f.s, channels = f.c * s * s, cols = DATA_GRADIENT ? channels : K, red = DATA_GRADIENT ? K : channels, kblocks = R2 * S2 * cblocks;
    const size_t items = static_cast<size_t>(n_tiles) * kblocks * bn * 8, stride = static_cast<size_t>(gridDim.x) * 256;
    for (size_t it = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x; it < items; it += stride) {
        const int chunk = static_cast<int>(it & 7), row = static_cast<int>((it >> 3) % bn);
        const size_t tile = (it >> 3) / bn;                                     // nt * kblocks + kb
        const int kb = static_cast<int>(tile % kblocks), nt = static_cast<int>(tile / kblocks);
        const int tap = kb / cblocks, u = tap / S2, v2 = tap - u * S2, c0 = (kb - tap * cblocks) * KB + chunk * 8, col = nt * bn + row;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = DATA_GRADIENT ? c0 + j : col, c2 = DATA_GRADIENT ? col : c0 + j;
            const int t = c2 / s, b = c2 - t * s, c = t / s, a = t - c * s, r = s * u + a, q = s * v2 + b;
            const bool there = col < cols && c0 + j < red && r < f.R && q < f.S;
            v[j] = there ? w[((static_cast<size_t>(k) * f.c + c) * f.R + r) * f.S + q] : 0.0f;
        }
        uint4 hi, lo;
        split8(v, scale, hi, lo);
        char* dst = out + tile * (2 * bn * ROW_BYTES) + tc::swz(row, chunk);
        *reinterpret_cast<uint4*>(dst) = hi;
        *reinterpret_cast<uint4*>(dst + bn * ROW_BYTES) = lo;
    }
}

// ---- tensor-core side ---------------------------------------------------------------------------------------------

// Instruction descriptor: D = F32, A = B = F16; MN = both operands MN-major.
__host__ __device__ constexpr uint32_t idesc(int m, int n, bool mn) {
    return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24) | (mn ? 3u << 15 : 0u);
}

// MN-major operand: 128-byte rows (one position, 64 channels) with the 128-byte swizzle; 8-position groups 1024 bytes apart,
// the second 64 rows (or columns) of the operand lbo bytes behind the first.
__device__ __forceinline__ uint64_t desc_mn(uint32_t saddr, uint32_t lbo) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(lbo >> 4) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

// D = A B + (accumulate ? D 2^-SHIFT : 0), K = 16
template <int CTAS, int SHIFT>
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate) {
    static_assert(CTAS == 1 || CTAS == 2, "");
    if constexpr (CTAS == 1 && SHIFT == 0)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(accumulate) : "memory");
    else if constexpr (CTAS == 1)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, %5;\n\t}"
                     ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(accumulate), "n"(SHIFT) : "memory");
    else if constexpr (SHIFT == 0)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p, %5;\n\t}"
                     ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(accumulate), "n"(SHIFT) : "memory");
}

// A block of 64 of the reduction is four k slices, STEP 16-byte units apart in both operands.  A chain of blocks forms first all
// its cross products, then the main ones, the first of which scales what is there by 2^-11.  The tensor core truncates when it
// adds into its accumulator, so chains are kept short (24 MMAs) and their sums are added in registers.
template <int CTAS, int STEP>
__device__ __forceinline__ void mma_cross(uint32_t d, uint64_t ah, uint64_t al, uint64_t bh, uint64_t bl, uint32_t id, bool fresh) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        mma<CTAS, 0>(d, al + ks * STEP, bh + ks * STEP, id, ks ? 1u : (fresh ? 0u : 1u));
        mma<CTAS, 0>(d, ah + ks * STEP, bl + ks * STEP, id, 1u);
    }
}
template <int CTAS, int STEP>
__device__ __forceinline__ void mma_main(uint32_t d, uint64_t ah, uint64_t bh, uint32_t id, bool first) {
    if (first) mma<CTAS, 11>(d, ah, bh, id, 1u);
    else mma<CTAS, 0>(d, ah, bh, id, 1u);
#pragma unroll
    for (int ks = 1; ks < 4; ++ks) mma<CTAS, 0>(d, ah + ks * STEP, bh + ks * STEP, id, 1u);
}
// For 64 columns the hi and lo tiles of B lie one behind the other and are taken as one operand of 128 columns (two MMAs per
// k slice instead of three; a narrow MMA does not take less time in proportion): D[0, 64) = a_hi b_hi, D[64, 128) = a_hi b_lo +
// a_lo b_hi.  The drain adds the halves, the second times 2^-11.
template <int STEP>
__device__ __forceinline__ void mma_merged(uint32_t d, uint64_t ah, uint64_t al, uint64_t bh, uint32_t id, uint32_t id_wide, bool fresh) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
        mma<1, 0>(d, ah + ks * STEP, bh + ks * STEP, id_wide, ks ? 1u : (fresh ? 0u : 1u));
        mma<1, 0>(d + 64, al + ks * STEP, bh + ks * STEP, id, 1u);
    }
}

// Sums in registers, two to a 64-bit register: one instruction adds both, each rounded to nearest.
__device__ __forceinline__ void add2(uint64_t& acc, uint32_t lo, uint32_t hi) {
    asm("{\n\t.reg .b64 v;\n\tmov.b64 v, {%1, %2};\n\tadd.rn.f32x2 %0, %0, v;\n\t}" : "+l"(acc) : "r"(lo), "r"(hi));
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint32_t lo, uint32_t hi, float f) {
    asm("{\n\t.reg .b64 v, m;\n\tmov.b64 v, {%1, %2};\n\tmov.b64 m, {%3, %3};\n\tfma.rn.f32x2 %0, v, m, %0;\n\t}" : "+l"(acc) : "r"(lo), "r"(hi), "f"(f));
}
__device__ __forceinline__ float sum_of(const uint64_t* acc, int j) {
    return __uint_as_float(static_cast<uint32_t>(acc[j >> 1] >> ((j & 1) * 32)));
}
// 16 columns of this warp's 32 lanes, without the wait
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
// The registers pass through, so that no use of them is moved in front of the wait.
template <int N>
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[N]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}

// Adds NACC columns of a finished accumulator to a thread's sums (CROSS: and f times the NACC columns `cross` further);
// `done` is called as soon as the last of them has been read.
template <int NACC, bool CROSS, class Done>
__device__ __forceinline__ void drain(uint32_t taddr, uint32_t cross, uint64_t* acc, Done done, float f = 1.0f / 2048.0f) {
    constexpr int LD = CROSS ? 16 : (NACC >= 32 ? 32 : 16);
#pragma unroll
    for (int c = 0; c < NACC; c += LD) {
        uint32_t v[CROSS ? 32 : LD];
        tmem_ld16(taddr + c, v);
        if constexpr (CROSS) tmem_ld16(taddr + cross + c, v + 16);
        else if constexpr (LD == 32) tmem_ld16(taddr + c + 16, v + 16);
        tmem_wait(v);
        if (c + LD >= NACC) done();
#pragma unroll
        for (int j = 0; j < LD; j += 2) add2(acc[(c + j) / 2], v[j], v[j + 1]);
        if constexpr (CROSS) {
#pragma unroll
            for (int j = 0; j < 16; j += 2) fma2(acc[(c + j) / 2], v[16 + j], v[17 + j], f);
        }
    }
}

}  // namespace split16
}  // namespace vdnn
