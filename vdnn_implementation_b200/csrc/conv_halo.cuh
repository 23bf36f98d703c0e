// Data gradient of a stride-1 convolution straight from NCHW, without workspace: implicit GEMM on tcgen05 with the gathered
// operand in tensor memory.
//
//   dx[pixel][col] = sum over (k, r, s) of dy[k][pixel + off + (r, s)] * w[k][col][R - 1 - r][S - 1 - s]
//
// The gather-fed kernel (gemm_tc.cuh) computes an address, a bounds test and a 4-byte global load for every element of every
// 128 x 32 operand tile, R * S times for each element of dy, and walks the weights a filter apart: 49 .. 61 TFLOP/s.  Here a
// tile is a box of bh x bw pixels of dx, and per chunk of a few filters
//   * three loader warps copy the box's region of dy with its halo -- once, not once per tap; zero outside the image, so
//     padding costs nothing later -- and the chunk's raw weights into shared memory (cp.async; any alignment and size);
//   * split warps form the operand blocks of up to 32 (k, r, s) from there: A element (pixel, kk) is one 4-byte shared-memory
//     load at pixel offset + element offset (table), split into tf32 hi / lo and written to TENSOR MEMORY (lane = pixel,
//     column = kk); the weights become K-major hi / lo tiles in shared memory;
//   * one warp issues the 3xTF32 MMAs, eight drain warps add finished accumulators in fp32 registers and store.
// The rows of all images form one list of rows, so small maps fill their boxes across images.
// What bounds it is the latency of the split warps' shared-memory loads (an instruction every seven clocks); a third group of
// them, paid for with registers, gave nothing.  Tiles of 64 and 32 columns, where an operand element is used less often, were
// slower than the gather (64 channels of 224 x 224: 1830 us against 1774), and so was the forward direction (572 against 567).
// Measured (B200), gather-fed kernel -> this one: 5x5, 96 <- 256 channels, 64 images of 27 x 27 1190 -> 715 us; 3x3, 256 <- 384,
// 128 of 13 x 13 630 -> 494; 3x3, 512 <- 512, 64 of 14 x 14 833 -> 635; 3x3, 256 <- 256, 32 of 56 x 56 1281 -> 1178.
#pragma once

#include "gemm_dense.cuh"

namespace vdnn {
namespace halo {

using tc::BK;
using tc::BM;

constexpr int DRAIN_WARPS = 8, GROUPS = 2, SPLIT_WARPS = 4 * GROUPS, LOAD_WARPS = 3;
constexpr int SPLIT_GROUP = 128, LOADERS = LOAD_WARPS * 32;
constexpr int LOAD_WARP = DRAIN_WARPS + SPLIT_WARPS, MMA_WARP = LOAD_WARP + LOAD_WARPS;
constexpr int THREADS = (MMA_WARP + 1) * 32;
constexpr int MIN_SLOTS = 2, MAX_SLOTS = 4;                      // operand blocks in flight: slots of tensor memory, B tiles
constexpr int SMEM_LIMIT = 227 * 1024;

template <int BN> struct Config {
    static_assert(BN % 32 == 0 && BN >= 96 && BN <= 128, "columns");
    static constexpr int B_BYTES = BN * BK * 4;                  // one of hi / lo
    static constexpr int A_COL = 256;                            // two accumulators below, MAX_SLOTS x 64 columns of A above
    static_assert(2 * BN <= A_COL, "tensor memory");
};

struct Params {
    const float* in;                     // dy: n x cin x h x w
    const float* w;
    float* out;                          // dx: n x n_cols x P x Q
    int n, cin, h, w_in, n_cols, P, Q, R, S, off_h, off_w;
    int bw, bh, boxes_w, rows_total;     // box, boxes per row, n * P rows of dx
    int v_height;                        // virtual input rows per image: P - 1 + R
    int rows_max, pitch, plane;          // input region of a box: rows, elements per row, elements per channel
    int chunk_c, chunk_total;            // filters per chunk, chunks
    int slots;                           // operand blocks in flight
    int b_pitch, b_vec;                  // raw weights: floats per filter; 16-byte copies allowed
    int a_raw_bytes, raw_bytes;          // bytes of the input part and of a whole raw stage
    FastDiv div_bw, div_P, div_V, div_pitch;
    long long units;
    int tiles_n, tiles_m;
    float alpha, beta;
};

__device__ __forceinline__ void cp4(uint32_t dst, const float* src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

// What a unit (row tile, column tile) is; the same for every role.
struct Unit { int g0, box, n0; };
__device__ __forceinline__ Unit unit_of(const Params& p, long long u, int bn) {
    Unit t;
    const int nt = static_cast<int>(u % p.tiles_n), tile = static_cast<int>(u / p.tiles_n);
    const int rt = tile / p.boxes_w;
    t.box = tile - rt * p.boxes_w;
    t.g0 = rt * p.bh;
    t.n0 = nt * bn;
    return t;
}

// A chunk's ceil(chunk_c * R * S / 8) k slices of 8 are dealt evenly to the fewest operand blocks ("items") of at most four
// slices.  All chunks have the same shape: filters past the tensor's last, and elements past a chunk's last, are zeros.
template <int BN>
__global__ void __launch_bounds__(THREADS, 1) dgrad_kernel(const Params p) {
    typedef Config<BN> Cfg;
    extern __shared__ char smem_raw[];
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    char* raw = tiles + p.slots * 2 * Cfg::B_BYTES;
    const int rs = p.R * p.S, kc = p.chunk_c * rs, slices = (kc + 7) >> 3, items = (slices + 3) >> 2;
    int* a_off = reinterpret_cast<int*>(raw + 2 * p.raw_bytes);      // [slices * 8] element (k, r, s) of a chunk: offset in the input region
    int* b_off = a_off + slices * 8;                                 // [slices * 8] ... and in the raw weights
    uint64_t* raw_full = reinterpret_cast<uint64_t*>(b_off + slices * 8);      // [2] copies have landed
    uint64_t* raw_empty = raw_full + 2;             // [2] split warps are through
    uint64_t* split_full = raw_empty + 2;           // [MAX_SLOTS]
    uint64_t* empty = split_full + MAX_SLOTS;       // [MAX_SLOTS] the MMAs have read the slot
    uint64_t* acc_ready = empty + MAX_SLOTS;        // [2]
    uint64_t* acc_free = acc_ready + 2;             // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 2);
    const int unit_items = items * p.chunk_total;

    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t == 0) {
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(tc::smem_u32(&raw_full[s]), LOADERS);
            tc::mbar_init(tc::smem_u32(&raw_empty[s]), SPLIT_WARPS);
            tc::mbar_init(tc::smem_u32(&acc_ready[s]), 1);
            tc::mbar_init(tc::smem_u32(&acc_free[s]), DRAIN_WARPS);
        }
        for (int s = 0; s < MAX_SLOTS; ++s) { tc::mbar_init(tc::smem_u32(&split_full[s]), SPLIT_GROUP); tc::mbar_init(tc::smem_u32(&empty[s]), 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int kk = t; kk < slices * 8; kk += THREADS) {
        const int c = kk / rs, tap = kk - c * rs, r = tap / p.S, s = tap - r * p.S;
        a_off[kk] = kk < kc ? c * p.plane + r * p.pitch + s : 0;
        b_off[kk] = kk < kc ? c * p.b_pitch + rs - 1 - tap : 0;
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    // pixel `row` of the unit's box: its image, output row and column; false where the box reaches past the tensor
    auto pixel_of = [&](const Unit& u, int row, uint32_t* n, uint32_t* y, int* x) -> bool {
        uint32_t i, j;
        p.div_bw.divmod(row, i, j);
        const uint32_t g = u.g0 + i;
        p.div_P.divmod(g, *n, *y);
        *x = u.box * p.bw + static_cast<int>(j);
        return static_cast<int>(i) < p.bh && static_cast<int>(g) < p.rows_total;
    };

    if (warp < DRAIN_WARPS) {
        // ------------------------------------------------------------------ accumulator drain + epilogue
        constexpr int NACC = BN / 2;
        const int col_beg = (warp >> 2) * NACC;
        const uint32_t tmem_mine = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(col_beg);
        const size_t pq = static_cast<size_t>(p.P) * p.Q;
        unsigned pair = 0;
        bool alive = true;
        for (long long uu = blockIdx.x; uu < p.units && alive; uu += gridDim.x) {
            const Unit u = unit_of(p, uu, BN);
            float acc[NACC];
#pragma unroll
            for (int j = 0; j < NACC; ++j) acc[j] = 0.0f;
            for (int i = 0; i < unit_items && alive; i += 2, ++pair) {
                const int b = pair & 1;
                bool ok = tc::mbar_wait(tc::smem_u32(&acc_ready[b]), (pair >> 1) & 1u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { atomicCAS(&tc::g_tc_error, 0, 103); alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c = 0; c < NACC; c += 16) {
                    float v[16];
                    tc::tmem_ld16(tmem_mine + static_cast<uint32_t>(b * BN + c), v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c + j] += v[j];
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(tc::smem_u32(&acc_free[b]));
            }
            uint32_t n, y;
            int x;
            const bool in = pixel_of(u, (warp & 3) * 32 + lane, &n, &y, &x);
            if (!alive || !in || x >= p.Q) continue;
            float* o = p.out + (static_cast<size_t>(n) * p.n_cols + u.n0 + col_beg) * pq + static_cast<size_t>(y) * p.Q + x;
            const int cols = p.n_cols - u.n0 - col_beg;
#pragma unroll
            for (int j = 0; j < NACC; ++j) {
                if (j < cols) {
                    const float v = p.alpha * acc[j];
                    *o = p.beta != 0.0f ? fmaf(p.beta, *o, v) : v;
                }
                o += pq;
            }
        }
    } else if (warp < LOAD_WARP) {
        // ------------------------------------------------------------------ split: group g takes every GROUPS-th item
        const unsigned g = (warp - DRAIN_WARPS) >> 2;
        const int row = (warp & 3) * 32 + lane;
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + Cfg::A_COL;
        unsigned item = 0, chunk = 0, slot = 0, slot_phase = 0;
        bool alive = true;
        for (long long uu = blockIdx.x; uu < p.units && alive; uu += gridDim.x) {
            const Unit u = unit_of(p, uu, BN);
            uint32_t n0, y0, n, y;
            int x;
            pixel_of(u, 0, &n0, &y0, &x);
            const bool in = pixel_of(u, row, &n, &y, &x);
            const int pix = in ? static_cast<int>((n - n0) * p.v_height + y - y0) * p.pitch + (x - u.box * p.bw) : 0;
            for (int c = 0; c < p.chunk_total && alive; ++c, ++chunk) {
                const int st = chunk & 1;
                bool ok = tc::mbar_wait(tc::smem_u32(&raw_full[st]), (chunk >> 1) & 1u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { atomicCAS(&tc::g_tc_error, 0, 101); alive = false; break; }
                const float* a_raw = reinterpret_cast<const float*>(raw + st * p.raw_bytes) + pix;
                const float* b_raw = reinterpret_cast<const float*>(raw + st * p.raw_bytes + p.a_raw_bytes) + row * rs;
                for (int i = 0; i < items; ++i, ++item) {
                    const unsigned my_slot = slot, my_phase = slot_phase;
                    if (++slot == static_cast<unsigned>(p.slots)) { slot = 0; slot_phase ^= 1u; }
                    if (item % GROUPS != g) continue;
                    // (a group's last item, GROUPS back, saw slots + GROUPS items back finished: with at least GROUPS slots this
                    // barrier is never two phases behind, where a parity wait would pass at once)
                    ok = tc::mbar_wait(tc::smem_u32(&empty[my_slot]), my_phase ^ 1u);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { atomicCAS(&tc::g_tc_error, 0, 101); alive = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const int s_beg = i * slices / items, s_end = (i + 1) * slices / items;
                    const uint32_t slot_col = tmem_lane + my_slot * (2 * BK);
                    char* b_hi = tiles + my_slot * (2 * Cfg::B_BYTES);
                    for (int s = s_beg; s < s_end; ++s) {
                        const int kk = s * 8;
                        const int4 o0 = *reinterpret_cast<const int4*>(a_off + kk), o1 = *reinterpret_cast<const int4*>(a_off + kk + 4);
                        float v[8] = {a_raw[o0.x], a_raw[o0.y], a_raw[o0.z], a_raw[o0.w], a_raw[o1.x], a_raw[o1.y], a_raw[o1.z], a_raw[o1.w]};
                        if (kk + 8 > kc) {
#pragma unroll
                            for (int e = 0; e < 8; ++e) if (kk + e >= kc) v[e] = 0.0f;
                        }
                        float hi[8], lo[8];
#pragma unroll
                        for (int e = 0; e < 8; e += 2) tc::split_tf32_x2(v[e], v[e + 1], hi[e], hi[e + 1], lo[e], lo[e + 1]);
                        tmem_st8(slot_col + (s - s_beg) * 8, hi);
                        tmem_st8(slot_col + BK + (s - s_beg) * 8, lo);
                    }
                    if (BN >= SPLIT_GROUP || row < BN) {
                        for (int s = s_beg; s < s_end; ++s) {
                            const int kk = s * 8;
                            const int4 o0 = *reinterpret_cast<const int4*>(b_off + kk), o1 = *reinterpret_cast<const int4*>(b_off + kk + 4);
                            float v[8] = {b_raw[o0.x], b_raw[o0.y], b_raw[o0.z], b_raw[o0.w], b_raw[o1.x], b_raw[o1.y], b_raw[o1.z], b_raw[o1.w]};
                            if (kk + 8 > kc) {
#pragma unroll
                                for (int e = 0; e < 8; ++e) if (kk + e >= kc) v[e] = 0.0f;
                            }
                            float4 h0, h1, l0, l1;
                            tc::split_tf32_x2(v[0], v[1], h0.x, h0.y, l0.x, l0.y);
                            tc::split_tf32_x2(v[2], v[3], h0.z, h0.w, l0.z, l0.w);
                            tc::split_tf32_x2(v[4], v[5], h1.x, h1.y, l1.x, l1.y);
                            tc::split_tf32_x2(v[6], v[7], h1.z, h1.w, l1.z, l1.w);
                            const uint32_t w0 = tc::swz(row, (s - s_beg) * 2), w1 = tc::swz(row, (s - s_beg) * 2 + 1);
                            *reinterpret_cast<float4*>(b_hi + w0) = h0;
                            *reinterpret_cast<float4*>(b_hi + w1) = h1;
                            *reinterpret_cast<float4*>(b_hi + Cfg::B_BYTES + w0) = l0;
                            *reinterpret_cast<float4*>(b_hi + Cfg::B_BYTES + w1) = l1;
                        }
                    }
                    __syncwarp();
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    tc::mbar_arrive(tc::smem_u32(&split_full[my_slot]));
                }
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(tc::smem_u32(&raw_empty[st]));
            }
        }
    } else if (warp < MMA_WARP) {
        // ------------------------------------------------------------------ loaders: input region and raw weights of a chunk
        const int lt = t - LOAD_WARP * 32;
        const int region = p.rows_max * p.pitch;
        const size_t hw = static_cast<size_t>(p.h) * p.w_in;
        unsigned chunk = 0;
        bool alive = true;
        for (long long uu = blockIdx.x; uu < p.units && alive; uu += gridDim.x) {
            const Unit u = unit_of(p, uu, BN);
            uint32_t n0, y0;
            p.div_P.divmod(u.g0, n0, y0);
            const uint32_t v0 = n0 * p.v_height + y0;
            const int x0 = u.box * p.bw + p.off_w;
            for (int c = 0; c < p.chunk_total && alive; ++c, ++chunk) {
                const int st = chunk & 1;
                if (!tc::mbar_wait(tc::smem_u32(&raw_empty[st]), ((chunk >> 1) & 1u) ^ 1u)) { atomicCAS(&tc::g_tc_error, 0, 101); alive = false; break; }
                const uint32_t a_dst = tc::smem_u32(raw + st * p.raw_bytes), b_dst = a_dst + p.a_raw_bytes;
                const int c0 = c * p.chunk_c, nc = min(p.chunk_c, p.cin - c0);       // filters past the last are zero-filled
                for (int pos = lt; pos < region; pos += LOADERS) {
                    uint32_t v, col, n, r;
                    p.div_pitch.divmod(pos, v, col);
                    p.div_V.divmod(v0 + v, n, r);
                    const int iy = static_cast<int>(r) + p.off_h, ix = x0 + static_cast<int>(col);
                    const bool in = static_cast<int>(n) < p.n && static_cast<unsigned>(iy) < static_cast<unsigned>(p.h) &&
                                    static_cast<unsigned>(ix) < static_cast<unsigned>(p.w_in);
                    const float* src = in ? p.in + (static_cast<size_t>(n) * p.cin + c0) * hw + static_cast<size_t>(iy) * p.w_in + ix : p.in;
                    const size_t step = in ? hw : 0;
                    uint32_t dst = a_dst + pos * 4;
                    for (int k = 0; k < nc; ++k, src += step, dst += p.plane * 4) cp4(dst, src, in);
                    for (int k = nc; k < p.chunk_c; ++k, dst += p.plane * 4) cp4(dst, p.in, false);
                }
                // raw weights: chunk_c filters, of each the R * S taps of BN columns
                const int len = BN * rs, len_in = min(BN, p.n_cols - u.n0) * rs;
                const size_t w_pitch = static_cast<size_t>(p.n_cols) * rs;
                for (int r = 0; r < p.chunk_c; ++r) {
                    const bool row_in = r < nc;
                    const float* src = row_in ? p.w + (c0 + r) * w_pitch + static_cast<size_t>(u.n0) * rs : p.w;
                    const uint32_t dst = b_dst + r * p.b_pitch * 4;
                    if (p.b_vec) {
                        for (int e = lt * 4; e < len; e += LOADERS * 4) {
                            const int bytes = row_in ? max(0, min(16, (len_in - e) * 4)) : 0;
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + e * 4), "l"(bytes ? src + e : p.w), "r"(bytes) : "memory");
                        }
                    } else {
                        for (int e = lt; e < len; e += LOADERS) {
                            const bool in = row_in && e < len_in;
                            cp4(dst + e * 4, in ? src + e : p.w, in);
                        }
                    }
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(&raw_full[st])) : "memory");
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else {
        // ------------------------------------------------------------------ MMA issuer (tc::elect_one)
        const bool elected = tc::elect_one();
        constexpr uint32_t IDESC = dense::Config<64, false>::idesc(BN);
        unsigned pair = 0, slot = 0, slot_phase = 0;
        bool ok = true;
        for (long long uu = blockIdx.x; uu < p.units && ok; uu += gridDim.x) {
            const Unit u = unit_of(p, uu, BN);
            int done = 0;
            for (int c = 0; c < p.chunk_total && ok; ++c) {
                for (int i = 0; i < items; ++i) {
                    const int b = pair & 1;
                    const bool fresh = !(done & 1);
                    if (fresh && pair >= 2 && !tc::mbar_wait(tc::smem_u32(&acc_free[b]), ((pair >> 1) - 1) & 1u)) { ok = false; break; }
                    if (!tc::mbar_wait(tc::smem_u32(&split_full[slot]), slot_phase)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t b_hi = tc::smem_u32(tiles + slot * (2 * Cfg::B_BYTES));
                    const uint64_t dbh = tc::make_desc(b_hi), dbl = tc::make_desc(b_hi + Cfg::B_BYTES);
                    const uint32_t a = tmem_base + Cfg::A_COL + slot * (2 * BK), d = tmem_base + static_cast<uint32_t>(b * BN);
                    const int ns = (i + 1) * slices / items - i * slices / items;
                    ++done;
                    const bool last = !fresh || done == unit_items;
                    if (elected) {
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks) {
                            if (ks < ns) {
                                const uint32_t add = (fresh && ks == 0) ? 0u : 1u;
                                dense::mma_tf32_ta(d, a + BK + ks * 8, dbh + ks * 2, IDESC, add);
                                dense::mma_tf32_ta(d, a + ks * 8, dbl + ks * 2, IDESC, 1u);
                                dense::mma_tf32_ta(d, a + ks * 8, dbh + ks * 2, IDESC, 1u);
                            }
                        }
                        tc::mma_commit(tc::smem_u32(&empty[slot]));
                        if (last) tc::mma_commit(tc::smem_u32(&acc_ready[b]));
                    }
                    __syncwarp();
                    if (last) ++pair;
                    if (++slot == static_cast<unsigned>(p.slots)) { slot = 0; slot_phase ^= 1u; }
                }
            }
        }
        if (!ok) atomicCAS(&tc::g_tc_error, 0, 102);
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// Clocks of one 8-wide k slice on tiles of bn columns (measured: an MMA of 96 columns takes 50 clocks, of 128 columns 64).
inline int slice_clocks(int bn) { return bn == 96 ? 150 : 192; }

// Columns of a tile: those with the least work in all; 0 where most of a tile would be padding.
inline int tile_n(int cols) {
    if (cols <= 64) return 0;
    return ceil_div(cols, 96) * slice_clocks(96) < ceil_div(cols, 128) * slice_clocks(128) ? 96 : 128;
}

// One problem: what the kernel's parameters are made from.
struct Problem {
    int n, cin, h, w;                    // dy
    int n_cols, P, Q;                    // dx
    int R, S, off_h, off_w;              // dy row of dx row y under (reversed) tap r: y + off_h + r
};

// Rows of the input region of a box of bh output rows, wherever it starts in an image: one per row, R - 1 more, and R - 1 more
// again at each boundary between images that it can cross.
inline int region_rows(const Problem& q, int bh) {
    const int crossed = (q.P + bh - 2) / q.P;
    return bh + (q.R - 1) * (1 + (crossed < q.n - 1 ? crossed : q.n - 1));
}

// Shared-memory loads of a warp's 32 pixels: the most that fall into one bank, for a row pitch.
inline int bank_conflicts(int bw, int bh, int pitch) {
    int most = 0;
    for (int w = 0; w < 4; ++w) {
        int bank[32] = {0};
        for (int l = 0; l < 32; ++l) {
            const int m = w * 32 + l;
            if (m >= bw * bh) break;
            const int b = ((m / bw) * pitch + m % bw) & 31;
            if (++bank[b] > most) most = bank[b];
        }
    }
    return most;
}

// Chooses box, chunk and slots; false where no choice fits (a region too large for shared memory).
inline bool plan(const Problem& q, int bn, Params* p) {
    const int rs = q.R * q.S;
    const long long rows = static_cast<long long>(q.n) * q.P;
    const long long v_rows = static_cast<long long>(q.n) * (q.P - 1 + static_cast<long long>(q.R));
    if (rows > 0x3fffffffLL || v_rows > 0x3fffffffLL) return false;
    // The box with the least work: tiles, plus the region that each of them loads.
    double best = -1.0;
    for (int k = 1; k <= q.Q; ++k) {
        const int bw = ceil_div(q.Q, k);
        if (bw > BM || (k > 1 && bw == ceil_div(q.Q, k - 1))) continue;
        const int bh = BM / bw < rows ? BM / bw : static_cast<int>(rows);
        const int rr = region_rows(q, bh), cols = bw - 1 + q.S;
        const double cost = static_cast<double>(ceil_div<long long>(rows, bh)) * k * (128.0 + 0.04 * rr * cols);
        if (best < 0.0 || cost < best) {
            best = cost;
            p->bw = bw; p->bh = bh; p->boxes_w = k; p->rows_max = rr; p->pitch = cols;
        }
        if (bw <= 4) break;
    }
    if (best < 0.0) return false;
    const int cols = p->pitch;
    for (int extra = 0, conflicts = 99; extra < 8 && conflicts > 1; ++extra) {
        const int c = bank_conflicts(p->bw, p->bh, cols + extra);
        if (c < conflicts) { conflicts = c; p->pitch = cols + extra; }
    }
    p->plane = p->rows_max * p->pitch;
    // Filters per chunk: the fewest clocks for the whole reduction -- filters rounded up to whole chunks, elements to whole
    // slices, about 60 clocks of hand-over per item and 200 per chunk -- among those that leave room for two raw stages and
    // a slot for each split group.
    const int b_tile = 2 * bn * BK * 4, pitch = ceil_div(bn * rs, 4) * 4;
    double least = -1.0;
    for (int cc = 1; cc <= 64 && cc <= q.cin; ++cc) {
        const int slices = ceil_div(cc * rs, 8), items = ceil_div(slices, 4);
        const long long a_raw = (static_cast<long long>(cc) * p->plane * 4 + 15) / 16 * 16;
        const long long raw = a_raw + static_cast<long long>(cc) * pitch * 4;
        const long long fixed = 2 * raw + 2LL * slices * 8 * 4 + 1024 + 256;
        const long long slots = (SMEM_LIMIT - fixed) / b_tile;
        if (fixed > SMEM_LIMIT || slots < MIN_SLOTS) break;
        const double cost = ceil_div(q.cin, cc) * (static_cast<double>(slices) * slice_clocks(bn) + 60.0 * items + 200.0);
        if (least < 0.0 || cost < least) {
            least = cost;
            p->chunk_c = cc; p->b_pitch = pitch; p->a_raw_bytes = static_cast<int>(a_raw); p->raw_bytes = static_cast<int>(raw);
            p->slots = slots > MAX_SLOTS ? MAX_SLOTS : static_cast<int>(slots);
        }
    }
    if (least < 0.0) return false;
    p->chunk_total = ceil_div(q.cin, p->chunk_c);
    p->tiles_m = static_cast<int>(ceil_div<long long>(rows, p->bh)) * p->boxes_w;
    p->tiles_n = ceil_div(q.n_cols, bn);
    p->units = static_cast<long long>(p->tiles_m) * p->tiles_n;
    return true;
}

// Fills in what the plan does not depend on.
inline void complete(const Problem& q, const float* in, const float* w, Params* p) {
    p->in = in; p->w = w;
    p->n = q.n; p->cin = q.cin; p->h = q.h; p->w_in = q.w; p->n_cols = q.n_cols; p->P = q.P; p->Q = q.Q; p->R = q.R; p->S = q.S;
    p->off_h = q.off_h; p->off_w = q.off_w;
    p->rows_total = q.n * q.P;
    p->v_height = q.P - 1 + q.R;
    p->div_bw = FastDiv(p->bw); p->div_P = FastDiv(q.P); p->div_V = FastDiv(p->v_height); p->div_pitch = FastDiv(p->pitch);
    p->b_vec = static_cast<size_t>(q.n_cols) * q.R * q.S % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0;
}

template <int BN>
int launch_bn(const Params& p, cudaStream_t stream) {
    const int slices = ceil_div(p.chunk_c * p.R * p.S, 8);
    const int smem = p.slots * 2 * Config<BN>::B_BYTES + 2 * p.raw_bytes + 2 * slices * 8 * 4 + 1024 + 256;
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
    auto kern = dgrad_kernel<BN>;
    VDNN_ALLOW_SHARED(dev, kern, SMEM_LIMIT);
    const int grid = static_cast<int>(p.units < sm_count() ? p.units : sm_count());
    kern<<<grid, THREADS, smem, stream>>>(p);
    VDNN_LAUNCHED();
    return VDNN_OK;
}

inline int launch(int bn, const Params& p, cudaStream_t stream) {
    if (bn == 96) return launch_bn<96>(p, stream);
    return launch_bn<128>(p, stream);
}

}  // namespace halo
}  // namespace vdnn
