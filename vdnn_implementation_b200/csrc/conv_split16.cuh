// TMA-fed convolution kernels for sm_100a (PERF_OPT, stride 1) on operands split into pairs of f16 (split16.cuh).
//
// Passes bound by bandwidth rewrite the gathered tensors once per call as lists of positions in workspace: image after image,
// row after row, every row followed by zero positions and every image by zero rows, wide enough that a filter tap's shift never
// reaches real data of a neighbouring row or image (the zeros are the padding).  Position q holds blocks of 64 channels, 128
// bytes each, in a hi and a lo list.  A tap is then a constant shift of the list, no matter which of the three products is
// formed, and all of them use the lists in one geometry (list_geometry).
//
// The contraction kernels spend no instruction on operand elements: a warp of its own issues tensor copies that complete a
// stage's "full" barrier by byte count, one thread issues the MMAs, and 16 warps add each finished accumulator (two or three
// blocks of 64 of the reduction, 24 chained MMAs) into fp32 registers and run the epilogue.  All barrier waits are bounded.
//   strip_kernel   forward and data gradient.  An output tile is 128 or 256 consecutive positions x BN columns; the operand tiles
//                  of the taps of one filter row are windows, one position apart, of ONE strip of 128 + S - 1 positions, which
//                  is fetched once and read through descriptors that start S * 128 bytes apart (the tensor core derives the
//                  swizzle phase of a row from its address, so a window needs nothing but its start address).
//   wgrad_kernel   filter gradient: the reduction runs over positions, both operands are MN-major; the 128 rows of a tile are
//                  two groups of (tap, 64-channel block), and groups of one filter row share a strip likewise.
// CTAS = 2: on pairs of CTAs (clusters of two on neighbouring SMs, tcgen05 cta_group::2).  Each CTA stages its own 128 rows and
// half of the column operand; copies complete on the leader's barrier, which the leader arms with the bytes of both; one thread
// of the leader issues the MMAs and its commits arrive in both CTAs; each CTA drains its own rows, and hands the accumulator back
// by a remote arrival; tensor memory is allocated and released by the same warp of both, around cluster barriers.
//
// What bounds them (B200, batch 32, whole calls with all passes, us; in parentheses the same layer on pairs of tf32 values,
// which these kernels replaced):
//   512 -> 512 @ 28 x 28    forward 277 (465), three gradients 588 (1013): tensor pipe at 86 % of its active cycles, at 1.54 GHz
//                           under the power cap
//   128 -> 128 @ 112 x 112  360 (644), 779 (1428): an MMA of 128 columns takes 93 clocks, not 64
//   64 -> 64 @ 224 x 224    530 (805), 1285 (2197): half of it passes over the operands at 5.3 .. 6.7 TB/s; an MMA of 64 columns
//                           takes 65 clocks
// What was measured and not taken: 64 columns on pairs (410 against 325 us for the kernel alone), with the filters of all taps
// resident in shared memory (363), L2 prefetches of the next strips (no change), chains of one block of 64 (7 % slower in the
// filter gradient of 512 filters), the filter gradient of 128 filters on pairs (2 % slower).
//
// No copy carries a cluster multicast qualifier, and every tensor map covers this GPU's own workspace only.
#pragma once

#include <atomic>

#include "split16.cuh"
#include "tensor_map.cuh"

namespace vdnn {
namespace split16 {

constexpr int BM = 128;
constexpr int DRAIN_WARPS = 16;
constexpr int THREADS = (DRAIN_WARPS + 2) * 32;      // + the copying warp and the issuing warp
constexpr int STRIP_TAPS = 9;                        // taps of a filter row that share a strip; wider filters take a strip per tap
constexpr int SMEM_LIMIT = 227 * 1024;

// One product over a gathered tensor: list row of output row y under tap r is y + tap_sign * r + off_h (columns likewise).
struct Problem {
    int n, cin, in_h, in_w;        // the gathered tensor (x for forward, dy for the data gradient)
    int out_h, out_w, n_cols;      // output grid and channels
    int R, S, tap_sign, off_h, off_w;
    int wp, lp;                    // list geometry of the layer
    Fold fold;                     // strided layers: the tensor x or dx, whose folded form the above describes
};

inline int padded_channels(int c) { return ceil_div(c, KB) * KB; }

__device__ __forceinline__ uint32_t cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Every thread of the block, or of both blocks of a pair.
template <int CTAS>
__device__ __forceinline__ void sync_all() {
    if constexpr (CTAS == 2) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else __syncthreads();
}
// A barrier of the leader (rank 0), as copies and remote arrivals of either CTA name it.
template <int CTAS>
__device__ __forceinline__ uint32_t leader_bar(const void* bar) {
    uint32_t a = tc::smem_u32(bar);
    if constexpr (CTAS == 2) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(a), "r"(0));
    return a;
}
template <int CTAS>
__device__ __forceinline__ void arrive_leader(uint32_t bar) {
    if constexpr (CTAS == 2) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
    else tc::mbar_arrive(bar);
}
// Once the MMAs issued so far have completed: an arrival on the barrier at this offset in every CTA.
template <int CTAS>
__device__ __forceinline__ void commit_all(const void* bar) {
    if constexpr (CTAS == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     ::"r"(tc::smem_u32(bar)), "h"(static_cast<uint16_t>(3)) : "memory");
    else tc::mma_commit(tc::smem_u32(bar));
}
template <int CTAS>
__device__ __forceinline__ void load_rows(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int row) {
    if constexpr (CTAS == 2)
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                     ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(row) : "memory");
    else tma::tma_load_rows(dst, map, bar, c0, row);
}
__device__ __forceinline__ void expect_bytes(const void* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(bar)), "r"(bytes) : "memory");
}
template <int CTAS>
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t columns) {
    if constexpr (CTAS == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(slot)), "r"(columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(slot)), "r"(columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}
template <int CTAS>
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t columns) {
    if constexpr (CTAS == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns) : "memory");
}

// ---- forward and data gradient ------------------------------------------------------------------------------------

struct StripParams {
    int wp, lp;                          // positions per row and per image
    long long total_pos;                 // n * lp
    FastDiv div_lp, div_wp;
    int out_h, out_w, n_cols;            // output grid and channels
    int S, cblocks;                      // taps per filter row and 64-channel blocks of the reduction
    int dh0, dh_step, row0, row_step;    // tap (r, s): strip starts dh0 + dh_step * r rows of wp above/below, window at row row0 + row_step * s
    int dw_min;                          // column shift of the strip's first row
    int groups_total, group_chunk;       // groups = (r, channel block); each split walks group_chunk of them
    int inner;                           // taps served by one strip: S, or 1 (one strip per tap: groups = (tap, channel block))
    int kblocks_total;
    float* out;
    const float* bias;
    float alpha, beta;
    int mode;
    size_t partial_stride;
    const Scales* scales;
    int product;
    Fold fold;                           // data gradient of a strided layer: where the columns lie in dx
};

constexpr int STRIP_HALF_BYTES = (BM + 8) * ROW_BYTES;             // 136 rows of 128 bytes, a multiple of the swizzle period

// BN columns, MH halves of 128 positions per CTA, CTAS CTAs.
template <int BN, int MH, int CTAS> struct StripConfig {
    static constexpr bool MERGED = BN == 64 && CTAS == 1;
    static constexpr int ACC_COLS = MERGED ? 2 * BN : BN;
    static constexpr int COLS_HERE = BN / CTAS;                         // columns this CTA stages
    static constexpr int B_TILE_BYTES = COLS_HERE * ROW_BYTES;
    static constexpr int A_STAGE_BYTES = MH * 2 * STRIP_HALF_BYTES;
    static constexpr int B_STAGE_BYTES = 2 * B_TILE_BYTES;
    static constexpr int SA = 2, SB = 4;                                // strips and filter tiles in shared memory
    static constexpr int CHAIN = MERGED ? 3 : 2;                        // k blocks per accumulator hand-over
    static constexpr int BUFS = 512 / (MH * ACC_COLS);    // accumulators: what the drain may lag behind
    static constexpr int TMEM_COLS = BUFS * MH * ACC_COLS;
    static constexpr int SMEM_BYTES = SA * A_STAGE_BYTES + SB * B_STAGE_BYTES + 1024 + 256;
    static constexpr uint32_t IDESC = idesc(BM * CTAS, BN, false);
    static constexpr uint32_t IDESC_WIDE = idesc(BM, 2 * BN <= 256 ? 2 * BN : 256, false);
    static_assert(TMEM_COLS <= 512 && SMEM_BYTES <= SMEM_LIMIT, "");
};

// Columns (c, a, b) of position (y, x) of a folded dx: pixel (s y + a - pad_h, s x + b - pad_w) of channel c.
template <int N>
__device__ __forceinline__ void store_folded(const StripParams& p, const uint64_t (&acc)[N], int col0, int n, int y, int x, const Unscale& value) {
    const int s = p.fold.s;
    int t = col0 / s, b = col0 - t * s, c = t / s, a = t - c * s;
    float* out = p.out + static_cast<size_t>(n) * p.fold.c * p.fold.h * p.fold.w;
    if (p.mode == EPI_PARTIAL) out += static_cast<size_t>(blockIdx.z) * p.partial_stride;
#pragma unroll
    for (int j = 0; j < 2 * N; ++j) {
        const int h = s * y + a - p.fold.pad_h, w = s * x + b - p.fold.pad_w;
        if (col0 + j < p.n_cols && static_cast<unsigned>(h) < static_cast<unsigned>(p.fold.h) && static_cast<unsigned>(w) < static_cast<unsigned>(p.fold.w)) {
            float* dst = out + (static_cast<size_t>(c) * p.fold.h + h) * p.fold.w + w;
            float v = value(sum_of(acc, j));
            if (p.beta != 0.0f) v = fmaf(p.beta, *dst, v);
            *dst = v;
        }
        if (++b == s) { b = 0; if (++a == s) { a = 0; ++c; } }
    }
}

template <int BN, int MH, int CTAS>
__global__ void __launch_bounds__(THREADS, 1)
strip_kernel(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo, const __grid_constant__ CUtensorMap map_b,
             const StripParams p) {
    typedef StripConfig<BN, MH, CTAS> Cfg;
    constexpr int SA = Cfg::SA, SB = Cfg::SB, BUFS = Cfg::BUFS;
    constexpr int TILE_ROWS = BM * MH * CTAS;
    extern __shared__ char smem_raw[];
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    char* b_ring = tiles + SA * Cfg::A_STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(b_ring + SB * Cfg::B_STAGE_BYTES);
    uint64_t* a_full = bars;               // [SA]  in the leader
    uint64_t* a_empty = a_full + SA;       // [SA]
    uint64_t* b_full = a_empty + SA;       // [SB]  in the leader
    uint64_t* b_empty = b_full + SB;       // [SB]
    uint64_t* acc_ready = b_empty + SB;    // [BUFS]
    uint64_t* acc_free = acc_ready + BUFS; // [BUFS]  in the leader
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + BUFS);

    // Persistent along x: a CTA (pair) walks every gridDim-th output tile of its column tile (blockIdx.y) and split of the
    // reduction (blockIdx.z).  The three roles loop over the tiles independently and keep their ring and accumulator counters
    // running, so the next tile's loads are in flight, and its first MMAs issued, while a tile's results are being stored.
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const uint32_t rank = CTAS == 2 ? cta_rank() : 0u;
    const bool leader = rank == 0;
    const unsigned first = blockIdx.x / CTAS, step = gridDim.x / CTAS;
    const int n0 = blockIdx.y * BN;
    const int g_beg = blockIdx.z * p.group_chunk;
    const int g_end = min(p.groups_total, g_beg + p.group_chunk);
    const int ngroups = g_beg < g_end ? g_end - g_beg : 0;
    const int nkb = ngroups * p.inner;                 // k blocks per tile
    const uint32_t strip_bytes = static_cast<uint32_t>(BM + p.inner - 1) * ROW_BYTES;

    if (t == 0) {
        for (int s = 0; s < SA; ++s) { tc::mbar_init(tc::smem_u32(&a_full[s]), 1); tc::mbar_init(tc::smem_u32(&a_empty[s]), 1); }
        for (int s = 0; s < SB; ++s) { tc::mbar_init(tc::smem_u32(&b_full[s]), 1); tc::mbar_init(tc::smem_u32(&b_empty[s]), 1); }
        for (int b = 0; b < BUFS; ++b) { tc::mbar_init(tc::smem_u32(&acc_ready[b]), 1); tc::mbar_init(tc::smem_u32(&acc_free[b]), CTAS * DRAIN_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == DRAIN_WARPS + 1) tmem_alloc<CTAS>(tmem_slot, Cfg::TMEM_COLS);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    sync_all<CTAS>();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    tc::follow_up();            // not before the tensor memory is allocated: a follower could take it and wait for this kernel
    tc::after_predecessor();
    const long long num_tiles = p.scales->wide[p.product] ? 0 : (p.total_pos + TILE_ROWS - 1) / TILE_ROWS;

    if (warp < DRAIN_WARPS) {
        // ------------------------------------------------------------------ accumulator drain + epilogue (this CTA's rows)
        constexpr int NACC = BN / (DRAIN_WARPS / 4);
        const int col_beg = (warp >> 2) * NACC;
        const uint32_t tmem_mine = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(col_beg);
        const size_t plane = static_cast<size_t>(p.out_h) * p.out_w;
        const uint32_t free0 = leader_bar<CTAS>(&acc_free[0]);
        const Unscale value = unscale(p.scales, p.product, p.mode == EPI_PARTIAL ? 1.0f : p.alpha);
        bool alive = true;
        unsigned i = 0;                                     // running count of accumulator hand-overs
        const int handovers = (nkb + Cfg::CHAIN - 1) / Cfg::CHAIN;
        for (long long tile = first; tile < num_tiles && alive; tile += step) {
            uint64_t acc[MH][NACC / 2];
#pragma unroll
            for (int h = 0; h < MH; ++h)
#pragma unroll
                for (int j = 0; j < NACC / 2; ++j) acc[h][j] = 0;
            for (int k = 0; k < handovers && alive; ++k, ++i) {
                const unsigned b = i % BUFS;
                bool ok = tc::mbar_wait(tc::smem_u32(&acc_ready[b]), (i / BUFS) & 1u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { atomicCAS(&tc::g_tc_error, 0, 103); alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int h = 0; h < MH; ++h)
                    drain<NACC, Cfg::MERGED>(tmem_mine + static_cast<uint32_t>((b * MH + h) * Cfg::ACC_COLS), BN, acc[h], [&]() {
                        if (h < MH - 1) return;
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) arrive_leader<CTAS>(free0 + b * 8);
                    });
            }
#pragma unroll
            for (int h = 0; h < MH; ++h) {
                const long long q = tile * TILE_ROWS + (rank * MH + h) * BM + (warp & 3) * 32 + lane;      // this thread's position
                if (!alive || q >= p.total_pos) continue;
                uint32_t n, rem, y, x;
                p.div_lp.divmod(static_cast<uint32_t>(q), n, rem);
                p.div_wp.divmod(rem, y, x);
                if (static_cast<int>(y) >= p.out_h || static_cast<int>(x) >= p.out_w) continue;
                const int col0 = n0 + col_beg;
                if (p.fold.s > 1) {
                    store_folded(p, acc[h], col0, static_cast<int>(n), static_cast<int>(y), static_cast<int>(x), value);
                    continue;
                }
                float* dst = p.out + (static_cast<size_t>(n) * p.n_cols + col0) * plane + static_cast<size_t>(y) * p.out_w + x;
                if (p.mode == EPI_PARTIAL) dst += static_cast<size_t>(blockIdx.z) * p.partial_stride;
                if (p.beta == 0.0f && col0 + NACC <= p.n_cols) {
                    const float* bias = p.bias ? p.bias + col0 : nullptr;
#pragma unroll
                    for (int j = 0; j < NACC; ++j) {
                        const float v = value(sum_of(acc[h], j));
                        *dst = bias ? v + bias[j] : v;
                        dst += plane;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < NACC; ++j) {
                        if (col0 + j < p.n_cols) {
                            float v = value(sum_of(acc[h], j));
                            if (p.bias) v += p.bias[col0 + j];
                            if (p.beta != 0.0f) v = fmaf(p.beta, *dst, v);
                            *dst = v;
                        }
                        dst += plane;
                    }
                }
            }
        }
    } else if (warp == DRAIN_WARPS) {
        // ------------------------------------------------------------------ copies: strips and filter tiles
        const bool elected = tc::elect_one();
        // rows of the packed filters: per (column tile, k block) BN rows of hi, then BN of lo
        const long long b_row0 = static_cast<long long>(blockIdx.y) * p.kblocks_total * (2 * BN) + rank * Cfg::COLS_HERE;
        unsigned i = 0, gcount = 0;                     // running k-block and strip counts (ring positions)
        bool ok = true;
        for (long long tile = first; tile < num_tiles && ok; tile += step) {
            const long long m0 = tile * TILE_ROWS + rank * (BM * MH);
            for (int g = 0; g < ngroups && ok; ++g, ++gcount) {
                const int group = g_beg + g;
                const int outer = group / p.cblocks, cb = group - outer * p.cblocks;
                const int r = p.inner == 1 ? outer / p.S : outer, s_first = p.inner == 1 ? outer - r * p.S : 0;
                const int sa = gcount % SA;
                if (!tc::mbar_wait(tc::smem_u32(&a_empty[sa]), ((gcount / SA) & 1u) ^ 1u)) { ok = false; break; }
                // first row of the strip: the tile's position shifted by the filter row and by the leftmost tap (or, with
                // one strip per tap, by that tap)
                const int row = static_cast<int>(m0 + static_cast<long long>(p.dh0 + p.dh_step * r) * p.wp + p.dw_min +
                                                 (p.inner == 1 ? p.row0 + p.row_step * s_first : 0));
                const uint32_t abar = leader_bar<CTAS>(&a_full[sa]);
                const uint32_t ast = tc::smem_u32(tiles + sa * Cfg::A_STAGE_BYTES);
                if (elected) {
                    if (leader) expect_bytes(&a_full[sa], CTAS * MH * 2u * strip_bytes);
#pragma unroll
                    for (int h = 0; h < MH; ++h) {
                        load_rows<CTAS>(ast + h * 2 * STRIP_HALF_BYTES, &map_hi, abar, cb * KB, row + h * BM);
                        load_rows<CTAS>(ast + h * 2 * STRIP_HALF_BYTES + STRIP_HALF_BYTES, &map_lo, abar, cb * KB, row + h * BM);
                    }
                }
                __syncwarp();
                for (int sx = 0; sx < p.inner; ++sx, ++i) {
                        const int sb = i % SB;
                        if (!tc::mbar_wait(tc::smem_u32(&b_empty[sb]), ((i / SB) & 1u) ^ 1u)) { ok = false; break; }
                        const int kb = (r * p.S + s_first + sx) * p.cblocks + cb;
                        const uint32_t bbar = leader_bar<CTAS>(&b_full[sb]);
                        const uint32_t bst = tc::smem_u32(b_ring + sb * Cfg::B_STAGE_BYTES);
                        const int brow = static_cast<int>(b_row0 + static_cast<long long>(kb) * (2 * BN));
                        if (elected) {
                            if (leader) expect_bytes(&b_full[sb], CTAS * Cfg::B_STAGE_BYTES);
                            load_rows<CTAS>(bst, &map_b, bbar, 0, brow);
                            load_rows<CTAS>(bst + Cfg::B_TILE_BYTES, &map_b, bbar, 0, brow + BN);
                        }
                        __syncwarp();
                    }
            }
        }
        if (!ok) atomicCAS(&tc::g_tc_error, 0, 101);
    } else if (leader) {
        // ------------------------------------------------------------------ MMA issuer (tc::elect_one)
        const bool elected = tc::elect_one();
        unsigned i = 0, gcount = 0, handover = 0;
        bool ok = true;
        // the block before the present one, where its main products are still to be issued
        uint32_t held_a = 0;
        int held_sb = 0, held_sa = 0;
        bool held_strip = false;
        for (long long tile = first; tile < num_tiles && ok; tile += step) {
            int kb_in_tile = 0, in_chain = 0;
            for (int g = 0; g < ngroups && ok; ++g, ++gcount) {
                const int sa = gcount % SA;
                if (!tc::mbar_wait(tc::smem_u32(&a_full[sa]), (gcount / SA) & 1u)) { ok = false; break; }
                const uint32_t a_hi0 = tc::smem_u32(tiles + sa * Cfg::A_STAGE_BYTES);
                for (int sx = 0; sx < p.inner; ++sx, ++i, ++kb_in_tile) {
                    const int sb = i % SB, b = handover % BUFS;
                    // hand-overs h and h - BUFS share an accumulator: the drain warps must have emptied it
                    if (in_chain == 0 && handover >= BUFS && !tc::mbar_wait(tc::smem_u32(&acc_free[b]), (handover / BUFS - 1) & 1u)) { ok = false; break; }
                    if (!tc::mbar_wait(tc::smem_u32(&b_full[sb]), (i / SB) & 1u)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_hi = a_hi0 + (p.inner == 1 ? 0u : static_cast<uint32_t>(p.row0 + p.row_step * sx) * ROW_BYTES);
                    const uint32_t b_hi = tc::smem_u32(b_ring + sb * Cfg::B_STAGE_BYTES);
                    const bool last_tap = sx == p.inner - 1, last = in_chain == Cfg::CHAIN - 1 || kb_in_tile == nkb - 1;
                    if (elected) {
#pragma unroll
                        for (int h = 0; h < MH; ++h) {      // the row halves share the filter tile
                            const uint32_t d = tmem_base + static_cast<uint32_t>((b * MH + h) * Cfg::ACC_COLS);
                            const uint32_t a = a_hi + h * 2 * STRIP_HALF_BYTES;
                            if constexpr (Cfg::MERGED)
                                mma_merged<2>(d, tc::make_desc(a), tc::make_desc(a + STRIP_HALF_BYTES), tc::make_desc(b_hi), Cfg::IDESC, Cfg::IDESC_WIDE, in_chain == 0);
                            else
                                mma_cross<CTAS, 2>(d, tc::make_desc(a), tc::make_desc(a + STRIP_HALF_BYTES), tc::make_desc(b_hi),
                                                   tc::make_desc(b_hi + Cfg::B_TILE_BYTES), Cfg::IDESC, in_chain == 0);
                        }
                        if constexpr (Cfg::MERGED) {
                            commit_all<CTAS>(&b_empty[sb]);
                            if (last_tap) commit_all<CTAS>(&a_empty[sa]);
                        } else if (last) {
                            if (in_chain) {
#pragma unroll
                                for (int h = 0; h < MH; ++h)
                                    mma_main<CTAS, 2>(tmem_base + static_cast<uint32_t>((b * MH + h) * Cfg::ACC_COLS), tc::make_desc(held_a + h * 2 * STRIP_HALF_BYTES),
                                                      tc::make_desc(tc::smem_u32(b_ring + held_sb * Cfg::B_STAGE_BYTES)), Cfg::IDESC, true);
                                commit_all<CTAS>(&b_empty[held_sb]);
                                if (held_strip) commit_all<CTAS>(&a_empty[held_sa]);
                            }
#pragma unroll
                            for (int h = 0; h < MH; ++h)
                                mma_main<CTAS, 2>(tmem_base + static_cast<uint32_t>((b * MH + h) * Cfg::ACC_COLS), tc::make_desc(a_hi + h * 2 * STRIP_HALF_BYTES),
                                                  tc::make_desc(b_hi), Cfg::IDESC, in_chain == 0);
                            commit_all<CTAS>(&b_empty[sb]);
                            if (last_tap) commit_all<CTAS>(&a_empty[sa]);
                        }
                        if (last) commit_all<CTAS>(&acc_ready[b]);
                    }
                    __syncwarp();
                    held_a = a_hi; held_sb = sb; held_sa = sa; held_strip = last_tap;
                    if (last) { in_chain = 0; ++handover; }
                    else ++in_chain;
                }
            }
        }
        if (!ok) atomicCAS(&tc::g_tc_error, 0, 102);
    }

    // a pair: both CTAs are through with each other's shared memory, barriers and tensor memory before either leaves
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    sync_all<CTAS>();
    if (warp == DRAIN_WARPS + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_free<CTAS>(tmem_base, Cfg::TMEM_COLS);
    }
}

// ---- filter gradient ----------------------------------------------------------------------------------------------
//
//   dw[k][c][r][s] = sum over positions q of dy[q][k] * x[q + (r - pad_h) * wp + (s - pad_w)][c]
//
// dy is zero in the gaps, so the sum may run over all positions.  A row group is (64-channel block u, tap): g = u * R * S + tap;
// a CTA takes group_chunk consecutive groups, two to a 128-row tile, up to T tiles, against one slice of dy.  Groups of one
// filter row are windows of one strip of 64 + S - 1 positions (the descriptor's leading-dimension offset takes any distance
// between the two groups of a tile).  On pairs both CTAs take the same taps, of the channel blocks 2 u and 2 u + 1: the
// descriptors of one MMA hold in both.

struct WgradParams {
    int wp;
    int R, S, inner, cblocks;            // inner: taps per strip, S or 1
    int off_h, off_w;                    // x position of dy position q under tap (r, s): q + (r + off_h) * wp + (s + off_w)
    int groups, group_chunk;
    int strips, a_half;                  // strips a stage has room for, bytes of one half of a strip
    int stages;
    int kb_total, kb_chunk;              // 64-position blocks of the reduction, and how many of them one split walks
    int C, n_cols, cols_padded;          // dw is [n_cols][C][R * S]
    float* out;
    float alpha, beta;
    int mode;
    size_t partial_stride;
    const Scales* scales;
    Fold fold;                           // strided layers: the filters as they are
};

constexpr int WGRAD_MAX_STAGES = 6;

template <int BN, int T, int CTAS> struct WgradConfig {
    static constexpr int ACC_COLS = BN;
    static constexpr int DEPTH = 512 / (T * ACC_COLS) > 1 ? 2 : 1;       // accumulators per tile
    static constexpr int SLOTS = DEPTH * T;
    static constexpr int TMEM_COLS = SLOTS * ACC_COLS <= 256 ? 256 : 512;
    static constexpr int CHAIN = 2;                                      // k blocks per accumulator hand-over
    static constexpr int BOXES = BN / CTAS / KB;                         // boxes of 64 filters of dy this CTA stages
    static constexpr int BOX_BYTES = 64 * ROW_BYTES;
    static constexpr int B_BYTES = 2 * BOXES * BOX_BYTES;
    static constexpr uint32_t IDESC = idesc(BM * CTAS, BN, true);
    static_assert(SLOTS * ACC_COLS <= 512, "");
};

template <int BN, int T, int CTAS>
__global__ void __launch_bounds__(THREADS, 1)
wgrad_kernel(const __grid_constant__ CUtensorMap x_hi, const __grid_constant__ CUtensorMap x_lo, const __grid_constant__ CUtensorMap dy_hi,
             const __grid_constant__ CUtensorMap dy_lo, const WgradParams p) {
    typedef WgradConfig<BN, T, CTAS> Cfg;
    constexpr int SLOTS = Cfg::SLOTS, DEPTH = Cfg::DEPTH;
    extern __shared__ char smem_raw[];
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const int a_bytes = p.strips * 2 * p.a_half, stage_bytes = a_bytes + Cfg::B_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + p.stages * stage_bytes);
    uint64_t* full = bars;                            // [stages]  in the leader
    uint64_t* empty = full + WGRAD_MAX_STAGES;        // [stages]
    uint64_t* acc_ready = empty + WGRAD_MAX_STAGES;   // [SLOTS]
    uint64_t* acc_free = acc_ready + SLOTS;           // [SLOTS]   in the leader
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + SLOTS);

    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const uint32_t rank = CTAS == 2 ? cta_rank() : 0u;
    const bool leader = rank == 0;
    const int g0 = static_cast<int>(blockIdx.x / CTAS) * p.group_chunk;
    const int g1 = min(p.groups, g0 + p.group_chunk);
    const int my_tiles = (g1 - g0 + 1) / 2;
    const int n0 = blockIdx.y * BN;
    const int kb_beg = blockIdx.z * p.kb_chunk;
    const int kb_end = min(p.kb_total, kb_beg + p.kb_chunk);

    if (t == 0) {
        for (int s = 0; s < p.stages; ++s) { tc::mbar_init(tc::smem_u32(&full[s]), 1); tc::mbar_init(tc::smem_u32(&empty[s]), 1); }
        for (int b = 0; b < SLOTS; ++b) { tc::mbar_init(tc::smem_u32(&acc_ready[b]), 1); tc::mbar_init(tc::smem_u32(&acc_free[b]), CTAS * DRAIN_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == DRAIN_WARPS + 1) tmem_alloc<CTAS>(tmem_slot, Cfg::TMEM_COLS);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    sync_all<CTAS>();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    tc::follow_up();
    tc::after_predecessor();
    const bool skip = p.scales->wide[FILTER] != 0;
    const int nkb = skip || kb_beg >= kb_end ? 0 : kb_end - kb_beg;

    if (warp < DRAIN_WARPS) {
        constexpr int NACC = BN / (DRAIN_WARPS / 4);
        const int col_beg = (warp >> 2) * NACC;
        const uint32_t tmem_mine = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(col_beg);
        const uint32_t free0 = leader_bar<CTAS>(&acc_free[0]);
        uint64_t acc[T][NACC / 2];
#pragma unroll
        for (int j = 0; j < T; ++j)
#pragma unroll
            for (int c = 0; c < NACC / 2; ++c) acc[j][c] = 0;
        bool alive = true;
        for (int i = 0, c = 0; i < nkb && alive; i += Cfg::CHAIN, ++c) {
            const unsigned at = DEPTH == 2 ? c & 1 : 0, phase = (DEPTH == 2 ? c >> 1 : c) & 1;
#pragma unroll
            for (int j = 0; j < T; ++j) {
                if (j >= my_tiles || !alive) continue;
                const unsigned slot = j * DEPTH + at;
                bool ok = tc::mbar_wait(tc::smem_u32(&acc_ready[slot]), phase);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { atomicCAS(&tc::g_tc_error, 0, 103); alive = false; continue; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                drain<NACC, false>(tmem_mine + slot * Cfg::ACC_COLS, 0, acc[j], [&]() {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) arrive_leader<CTAS>(free0 + slot * 8);
                });
            }
        }
        // this thread's rows: group 2 j + (row >> 6) of the CTA, channel row & 63 of its block
        const Unscale value = unscale(p.scales, FILTER, p.mode == EPI_PARTIAL ? 1.0f : p.alpha);
        const int taps = p.R * p.S, row = (warp & 3) * 32 + lane;
        const size_t crs = p.fold.s > 1 ? static_cast<size_t>(p.fold.c) * p.fold.R * p.fold.S : static_cast<size_t>(p.C) * taps;
#pragma unroll
        for (int j = 0; j < T; ++j) {
            const int group = g0 + 2 * j + (row >> 6);
            if (!alive || skip || group >= g1) continue;
            const int u = group / taps, tap = group - u * taps;
            const int ch = (u * CTAS + static_cast<int>(rank)) * KB + (row & 63);
            if (ch >= p.C) continue;
            float* o = p.out + static_cast<size_t>(ch) * taps + tap;
            if (p.fold.s > 1) {
                const int s = p.fold.s, v = ch / s, c = v / s, r = s * (tap / p.S) + v - c * s, q = s * (tap % p.S) + ch - v * s;
                if (r >= p.fold.R || q >= p.fold.S) continue;
                o = p.out + (static_cast<size_t>(c) * p.fold.R + r) * p.fold.S + q;
            }
            if (p.mode == EPI_PARTIAL) o += static_cast<size_t>(blockIdx.z) * p.partial_stride;
#pragma unroll
            for (int c = 0; c < NACC; ++c) {
                const int col = n0 + col_beg + c;
                if (col < p.n_cols) {
                    float* q = o + static_cast<size_t>(col) * crs;
                    float v = value(sum_of(acc[j], c));
                    if (p.beta != 0.0f) v = fmaf(p.beta, *q, v);
                    *q = v;
                }
            }
        }
    } else if (warp == DRAIN_WARPS) {
        const bool elected = tc::elect_one();
        const int st0 = g0 / p.inner, nstrips = (g1 - 1) / p.inner - st0 + 1, strips_per_u = p.R * p.S / p.inner;
        const int col_boxes = min(BN, p.cols_padded - n0) / KB;                                  // of the CTA or pair
        const int box0 = static_cast<int>(rank) * Cfg::BOXES, my_boxes = max(0, min(Cfg::BOXES, col_boxes - box0));
        const uint32_t strip_bytes = static_cast<uint32_t>(64 + p.inner - 1) * ROW_BYTES;
        // (past the last channel block of an odd number the peer's strips read as zeros: they lie outside the map)
        const uint32_t stage_tx = CTAS * static_cast<uint32_t>(nstrips) * 2u * strip_bytes + static_cast<uint32_t>(2 * col_boxes * Cfg::BOX_BYTES);
        bool ok = true;
        for (int i = 0, s = 0, phase = 1; i < nkb; ++i) {
            if (!tc::mbar_wait(tc::smem_u32(&empty[s]), static_cast<uint32_t>(phase))) { ok = false; break; }
            const long long q0 = static_cast<long long>(kb_beg + i) * 64;           // first dy position of the block
            const uint32_t bar = leader_bar<CTAS>(&full[s]);
            const uint32_t st = tc::smem_u32(tiles + s * stage_bytes);
            if (elected) {
                if (leader) expect_bytes(&full[s], stage_tx);
                for (int h = 0; h < nstrips; ++h) {
                    const int u = (st0 + h) / strips_per_u, rest = st0 + h - u * strips_per_u;
                    const int r = p.inner == 1 ? rest / p.S : rest, sx = p.inner == 1 ? rest - r * p.S : 0;
                    const int c0 = (u * CTAS + static_cast<int>(rank)) * KB;
                    const int row = static_cast<int>(q0 + static_cast<long long>(r + p.off_h) * p.wp + p.off_w + sx);
                    load_rows<CTAS>(st + h * 2 * p.a_half, &x_hi, bar, c0, row);
                    load_rows<CTAS>(st + h * 2 * p.a_half + p.a_half, &x_lo, bar, c0, row);
                }
                for (int j = 0; j < my_boxes; ++j) {
                    const int c0 = n0 + (box0 + j) * KB;
                    load_rows<CTAS>(st + a_bytes + j * Cfg::BOX_BYTES, &dy_hi, bar, c0, static_cast<int>(q0));
                    load_rows<CTAS>(st + a_bytes + (Cfg::BOXES + j) * Cfg::BOX_BYTES, &dy_lo, bar, c0, static_cast<int>(q0));
                }
            }
            __syncwarp();
            if (++s == p.stages) { s = 0; phase ^= 1; }
        }
        if (!ok) atomicCAS(&tc::g_tc_error, 0, 101);
    } else if (leader) {
        const bool elected = tc::elect_one();
        const int st0 = g0 / p.inner;
        // byte offset of a group's first row in the stage
        auto group_at = [&](int g) {
            const int strip = g / p.inner;
            return static_cast<uint32_t>((strip - st0) * 2 * p.a_half + (g - strip * p.inner) * ROW_BYTES);
        };
        uint32_t at[T], lbo[T];
#pragma unroll
        for (int j = 0; j < T; ++j) {
            const int g = g0 + 2 * j;
            at[j] = g < g1 ? group_at(g) : 0u;
            // a single last group: the second 64 rows read one position on and are dropped
            lbo[j] = g + 1 < g1 ? group_at(g + 1) - at[j] : static_cast<uint32_t>(ROW_BYTES);
        }
        bool ok = true;
        for (int i = 0, c = 0, s = 0, phase = 0; i < nkb && ok; i += Cfg::CHAIN, ++c) {
            const int blocks = min(Cfg::CHAIN, nkb - i), s0 = s;
            const int at_slot = DEPTH == 2 ? c & 1 : 0, lap = DEPTH == 2 ? c >> 1 : c;
            for (int k = 0; k < blocks && ok; ++k) {          // cross products
                if (!tc::mbar_wait(tc::smem_u32(&full[s]), static_cast<uint32_t>(phase))) { ok = false; break; }
                const uint32_t a0 = tc::smem_u32(tiles + s * stage_bytes), b_hi = a0 + a_bytes;
                const uint64_t dbh = desc_mn(b_hi, Cfg::BOX_BYTES), dbl = desc_mn(b_hi + Cfg::BOXES * Cfg::BOX_BYTES, Cfg::BOX_BYTES);
#pragma unroll
                for (int j = 0; j < T; ++j) {
                    if (j >= my_tiles || !ok) continue;
                    const int slot = j * DEPTH + at_slot;
                    if (k == 0 && lap > 0 && !tc::mbar_wait(tc::smem_u32(&acc_free[slot]), (lap - 1) & 1u)) { ok = false; continue; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (elected)
                        mma_cross<CTAS, 2048 / 16>(tmem_base + slot * Cfg::ACC_COLS, desc_mn(a0 + at[j], lbo[j]), desc_mn(a0 + at[j] + p.a_half, lbo[j]), dbh, dbl,
                                                   Cfg::IDESC, k == 0);
                    __syncwarp();
                }
                if (++s == p.stages) { s = 0; phase ^= 1; }
            }
            for (int k = 0, sm = s0; k < blocks && ok; ++k) { // main products
                const uint32_t a0 = tc::smem_u32(tiles + sm * stage_bytes);
                const uint64_t dbh = desc_mn(a0 + a_bytes, Cfg::BOX_BYTES);
                if (elected) {
#pragma unroll
                    for (int j = 0; j < T; ++j) {
                        if (j >= my_tiles) continue;
                        const int slot = j * DEPTH + at_slot;
                        mma_main<CTAS, 2048 / 16>(tmem_base + slot * Cfg::ACC_COLS, desc_mn(a0 + at[j], lbo[j]), dbh, Cfg::IDESC, k == 0);
                        if (k == blocks - 1) commit_all<CTAS>(&acc_ready[slot]);
                    }
                    commit_all<CTAS>(&empty[sm]);
                }
                __syncwarp();
                if (++sm == p.stages) sm = 0;
            }
        }
        if (!ok) atomicCAS(&tc::g_tc_error, 0, 102);
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    sync_all<CTAS>();
    if (warp == DRAIN_WARPS + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_free<CTAS>(tmem_base, Cfg::TMEM_COLS);
    }
}

// ---- host side ----------------------------------------------------------------------------------------------------

// Positions per row and rows per image of a layer's lists (wp, hp), such that in all three products a tap's shift ends on the
// right element or on a zero: x needs pad zeros behind every row and image, dy (Q = W + 2 pad - S + 1 columns) needs S - 1 - pad.
struct ListGeom { int wp, hp; };
inline ListGeom list_geometry(int h, int w, int p, int q, int pad_h, int pad_w) {
    return {w + pad_w > q ? w + pad_w : q, h + pad_h > p ? h + pad_h : p};
}

// Bytes of the two lists of n images of c channels.
inline size_t list_bytes(long long n, int c, int lp) { return 2 * static_cast<size_t>(n) * lp * padded_channels(c) * sizeof(__half); }

// Writes the lists of n images of src (list_bytes() bytes at `lists`, 128-byte aligned).  sums: see ListJob, or null.  fresh: the
// magnitudes are found but the scale record has not been written (see few_parts).
inline int write_lists(const float* src, char* lists, int n, int c, int h, int w, int wp, int lp, const ScaleParts& sp, int op, bool fresh, cudaStream_t stream,
                       float* sums = nullptr, float sum_scale = 0.0f) {
    ListJob j;
    j.src = src; j.C = c; j.cp = padded_channels(c); j.H = h; j.W = w; j.wp = wp; j.lp = lp; j.op = op; j.sums = sums; j.sum_scale = sum_scale;
    j.hi = reinterpret_cast<__half*>(lists);
    j.lo = j.hi + static_cast<size_t>(n) * lp * j.cp;
    if (j.cp / KB > 65535 || n > 65535) return VDNN_ERR_UNSUPPORTED;
    const int tiles = ceil_div(h * w, LIST_PIXELS);
    // sums: fewer atomics with more tiles a block, as long as ten blocks are left for every SM
    const long long all = static_cast<long long>(tiles) * (j.cp / KB) * n, per = all / (10 * sm_count());
    j.tiles = sums ? static_cast<int>(per < 1 ? 1 : (per > 16 ? 16 : per)) : 1;
    const dim3 grid(ceil_div(tiles, j.tiles), j.cp / KB, n);
    const bool vec = h * w % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
    auto kern = sums ? (vec ? lists_kernel<true, true> : lists_kernel<true, false>) : (vec ? lists_kernel<false, true> : lists_kernel<false, false>);
    VDNN_CUDA(tc::launch_early(kern, grid, 256, 0, stream, j, sp, fresh ? 1 : 0));
    VDNN_LAUNCHED();
    return VDNN_OK;
}
// The lists of a folded x: n images of h2 x w2 positions.
inline int write_folded_lists(const float* x, char* lists, int n, const Fold& f, int h2, int w2, const ScaleParts& sp, bool fresh, cudaStream_t stream) {
    const int cp = padded_channels(f.c * f.s * f.s), cblocks = cp / KB;
    __half* hi = reinterpret_cast<__half*>(lists);
    __half* lo = hi + static_cast<size_t>(n) * h2 * w2 * cp;
    const dim3 grid(ceil_div(w2, 64), h2, n * cblocks);
    if (grid.y > 65535u || grid.z > 65535u) return VDNN_ERR_UNSUPPORTED;
    auto kern = f.s == 2 ? fold_lists_kernel<2> : (f.s == 3 ? fold_lists_kernel<3> : fold_lists_kernel<4>);
    VDNN_CUDA(tc::launch_early(kern, grid, 256, 0, stream, x, hi, lo, f, cp, h2, w2, cblocks, sp, fresh ? 1 : 0));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

// Every block of lists_kernel may add the parts of the magnitudes up itself: a load for each thread.
inline bool few_parts(const ScaleParts& sp) { return sp.blocks[0] <= 256 && sp.blocks[1] <= 256 && sp.blocks[2] <= 256; }

// Blocks of magnitude_kernel for an operand of n elements: 16 elements a thread and turn, 2 turns before a block is added.
inline int magnitude_blocks(size_t n) {
    const size_t b = ceil_div<size_t>(n, 8192);
    return static_cast<int>(b > PARTS ? PARTS : b);
}
// `area`: SCALE_BYTES of workspace.  Operands that a call does not have are null.
inline ScaleParts scale_parts(char* area, size_t nx, size_t nw, size_t ndy) {
    ScaleParts sp;
    sp.scales = reinterpret_cast<Scales*>(area);
    sp.part = reinterpret_cast<uint2*>(area + 128);
    sp.blocks[OP_X] = magnitude_blocks(nx); sp.blocks[OP_W] = magnitude_blocks(nw); sp.blocks[OP_DY] = magnitude_blocks(ndy);
    return sp;
}
inline int find_magnitudes(const ScaleParts& sp, const float* x, size_t nx, const float* w, size_t nw, const float* dy, size_t ndy, cudaStream_t stream) {
    const unsigned blocks = static_cast<unsigned>(sp.blocks[0] + sp.blocks[1] + sp.blocks[2]);
    VDNN_CUDA(tc::launch_early(magnitude_kernel, dim3(blocks), 256, 0, stream, x, nx, w, nw, dy, ndy, sp));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

// Columns of an output tile of strip_kernel: with 256 columns on a pair an MMA reads the fewest operand bytes per flop, and two
// 128-position halves of a CTA share 128 columns of filters.  VDNN_STRIP_PAIRS=0: no pairs (comparison runs).
inline bool strip_pairs_enabled() {
    static const bool v = []() { const char* e = getenv("VDNN_STRIP_PAIRS"); return !e || e[0] != '0'; }();
    return v;
}
inline int strip_columns(int n_cols) { return n_cols <= 64 ? 64 : (n_cols < 256 || !strip_pairs_enabled() ? 128 : 256); }

inline size_t packed_bytes(int n_cols, int reduction, int taps) {
    const int bn = strip_columns(n_cols);
    return static_cast<size_t>(ceil_div(n_cols, bn)) * taps * (padded_channels(reduction) / KB) * 2 * bn * ROW_BYTES;
}

// Packs the filters and writes the call's scale record (find_magnitudes() has been called).
inline int pack_folded(bool data_gradient, const float* w, int K, const Fold& f, int R2, int S2, char* tiles, const ScaleParts& sp, cudaStream_t stream) {
    const int channels = f.c * f.s * f.s, cols = data_gradient ? channels : K, bn = strip_columns(cols), n_tiles = ceil_div(cols, bn);
    const int cblocks = padded_channels(data_gradient ? K : channels) / KB;
    const size_t items = static_cast<size_t>(n_tiles) * R2 * S2 * cblocks * bn * 8, cap = static_cast<size_t>(sm_count()) * 8;
    size_t blocks = ceil_div<size_t>(items, 256);
    if (blocks > cap) blocks = cap;
    const dim3 grid(static_cast<unsigned>(blocks));
    if (data_gradient) VDNN_CUDA(tc::launch_early(pack_folded_kernel<true>, grid, 256, 0, stream, w, K, f, R2, S2, bn, n_tiles, cblocks, tiles, sp));
    else VDNN_CUDA(tc::launch_early(pack_folded_kernel<false>, grid, 256, 0, stream, w, K, f, R2, S2, bn, n_tiles, cblocks, tiles, sp));
    VDNN_LAUNCHED();
    return VDNN_OK;
}
inline int pack_filters(bool data_gradient, const float* w, int K, int C, int R, int S, char* tiles, const ScaleParts& sp, cudaStream_t stream) {
    const int cols = data_gradient ? C : K, bn = strip_columns(cols), n_tiles = ceil_div(cols, bn), cblocks = padded_channels(data_gradient ? K : C) / KB;
    const size_t items = static_cast<size_t>(n_tiles) * R * cblocks * bn * 8, cap = static_cast<size_t>(sm_count()) * 8;
    size_t blocks = ceil_div<size_t>(items, 256);
    if (blocks > cap) blocks = cap;
    const dim3 grid(static_cast<unsigned>(blocks));
    if (data_gradient) VDNN_CUDA(tc::launch_early(pack_filters_kernel<true>, grid, 256, 0, stream, w, K, C, R, S, bn, n_tiles, cblocks, tiles, sp));
    else VDNN_CUDA(tc::launch_early(pack_filters_kernel<false>, grid, 256, 0, stream, w, K, C, R, S, bn, n_tiles, cblocks, tiles, sp));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

inline int make_half_map(CUtensorMap* map, const void* base, size_t cols, size_t rows, int box_cols, int box_rows, CUtensorMapSwizzle swizzle) {
    tma::EncodeTiledFn enc = tma::encode_tiled();
    if (!enc) return VDNN_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * sizeof(__half)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t elem[2] = {1u, 1u};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? VDNN_OK : VDNN_ERR_CUDA;
}
inline int make_list_maps(CUtensorMap* hi, CUtensorMap* lo, const char* lists, long long positions, int c, int rows) {
    const size_t cp = padded_channels(c);
    const __half* h = reinterpret_cast<const __half*>(lists);
    const int st = make_half_map(hi, h, cp, positions, KB, rows, CU_TENSOR_MAP_SWIZZLE_128B);
    return st != VDNN_OK ? st : make_half_map(lo, h + static_cast<size_t>(positions) * cp, cp, positions, KB, rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

// Launches a kernel of CTA pairs or single CTAs, set up while its predecessor still runs.
template <int CTAS, class Kernel, class... Args>
inline cudaError_t launch_ctas(Kernel kern, dim3 grid, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CTAS; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.gridDim = grid; cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cfg.attrs = attr; cfg.numAttrs = CTAS == 2 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// VDNN_TMA_BOXES=1 (comparison runs): one strip per tap whatever the filter's width, as filters wider than STRIP_TAPS need.
inline int taps_per_strip(int S) {
    static const bool single = []() { const char* e = getenv("VDNN_TMA_BOXES"); return e && *e && *e != '0'; }();
    return single || S > STRIP_TAPS ? 1 : S;
}

// Tiles of strip_kernel that the GPU works on at a time, and how many the problem has (in CTAs or pairs).
inline int strip_slots(int n_cols) { return strip_columns(n_cols) == 64 ? sm_count() : sm_count() / 2; }
inline long long strip_tiles(const Problem& q) {
    const int bn = strip_columns(q.n_cols);
    return ceil_div<long long>(static_cast<long long>(q.n) * q.lp, bn == 128 ? 512 : 256) * ceil_div(q.n_cols, bn);
}

template <int BN, int MH, int CTAS>
int strip_launch_as(const Problem& q, const char* lists, const char* b_tiles, float* out, const float* bias, float alpha, float beta, int mode,
                    size_t partial_stride, int splits, int group_chunk, const Scales* scales, int product, cudaStream_t stream) {
    typedef StripConfig<BN, MH, CTAS> Cfg;
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
    auto kern = strip_kernel<BN, MH, CTAS>;
    VDNN_ALLOW_SHARED(dev, kern, Cfg::SMEM_BYTES);
    StripParams p;
    p.wp = q.wp; p.lp = q.lp;
    p.total_pos = static_cast<long long>(q.n) * q.lp;
    p.div_lp = FastDiv(q.lp); p.div_wp = FastDiv(q.wp);
    p.out_h = q.out_h; p.out_w = q.out_w; p.n_cols = q.n_cols;
    p.S = q.S; p.cblocks = padded_channels(q.cin) / KB;
    p.dh0 = q.off_h; p.dh_step = q.tap_sign;
    p.row0 = q.tap_sign > 0 ? 0 : q.S - 1; p.row_step = q.tap_sign;
    p.dw_min = q.tap_sign > 0 ? q.off_w : q.off_w - (q.S - 1);
    p.inner = taps_per_strip(q.S);
    p.groups_total = q.R * p.cblocks * (q.S / p.inner);
    p.group_chunk = group_chunk;
    p.kblocks_total = q.R * q.S * p.cblocks;
    p.out = out; p.bias = bias; p.alpha = alpha; p.beta = beta; p.mode = mode; p.partial_stride = partial_stride;
    p.scales = scales; p.product = product;
    p.fold = q.fold;
    if (product != DATA) p.fold.s = 1;
    const int ny = ceil_div(q.n_cols, BN);
    if (ny > 65535 || splits > 65535) return VDNN_ERR_UNSUPPORTED;
    CUtensorMap map_hi, map_lo, map_b;
    int st = make_list_maps(&map_hi, &map_lo, lists, p.total_pos, q.cin, BM + p.inner - 1);
    if (st != VDNN_OK) return st;
    // the packed filter tiles as rows of 128 bytes (they are stored swizzled already: the copy must not swizzle again)
    st = make_half_map(&map_b, b_tiles, KB, static_cast<size_t>(ny) * p.kblocks_total * (2 * BN), KB, Cfg::COLS_HERE, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (st != VDNN_OK) return st;
    // persistent along x: as many CTAs (pairs) as the GPU holds at once (all column tiles and splits of an output tile run side
    // by side, so that they share its strips through L2)
    const long long tiles = ceil_div<long long>(p.total_pos, BM * MH * CTAS);
    long long slots = sm_count();
    if constexpr (CTAS == 2) {
        // a property of kernel and device: asked for once
        static std::atomic<int> resident_on[64];
        int resident = dev < 64 ? resident_on[dev].load(std::memory_order_relaxed) : 0;
        if (resident == 0) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(2 * (sm_count() / 2)); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
            cfg.attrs = attr; cfg.numAttrs = 1;
            VDNN_CUDA(cudaOccupancyMaxActiveClusters(&resident, kern, &cfg));
            if (resident < 1) return VDNN_ERR_UNSUPPORTED;
            if (dev < 64) resident_on[dev].store(resident, std::memory_order_relaxed);
        }
        slots = resident;
    }
    long long gx = slots / (static_cast<long long>(ny) * splits);
    if (gx < 1) gx = 1;
    if (gx > tiles) gx = tiles;
    VDNN_CUDA((launch_ctas<CTAS>(kern, dim3(static_cast<unsigned>(gx * CTAS), ny, splits), Cfg::SMEM_BYTES, stream, map_hi, map_lo, map_b, p)));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

// The contraction over lists and packed filters.  group_chunk: (strip of a filter row or tap, channel block) groups per split.
inline int strip_groups(const Problem& q) { return q.R * (padded_channels(q.cin) / KB) * (q.S / taps_per_strip(q.S)); }
inline int strip_launch(const Problem& q, const char* lists, const char* b_tiles, float* out, const float* bias, float alpha, float beta, int mode,
                        size_t partial_stride, int splits, int group_chunk, const Scales* scales, int product, cudaStream_t stream) {
    switch (strip_columns(q.n_cols)) {
    case 64: return strip_launch_as<64, 2, 1>(q, lists, b_tiles, out, bias, alpha, beta, mode, partial_stride, splits, group_chunk, scales, product, stream);
    case 128: return strip_launch_as<128, 2, 2>(q, lists, b_tiles, out, bias, alpha, beta, mode, partial_stride, splits, group_chunk, scales, product, stream);
    default: return strip_launch_as<256, 1, 2>(q, lists, b_tiles, out, bias, alpha, beta, mode, partial_stride, splits, group_chunk, scales, product, stream);
    }
}

struct WgradProblem {
    int n, c, h, w;          // x
    int k, p, q;             // dy: n x k x p x q
    int R, S, pad_h, pad_w;
    int wp, lp;
    Fold fold;
    size_t filter_elems() const { return static_cast<size_t>(k) * fold.c * fold.R * fold.S; }
};

// How a filter gradient is cut.
struct WgradPlan { int bn, tiles, ctas; int groups, chunk, strips, a_half, stages; int kb_total, kb_chunk, splits; size_t smem; };

inline WgradPlan wgrad_plan(const WgradProblem& q) {
    static const bool pairs = []() { const char* e = getenv("VDNN_WGRAD_PAIRS"); return !e || e[0] != '0'; }();
    WgradPlan w;
    const int taps = q.R * q.S, cblocks = padded_channels(q.c) / KB, inner = taps_per_strip(q.S);
    w.bn = q.k <= 64 ? 64 : (q.k < 256 ? 128 : 256);
    w.ctas = w.bn == 256 ? 2 : 1;
    // a pair takes two channel blocks: an odd one leaves its last pair half empty
    if (w.bn == 256 && (!pairs || cblocks == 1 || cblocks == 3)) { w.bn = 128; w.ctas = 1; }
    w.tiles = w.bn == 64 ? 5 : (w.bn == 128 ? 2 : 1);
    w.groups = ceil_div(cblocks, w.ctas) * taps;
    w.a_half = ceil_div((KB + inner - 1) * ROW_BYTES, 1024) * 1024;
    const int b_bytes = 2 * (w.bn / w.ctas) * ROW_BYTES;
    w.chunk = taps <= 2 * w.tiles && taps > w.tiles ? taps : 2 * w.tiles;
    if (w.chunk > w.groups) w.chunk = w.groups;
    for (;; w.chunk = w.chunk > 2 ? (w.chunk - 1) / 2 * 2 : 1) {
        w.strips = 1;
        for (int g = 0; g < w.groups; g += w.chunk) {
            const int last = (g + w.chunk < w.groups ? g + w.chunk : w.groups) - 1, s = last / inner - g / inner + 1;
            if (s > w.strips) w.strips = s;
        }
        const int stage = w.strips * 2 * w.a_half + b_bytes, room = SMEM_LIMIT - 1024 - 512;
        w.stages = room / stage;
        if (w.stages >= 3 || w.chunk <= 2) {
            if (w.stages > WGRAD_MAX_STAGES) w.stages = WGRAD_MAX_STAGES;
            w.smem = static_cast<size_t>(w.stages) * stage + 1024 + 512;
            break;
        }
    }
    w.kb_total = static_cast<int>(ceil_div<long long>(static_cast<long long>(q.n) * q.lp, 64));
    // As many splits of the reduction as fill the GPU, with the fewest waves that keep it nearly full (every split leaves
    // a partial result to be added), four blocks each at least.
    const long ctas = static_cast<long>(ceil_div(w.groups, w.chunk)) * w.ctas * ceil_div(q.k, w.bn);
    long best = 1;
    double best_use = 0.0;
    for (int waves = 1; waves <= 4; ++waves) {
        const long s = static_cast<long>(waves) * sm_count() / ctas;
        if (s < 1) continue;
        const double use = static_cast<double>(s * ctas) / (static_cast<double>(waves) * sm_count());
        if (use > best_use + 0.04) { best_use = use; best = s; }
    }
    if (best > w.kb_total / 4) best = w.kb_total / 4;
    if (best > 1024) best = 1024;
    if (best < 1) best = 1;
    w.kb_chunk = ceil_div(w.kb_total, static_cast<int>(best));
    w.splits = ceil_div(w.kb_total, w.kb_chunk);
    return w;
}

inline size_t wgrad_partial_bytes(const WgradProblem& q) {
    const WgradPlan w = wgrad_plan(q);
    return w.splits > 1 ? static_cast<size_t>(w.splits) * q.filter_elems() * sizeof(float) : 0;
}

template <int BN, int T, int CTAS>
int wgrad_launch_as(const WgradProblem& q, const WgradPlan& w, const char* x_lists, const char* dy_lists, float* partial, float* dw, float alpha, float beta,
                    const Scales* scales, cudaStream_t stream) {
    typedef WgradConfig<BN, T, CTAS> Cfg;
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
    auto kern = wgrad_kernel<BN, T, CTAS>;
    VDNN_ALLOW_SHARED(dev, kern, SMEM_LIMIT);
    static_assert((2 * WGRAD_MAX_STAGES + 2 * Cfg::SLOTS + 1) * 8 <= 512, "barriers fit behind the stages");
    WgradParams p;
    p.wp = q.wp;
    p.R = q.R; p.S = q.S; p.inner = taps_per_strip(q.S); p.cblocks = padded_channels(q.c) / KB;
    p.off_h = -q.pad_h; p.off_w = -q.pad_w;
    p.groups = w.groups; p.group_chunk = w.chunk; p.strips = w.strips; p.a_half = w.a_half; p.stages = w.stages;
    p.kb_total = w.kb_total; p.kb_chunk = w.kb_chunk;
    p.C = q.c; p.n_cols = q.k; p.cols_padded = padded_channels(q.k);
    p.partial_stride = q.filter_elems();
    p.fold = q.fold;
    if (w.splits > 1) { p.out = partial; p.alpha = 1.0f; p.beta = 0.0f; p.mode = EPI_PARTIAL; }
    else { p.out = dw; p.alpha = alpha; p.beta = beta; p.mode = EPI_DIRECT; }
    p.scales = scales;
    const long long positions = static_cast<long long>(q.n) * q.lp;
    CUtensorMap maps[4];
    int st = make_list_maps(&maps[0], &maps[1], x_lists, positions, q.c, KB + p.inner - 1);
    if (st != VDNN_OK) return st;
    st = make_list_maps(&maps[2], &maps[3], dy_lists, positions, q.k, KB);
    if (st != VDNN_OK) return st;
    const dim3 grid(ceil_div(w.groups, w.chunk) * CTAS, ceil_div(q.k, BN), w.splits);
    if (grid.y > 65535u || grid.z > 65535u) return VDNN_ERR_UNSUPPORTED;
    VDNN_CUDA((launch_ctas<CTAS>(kern, grid, w.smem, stream, maps[0], maps[1], maps[2], maps[3], p)));
    VDNN_LAUNCHED();
    return VDNN_OK;
}

// The filter gradient of the lists of q.n images; partial: wgrad_partial_bytes() bytes, to be added up where w.splits > 1.
inline int wgrad_launch(const WgradProblem& q, const WgradPlan& w, const char* x_lists, const char* dy_lists, float* partial, float* dw, float alpha,
                        float beta, const Scales* scales, cudaStream_t stream) {
    if (w.bn == 64) return wgrad_launch_as<64, 5, 1>(q, w, x_lists, dy_lists, partial, dw, alpha, beta, scales, stream);
    if (w.bn == 128) return wgrad_launch_as<128, 2, 1>(q, w, x_lists, dy_lists, partial, dw, alpha, beta, scales, stream);
    return wgrad_launch_as<256, 1, 2>(q, w, x_lists, dy_lists, partial, dw, alpha, beta, scales, stream);
}

}  // namespace split16
}  // namespace vdnn
