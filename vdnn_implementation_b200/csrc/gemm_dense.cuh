// Dense fp32-accurate GEMM on tcgen05 with the A operand in tensor memory: C(m x n, column-major) = alpha op(A) op(B) + beta C.
//
// This is what the fully connected layers run on: one operand is a weight matrix of hundreds of megabytes, the other a batch
// of at most a few hundred rows, so the call is bound by streaming the weights -- if enough bytes are in flight and the
// shared memory is not the bottleneck first.  The gather-fed kernel (gemm_tc.cuh) had one k block in flight per SM and moved
// every operand element through registers and twice (hi, lo) through shared memory.  Here
//   * one warp (its elected lane) fetches raw fp32 tiles of both operands with tensor copies into a ring of 4 .. 7 stages (96 .. 170 KB in
//     flight per SM);
//   * two or three groups of four warps, taking stages in turn, split them into tf32 hi / lo: the A tile goes from shared memory through registers into TENSOR MEMORY
//     (tcgen05.st; lane = row, column = k), where tcgen05.mma reads it without touching shared memory, whatever its
//     orientation in memory was; the B tile is split in place (hi over the raw values, lo beside it);
//   * one warp walks the stages and an elected lane of it issues the 3xTF32 MMAs, eight warps add finished accumulators into fp32 registers and store.
// Shared-memory traffic per 128 x 64 x 32 block is 704 clocks' worth instead of 1344 with A staged as hi / lo tiles, just
// under what HBM delivers (16 KB of weights in 712 clocks).
// Measured (batch 64, 25088 -> 4096, flushed L2, B200; 411 MB of weights = 63 us at copy rate), gather-fed kernel before ->
// now: output 200 -> 106 us, data gradient 258 -> 114, filter gradient 311 -> 143, weight step in place 882 -> 191.
#pragma once

#include <atomic>

#include "gemm_tc.cuh"
#include "tensor_map.cuh"

namespace vdnn {
namespace dense {

using tc::BK;
using tc::BM;

constexpr int DRAIN_WARPS = 8;
constexpr int SPLIT_GROUP = 4 * 32;                                  // threads that split one stage: a row of A each

// STAGED: C goes out through shared memory (short reductions, see tile_n), which costs stages.
template <int BN, bool STAGED> struct Config {
    static_assert(!STAGED || BN <= 64, "no room for C tiles beside 128-column stages");
    static constexpr int A_BYTES = BM * BK * 4;
    static constexpr int B_BYTES = BN * BK * 4;                      // hi (over the raw tile); lo follows
    static constexpr int STAGE_BYTES = A_BYTES + 2 * B_BYTES;
    // Splitting a stage takes its group about 1700 clocks from barrier to barrier, 500 of issue: three groups in turn keep up
    // with the memory; with 128 columns (registers for the wider accumulators, twice the MMA time per stage) two do.
    static constexpr int GROUPS = BN == 128 ? 2 : 3;
    static constexpr int TMA_WARP = DRAIN_WARPS + 4 * GROUPS, MMA_WARP = TMA_WARP + 1;
    static constexpr int THREADS = (MMA_WARP + 1) * 32;
    // MERGED: the lo tile of B follows the hi tile, so one MMA of 2 * BN columns forms a_hi * [b_hi | b_lo] and a second one
    // adds a_lo * b_hi: an MMA of up to 64 columns costs 45 clocks whatever its width, one of 128 columns 64.  The drain adds
    // the halves of the accumulator.
    static constexpr bool MERGED = BN <= 64;
    static constexpr int ACC_COLS = MERGED ? 2 * BN : BN;
    // two accumulators, then slots of 64 columns (32 hi, 32 lo) of A fill the 512 columns of tensor memory
    static constexpr int STAGES = BN == 128 ? 4 : (BN == 64 && STAGED ? 5 : 7);
    static constexpr int A_COL = 2 * ACC_COLS;
    static constexpr int A_SLOTS = (512 - A_COL) / (2 * BK) < STAGES ? (512 - A_COL) / (2 * BK) : STAGES;
    static constexpr int C_TILES = STAGED ? 2 : 0;                   // finished tiles, column by column
    static constexpr int C_BYTES = BM * BN * 4;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + C_TILES * C_BYTES + 1024 + 256;
    __host__ __device__ static constexpr uint32_t idesc(int cols) {
        return (1u << 4) | (2u << 7) | (2u << 10) | (static_cast<uint32_t>(cols >> 3) << 17) | (static_cast<uint32_t>(BM >> 4) << 24);
    }
};

struct Params {
    int M, N, tiles_m, kblocks, splits, kb_chunk;                    // k blocks of 32; a split walks kb_chunk of them
    long long tile0, units;                                          // first tile of the launch; its tiles * splits
    float* out;                                                      // element (i, j) at out[j * ldc + i]
    long long ldc;
    float alpha, beta;
};

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
                   "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]) : "memory");
}
// A finished 128 x BN tile from shared memory to its box of C, and the old values of such a box to shared memory.  Rows and
// columns outside the matrix are clipped.
__device__ __forceinline__ void tma_tile_out(const CUtensorMap* map, uint32_t src, int m, int n) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src), "r"(m), "r"(n) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr, uint32_t rank) {
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// Two groups of 16 columns, `apart` columns from each other, with one wait for both.
__device__ __forceinline__ void tmem_ld16_2(uint32_t taddr, int apart, float (&v)[16], float (&w)[16]) {
    uint32_t r[16], q[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
                 "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(r[8]),
                   "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15]), "=&r"(q[0]), "=&r"(q[1]),
                   "=&r"(q[2]), "=&r"(q[3]), "=&r"(q[4]), "=&r"(q[5]), "=&r"(q[6]), "=&r"(q[7]), "=&r"(q[8]), "=&r"(q[9]), "=&r"(q[10]),
                   "=&r"(q[11]), "=&r"(q[12]), "=&r"(q[13]), "=&r"(q[14]), "=&r"(q[15])
                 : "r"(taddr), "r"(taddr + static_cast<uint32_t>(apart)) : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) { v[i] = __uint_as_float(r[i]); w[i] = __uint_as_float(q[i]); }
}
__device__ __forceinline__ void drain_sync() {
    __syncwarp();
    asm volatile("bar.sync 1, %0;" ::"n"(DRAIN_WARPS * 32) : "memory");
}
// D += A * B with A in tensor memory.
__device__ __forceinline__ void mma_tf32_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// One 32-wide k block of the 3xTF32 product; A hi at tmem_a, lo 32 columns further; STEP as in tc::mma_block_3xtf32.
template <int STEP, bool MERGED>
__device__ __forceinline__ void mma_block_ta(uint32_t d_tmem, uint32_t tmem_a, uint64_t dbh, uint64_t dbl, uint32_t idesc, uint32_t idesc_wide,
                                             bool fresh) {
#pragma unroll
    for (int ks = 0; ks < BK / 8; ++ks) {
        const uint32_t acc = (fresh && ks == 0) ? 0u : 1u;
        if (MERGED) {
            mma_tf32_ta(d_tmem, tmem_a + ks * 8, dbh + ks * STEP, idesc_wide, acc);
            mma_tf32_ta(d_tmem, tmem_a + BK + ks * 8, dbh + ks * STEP, idesc, 1u);
        } else {
            mma_tf32_ta(d_tmem, tmem_a + BK + ks * 8, dbh + ks * STEP, idesc, acc);
            mma_tf32_ta(d_tmem, tmem_a + ks * 8, dbl + ks * STEP, idesc, 1u);
            mma_tf32_ta(d_tmem, tmem_a + ks * 8, dbh + ks * STEP, idesc, 1u);
        }
    }
}

// AK / BKM: the operand is contiguous along k (its tile has a 128-byte row of 32 k per m or n), else along m / n.
//   A, AK   box 32 k x 128 rows, 128-byte swizzle;   !AK  box 128 m x 32 k, no swizzle (rows of 512 bytes)
//   B, BKM  box 32 k x BN rows, 128-byte swizzle;    !BKM BN / 32 boxes of 32 n x 32 k, 32-byte-atom swizzle (MN-major MMA)
// Elements outside the matrices read as zero.
template <bool AK, bool BKM, int BN, bool STAGED>
__global__ void __launch_bounds__(Config<BN, STAGED>::THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_c,
            const Params p) {
    typedef Config<BN, STAGED> Cfg;
    constexpr int S = Cfg::STAGES;
    constexpr uint32_t B_MN = BKM ? 0u : 1u << 16;
    constexpr uint32_t IDESC = Cfg::idesc(BN) | B_MN, IDESC_WIDE = Cfg::idesc(Cfg::MERGED ? 2 * BN : BN) | B_MN;
    constexpr int TMA_WARP = Cfg::TMA_WARP, MMA_WARP = Cfg::MMA_WARP;
    extern __shared__ char smem_raw[];
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    float* c_tile = reinterpret_cast<float*>(tiles + S * Cfg::STAGE_BYTES);
    uint64_t* raw_full = reinterpret_cast<uint64_t*>(tiles + S * Cfg::STAGE_BYTES + Cfg::C_TILES * Cfg::C_BYTES);      // [S] tensor copies have landed
    uint64_t* split_full = raw_full + S;    // [S] both operands are split
    uint64_t* empty = split_full + S;       // [S] the MMAs have read the stage
    uint64_t* acc_ready = empty + S;        // [2]
    uint64_t* acc_free = acc_ready + 2;     // [2]
    uint64_t* c_full = acc_free + 2;        // [2] the old values of a C tile
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(c_full + 2);

    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (t == 0) {
        for (int s = 0; s < S; ++s) {
            tc::mbar_init(tc::smem_u32(&raw_full[s]), 1);
            tc::mbar_init(tc::smem_u32(&split_full[s]), SPLIT_GROUP);
            tc::mbar_init(tc::smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) { tc::mbar_init(tc::smem_u32(&acc_ready[b]), 1); tc::mbar_init(tc::smem_u32(&acc_free[b]), DRAIN_WARPS); tc::mbar_init(tc::smem_u32(&c_full[b]), 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    // Every role walks the same units: the splits of a tile side by side (they are one cluster), row tile before column tile.
    // The CTAs then work side by side along the contiguous direction of C: with column tiles fastest, a filter gradient
    // (25088 x 4096) was written in pieces of 512 bytes all over its 411 MB.
    auto unit_of = [&](long long u, int* m0, int* n0, int* kb0, int* nkb) {
        const long long tile = p.tile0 + u / p.splits;
        *m0 = static_cast<int>(tile % p.tiles_m) * BM;
        *n0 = static_cast<int>(tile / p.tiles_m) * BN;
        *kb0 = static_cast<int>(u % p.splits) * p.kb_chunk;
        *nkb = min(p.kblocks, *kb0 + p.kb_chunk) - *kb0;
    };
    int m0, n0, kb0, nkb;

    if (warp < DRAIN_WARPS) {
        // ------------------------------------------------------------------ accumulator drain + epilogue
        constexpr int NACC = BN / 2;
        const int col_beg = (warp >> 2) * NACC;
        const uint32_t tmem_mine = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(col_beg);
        unsigned pair = 0;
        bool alive = true;
        // STAGED: tiles go out, and with beta the old values of the NEXT unit's tile come in while this one is summed, by tensor
        // copies through two tiles of shared memory.  With one 4-byte load and store per lane and column the weight step of a
        // 25088 x 4096 layer took 490 us (822 MB), the plain product 220 (411 MB).
        const bool old_c = STAGED && p.beta != 0.0f;
        auto fetch_old = [&](long long u, int buf) {
            unit_of(u, &m0, &n0, &kb0, &nkb);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc::smem_u32(&c_full[buf])), "r"(Cfg::C_BYTES) : "memory");
            tma::tma_load_rows(tc::smem_u32(c_tile + buf * (Cfg::C_BYTES / 4)), &map_c, tc::smem_u32(&c_full[buf]), m0, n0);
        };
        unsigned unit = 0;
        if (old_c && t == 0 && blockIdx.x < p.units) fetch_old(blockIdx.x, 0);
        // (a warp whose wait expired waits no more, but walks the units to the end: it owes the others its part of drain_sync)
        for (long long u = blockIdx.x; u < p.units; u += gridDim.x, ++unit) {
            const int buf = unit & 1;
            if (old_c && alive && t == 0 && u + gridDim.x < p.units) {
                asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the last unit's tile has left its buffer
                fetch_old(u + gridDim.x, buf ^ 1);
            }
            unit_of(u, &m0, &n0, &kb0, &nkb);
            float acc[NACC];
#pragma unroll
            for (int j = 0; j < NACC; ++j) acc[j] = 0.0f;
            for (int i = 0; i < nkb && alive; i += 2, ++pair) {
                const int b = pair & 1;
                bool ok = tc::mbar_wait(tc::smem_u32(&acc_ready[b]), (pair >> 1) & 1u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { atomicCAS(&tc::g_tc_error, 0, 103); alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c = 0; c < NACC; c += 16) {
                    float v[16];
                    if (Cfg::MERGED) {
                        float w[16];
                        tmem_ld16_2(tmem_mine + static_cast<uint32_t>(b * Cfg::ACC_COLS + c), BN, v, w);
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[c + j] += v[j] + w[j];
                    } else {
                        tc::tmem_ld16(tmem_mine + static_cast<uint32_t>(b * Cfg::ACC_COLS + c), v);
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[c + j] += v[j];
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(tc::smem_u32(&acc_free[b]));
            }
            if (STAGED) {
                float* c = c_tile + buf * (Cfg::C_BYTES / 4) + col_beg * BM + (warp & 3) * 32 + lane;
                if (old_c) {
                    bool ok = !alive || tc::mbar_wait(tc::smem_u32(&c_full[buf]), (unit >> 1) & 1u);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) { atomicCAS(&tc::g_tc_error, 0, 103); alive = false; }
#pragma unroll
                    for (int j = 0; j < NACC; ++j) c[j * BM] = fmaf(p.beta, c[j * BM], p.alpha * acc[j]);
                } else {
                    if (t == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");      // the tile before the last has left
                    drain_sync();
#pragma unroll
                    for (int j = 0; j < NACC; ++j) c[j * BM] = p.alpha * acc[j];
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                drain_sync();
                if (t == 0 && alive) tma_tile_out(&map_c, tc::smem_u32(c_tile + buf * (Cfg::C_BYTES / 4)), m0, n0);
                continue;
            }
            if (p.splits > 1) {
                // the part goes to shared memory: this CTA's only unit, so the operand stages are done with
                float* c = reinterpret_cast<float*>(tiles) + col_beg * BM + (warp & 3) * 32 + lane;
#pragma unroll
                for (int j = 0; j < NACC; ++j) c[j * BM] = acc[j];
                continue;
            }
            // long reductions, and a C of odd alignment
            const int m = m0 + (warp & 3) * 32 + lane;
            if (!alive || m >= p.M) continue;
            float* o = p.out + static_cast<long long>(n0 + col_beg) * p.ldc + m;
            const int cols = p.N - n0 - col_beg;                    // of this thread's NACC
#pragma unroll
            for (int j = 0; j < NACC; ++j) {
                if (j < cols) {
                    const float v = p.alpha * acc[j];
                    *o = p.beta != 0.0f ? fmaf(p.beta, *o, v) : v;
                }
                o += p.ldc;
            }
        }
        if (STAGED && t == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else if (warp < TMA_WARP) {
        // ------------------------------------------------------------------ split: group g takes every GROUPS-th stage
        const int g = (warp - DRAIN_WARPS) >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + Cfg::A_COL;
        unsigned i = 0;
        bool alive = true;
        for (long long u = blockIdx.x; u < p.units && alive; u += gridDim.x) {
            unit_of(u, &m0, &n0, &kb0, &nkb);
            for (int kb = 0; kb < nkb; ++kb, ++i) {
                if (i % Cfg::GROUPS != static_cast<unsigned>(g)) continue;
                const int s = i % S;
                // The slot of tensor memory is free once the MMAs of k block i - A_SLOTS have read it.  This wait comes first:
                // it also proves that the stage's last copies (k block i - S, another group's) have landed.  A parity wait
                // tells a phase from its neighbours only; one that could be two phases ahead of its barrier passes at once.
                bool ok = true;
                if (i >= Cfg::A_SLOTS) {
                    const unsigned j = i - Cfg::A_SLOTS;
                    ok = tc::mbar_wait(tc::smem_u32(&empty[j % S]), (j / S) & 1u);
                }
                ok = ok && tc::mbar_wait(tc::smem_u32(&raw_full[s]), (i / S) & 1u);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { atomicCAS(&tc::g_tc_error, 0, 101); alive = false; break; }
                char* st = tiles + s * Cfg::STAGE_BYTES;
                const uint32_t slot = tmem_lane + (i % Cfg::A_SLOTS) * (2 * BK);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float hi[16], lo[16];
                    if (AK) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const float4 v = *reinterpret_cast<const float4*>(st + row * 128 + (((half * 4 + c) ^ (row & 7)) << 4));
                            tc::split_tf32_x2(v.x, v.y, hi[4 * c], hi[4 * c + 1], lo[4 * c], lo[4 * c + 1]);
                            tc::split_tf32_x2(v.z, v.w, hi[4 * c + 2], hi[4 * c + 3], lo[4 * c + 2], lo[4 * c + 3]);
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < 16; k += 2) {
                            const char* q = st + (half * 16 + k) * (BM * 4) + row * 4;
                            tc::split_tf32_x2(*reinterpret_cast<const float*>(q), *reinterpret_cast<const float*>(q + BM * 4), hi[k], hi[k + 1], lo[k],
                                              lo[k + 1]);
                        }
                    }
                    tmem_st16(slot + half * 16, hi);
                    tmem_st16(slot + BK + half * 16, lo);
                }
                float4* b_raw = reinterpret_cast<float4*>(st + Cfg::A_BYTES);
                float4* b_lo = reinterpret_cast<float4*>(st + Cfg::A_BYTES + Cfg::B_BYTES);
#pragma unroll
                for (int j = 0; j < BN * BK / 4 / SPLIT_GROUP; ++j) {
                    const int e = j * SPLIT_GROUP + row;
                    const float4 v = b_raw[e];
                    float4 h, l;
                    tc::split_tf32_x2(v.x, v.y, h.x, h.y, l.x, l.y);
                    tc::split_tf32_x2(v.z, v.w, h.z, h.w, l.z, l.w);
                    b_raw[e] = h;
                    b_lo[e] = l;
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                tc::mbar_arrive(tc::smem_u32(&split_full[s]));
            }
        }
    } else if (warp == TMA_WARP) {
        // ------------------------------------------------------------------ tensor copies
        if (lane == 0) {
            unsigned i = 0;
            bool ok = true;
            for (long long u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
                unit_of(u, &m0, &n0, &kb0, &nkb);
                for (int kb = 0; kb < nkb; ++kb, ++i) {
                    const int s = i % S;
                    if (!tc::mbar_wait(tc::smem_u32(&empty[s]), ((i / S) & 1u) ^ 1u)) { ok = false; break; }
                    const uint32_t bar = tc::smem_u32(&raw_full[s]);
                    const uint32_t st = tc::smem_u32(tiles + s * Cfg::STAGE_BYTES);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(Cfg::A_BYTES + Cfg::B_BYTES) : "memory");
                    const int k0 = (kb0 + kb) * BK;
                    tma::tma_load_rows(st, &map_a, bar, AK ? k0 : m0, AK ? m0 : k0);
                    if (BKM) {
                        tma::tma_load_rows(st + Cfg::A_BYTES, &map_b, bar, k0, n0);
                    } else {
#pragma unroll
                        for (int j = 0; j < BN / 32; ++j) tma::tma_load_rows(st + Cfg::A_BYTES + j * (32 * BK * 4), &map_b, bar, n0 + j * 32, k0);
                    }
                }
            }
            if (!ok) atomicCAS(&tc::g_tc_error, 0, 101);
        }
    } else {
        // ------------------------------------------------------------------ MMA issuer: the whole warp walks the loop (so that
        // addresses and descriptors stay in uniform registers), one elected lane issues
        const bool elected = tc::elect_one();
        unsigned i = 0, pair = 0;
        bool ok = true;
        for (long long u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
            unit_of(u, &m0, &n0, &kb0, &nkb);
            for (int kb = 0; kb < nkb; ++kb, ++i) {
                const int s = i % S, b = pair & 1;
                const bool fresh = !(kb & 1);
                // hand-overs `pair` and `pair - 2` share an accumulator: the drain warps must have emptied it
                if (fresh && pair >= 2 && !tc::mbar_wait(tc::smem_u32(&acc_free[b]), ((pair >> 1) - 1) & 1u)) { ok = false; break; }
                if (!tc::mbar_wait(tc::smem_u32(&split_full[s]), (i / S) & 1u)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t b_hi = tc::smem_u32(tiles + s * Cfg::STAGE_BYTES) + Cfg::A_BYTES, b_lo = b_hi + Cfg::B_BYTES;
                const uint32_t a = tmem_base + Cfg::A_COL + (i % Cfg::A_SLOTS) * (2 * BK), d = tmem_base + static_cast<uint32_t>(b * Cfg::ACC_COLS);
                const uint64_t dbh = BKM ? tc::make_desc(b_hi) : tma::make_desc_mn(b_hi), dbl = BKM ? tc::make_desc(b_lo) : tma::make_desc_mn(b_lo);
                const bool last = !fresh || kb == nkb - 1;
                if (elected) {
                    mma_block_ta<BKM ? 2 : 1024 / 16, Cfg::MERGED>(d, a, dbh, dbl, IDESC, IDESC_WIDE, fresh);
                    tc::mma_commit(tc::smem_u32(&empty[s]));
                    if (last) tc::mma_commit(tc::smem_u32(&acc_ready[b]));
                }
                __syncwarp();
                if (last) ++pair;
            }
        }
        if (!ok) atomicCAS(&tc::g_tc_error, 0, 102);
    }

    if (!STAGED && p.splits > 1) {
        // The CTAs of a cluster hold the parts of one tile; each adds a share of it, part 0 first, through distributed shared
        // memory.  (Adding parts to C with atomics cost a pass that scaled C, read and wrote C once per split, and left the
        // order of the sum to chance.)
        __syncwarp();
        cluster_sync();
        unit_of(blockIdx.x, &m0, &n0, &kb0, &nkb);
        constexpr int QUADS = BN * BM / 4;
        const int share = (QUADS + p.splits - 1) / p.splits, rank = static_cast<int>(blockIdx.x % static_cast<unsigned>(p.splits));
        const int end = min(QUADS, (rank + 1) * share);
        const bool vec = ((reinterpret_cast<uintptr_t>(p.out) & 15u) == 0) && p.ldc % 4 == 0;
        for (int e = rank * share + t; e < end; e += Cfg::THREADS) {
            const int m = m0 + (e % (BM / 4)) * 4, n = n0 + e / (BM / 4);
            if (m >= p.M || n >= p.N) continue;
            const uint32_t a = tc::smem_u32(tiles) + static_cast<uint32_t>(e) * 16u;
            float4 v = ld_cluster4(a, 0);
            for (int r = 1; r < p.splits; ++r) {
                const float4 w = ld_cluster4(a, static_cast<uint32_t>(r));
                v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
            }
            float* o = p.out + static_cast<long long>(n) * p.ldc + m;
            v.x *= p.alpha; v.y *= p.alpha; v.z *= p.alpha; v.w *= p.alpha;
            if (vec && m + 4 <= p.M) {
                if (p.beta != 0.0f) {
                    const float4 c = *reinterpret_cast<const float4*>(o);
                    v.x = fmaf(p.beta, c.x, v.x); v.y = fmaf(p.beta, c.y, v.y); v.z = fmaf(p.beta, c.z, v.z); v.w = fmaf(p.beta, c.w, v.w);
                }
                *reinterpret_cast<float4*>(o) = v;
            } else {
                const float part[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (m + q < p.M) o[q] = p.beta != 0.0f ? fmaf(p.beta, o[q], part[q]) : part[q];
            }
        }
        cluster_sync();                                              // nobody leaves while its part is being read
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// Columns of a tile.  A short reduction spends its time on C, not on the product: there 64-column tiles, which leave room
// for two C tiles in shared memory, are the faster ones.  Time with them over time without (B200, flushed L2): 25088 x 4096 and
// 4096 x 4096 at K = 64 0.80 .. 0.83, 128 0.97, 192 0.97 .. 1.03, 256 1.06, 384 1.12, 768 1.23; 4096 x 1000 0.89, 1.00, 1.00, 1.07,
// 1.16, 1.21.  Few columns leave SMs idle with wide tiles: 4096 x 200 and 9216 x 300 0.8 .. 0.9 up to K = 384, 1.00 at 1000;
// 1024 x 128 1.00 at 320, 1.14 at 512; 4096 x 32 1.00 at 320, 1.17 at 384.
inline bool short_reduction(int N, int K) { return K <= (N <= 320 ? 320 : 192); }
inline int tile_n(int N, int K) { return N <= 32 ? 32 : (N <= 64 || short_reduction(N, K) ? 64 : 128); }

constexpr int MAX_SPLITS = 8;                                        // CTAs of a portable cluster

// Split of the reduction for the last, partly filled wave of tiles (`rest` of them), the `splits` CTAs of a tile in one
// cluster.  A wave costs its k blocks plus about three for its start, three more for the sum over the cluster, and eight
// (3 us) where it needs a launch of its own after the full waves.  resident(s): clusters of s CTAs that run at once.
// Chosen against the best of 1 .. 8 on 15 shapes (1 .. 200 tiles, K = 512 .. 25088; B200, flushed L2): the same time on 14 of
// them, 2 % more on one (25088 x 64, K = 4096: five parts 113.7 us, two 111.6, none 129).  4096 x 64, K = 25088: four parts 104
// us, three 129, five 160; 9216 x 128, K = 4096: two 60, one 94, three 81; 12800 x 200, K = 640: none 41, two 42.
template <class Resident> inline int plan_splits(long long rest, int kblocks, bool own_launch, Resident resident) {
    int best = 1;
    double best_cost = kblocks + 3.0;
    for (int s = 2; s <= MAX_SPLITS && kblocks / s >= 2; ++s) {
        const int chunk = ceil_div(kblocks, s);
        if (ceil_div(kblocks, chunk) != s) continue;
        const int r = resident(s);
        if (r < 1) continue;
        const double cost = static_cast<double>(ceil_div<long long>(rest, r)) * (chunk + 6.0) + (own_launch ? 8.0 : 0.0);
        if (cost < best_cost) { best_cost = cost; best = s; }
    }
    return best;
}

// What the tensor copies need: 16-byte aligned matrices whose columns are a multiple of 16 bytes apart.
inline bool supported(const float* A, int lda, const float* B, int ldb) {
    return ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15u) == 0 && lda % 4 == 0 && ldb % 4 == 0;
}

inline void cluster_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int ctas, int threads, int smem) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(ctas); attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg->blockDim = dim3(threads);
    cfg->dynamicSmemBytes = smem;
    cfg->attrs = attr; cfg->numAttrs = 1;
}

template <bool AK, bool BKM, int BN, bool STAGED>
int launch_bn(const float* A, int lda, const float* B, int ldb, Params p, int K, cudaStream_t stream) {
    typedef Config<BN, STAGED> Cfg;
    int dev = 0;
    VDNN_CUDA(cudaGetDevice(&dev));
    auto kern = gemm_kernel<AK, BKM, BN, STAGED>;
    VDNN_ALLOW_SHARED(dev, kern, Cfg::SMEM_BYTES);
    CUtensorMap ma, mb;
    int st = AK ? tma::make_matrix_map(&ma, A, K, p.M, lda, BK, BM, CU_TENSOR_MAP_SWIZZLE_128B)
                : tma::make_matrix_map(&ma, A, p.M, K, lda, BM, BK, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (st != VDNN_OK) return st;
    st = BKM ? tma::make_matrix_map(&mb, B, K, p.N, ldb, BK, BN, CU_TENSOR_MAP_SWIZZLE_128B)
             : tma::make_matrix_map(&mb, B, p.N, K, ldb, 32, BK, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B);
    if (st != VDNN_OK) return st;
    CUtensorMap mc = ma;                                             // used by staged launches only
    if (STAGED) {
        st = tma::make_matrix_map(&mc, p.out, p.M, p.N, p.ldc, BM, BN, CU_TENSOR_MAP_SWIZZLE_NONE);
        if (st != VDNN_OK) return st;
    }
    p.tiles_m = ceil_div(p.M, BM); p.kblocks = ceil_div(K, BK);
    const long long tiles = static_cast<long long>(p.tiles_m) * ceil_div(p.N, BN);
    const int sms = sm_count();
    auto run = [&](long long tile0, long long count, int splits) {
        p.tile0 = tile0; p.units = count * splits; p.splits = splits; p.kb_chunk = ceil_div(p.kblocks, splits);
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        cluster_config(&cfg, attr, splits, Cfg::THREADS, Cfg::SMEM_BYTES);
        cfg.stream = stream;
        cfg.gridDim = dim3(static_cast<unsigned>(splits > 1 || p.units < sms ? p.units : sms));
        VDNN_CUDA(cudaLaunchKernelEx(&cfg, kern, ma, mb, mc, p));
        VDNN_LAUNCHED();
        return static_cast<int>(VDNN_OK);
    };
    auto resident = [&](int s) {
        // a property of kernel and device: asked for once
        static std::atomic<int> known[64][MAX_SPLITS + 1];
        int n = dev < 64 ? known[dev][s].load(std::memory_order_relaxed) : 0;
        if (n == 0) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            cluster_config(&cfg, attr, s, Cfg::THREADS, Cfg::SMEM_BYTES);
            cfg.gridDim = dim3(static_cast<unsigned>(sms / s * s));
            if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) { (void)cudaGetLastError(); n = -1; }
            if (dev < 64) known[dev][s].store(n, std::memory_order_relaxed);
        }
        return n;
    };
    const long long rest = tiles % sms, full = tiles - rest;
    const int splits = STAGED || rest == 0 ? 1 : plan_splits(rest, p.kblocks, full > 0, resident);
    if (splits == 1) return run(0, tiles, 1);
    st = full > 0 ? run(0, full, 1) : VDNN_OK;
    return st != VDNN_OK ? st : run(full, rest, splits);
}

template <bool AK, bool BKM>
int launch(const float* A, int lda, const float* B, int ldb, const Params& p, int K, cudaStream_t stream) {
    const int bn = tile_n(p.N, K);
    const bool staged = short_reduction(p.N, K) && p.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0;
    if (bn == 32) return staged ? launch_bn<AK, BKM, 32, true>(A, lda, B, ldb, p, K, stream) : launch_bn<AK, BKM, 32, false>(A, lda, B, ldb, p, K, stream);
    if (bn == 64) return staged ? launch_bn<AK, BKM, 64, true>(A, lda, B, ldb, p, K, stream) : launch_bn<AK, BKM, 64, false>(A, lda, B, ldb, p, K, stream);
    return launch_bn<AK, BKM, 128, false>(A, lda, B, ldb, p, K, stream);
}

}  // namespace dense
}  // namespace vdnn
