// Prefill GEMM for many tokens and tiles (chosen by estimated cost from 65 tokens on, see gemm_launch): y[m, rows] =
// x[m, K] . W[rows, K]^T on pairs of CTAs (tcgen05 cta_group::2).
//
// A pair computes 256 weight rows x 512 tokens (or 256, where there are few tiles): one tcgen05.mma of M = 256, N = 256 spans both SMs, each SM holding its
// own 128 rows of A (dequantized weights, fp16), HALF of the tokens of B and its own 128 accumulator rows in TMEM.
// What bounds the kernel is shared memory and power: per 64 k and 512 tokens (1024 MMA cycles) an SM moves 16 KB of A
// in by generic stores, 32 KB of B in by TMA, and 32 + 32 KB out to the tensor core -- 109 bytes per cycle of the 128 it
// can.  One CTA alone had to hold and read all of B: 172 bytes per cycle, and half the stages.
// Measured (Q4_0 [11008 x 4096], 2048 tokens): 171 us = 1.08 PFLOP/s against 217 us for one CTA per tile; Q4_K
// [14336 x 4096], 512 tokens: 65 us against 76 us.
//
// Warp roles in each CTA (448 threads):
//   warp 0      TMA producer: this CTA's tokens of a stage, [128 tokens x 64 k] per 256-token half, 128-byte swizzle
//   warp 1      leader (rank 0): issues the pair's MMAs and commits to the barriers of both CTAs;
//               rank 1: one thread tells the leader's `full` barrier that its own TMA data has landed
//   warps 4-7   epilogue of this CTA's 128 rows
//   warps 2,3,8-13  dequantization of this CTA's 128 rows
// One `full` barrier per stage, in the leader: the leader's TMA, eight dequant warps of either CTA and rank 1's word for
// its TMA arrive on it.  Everything the MMAs release (`s_empty`, `acc_full`) is committed to both CTAs by multicast.
//
// Work split ("stream-K"): all (tile, k-block) units form one sequence in tile order, cut into equal contiguous shares,
// one per pair, so every SM does the same number of MMA steps whatever the tile count.  A tile cut by a share boundary is
// finished by the pair that holds its first k-block: the pairs holding the rest reach their piece first (it is the
// head of their share), write it to a scratch buffer and publish the launch number; the owner reaches the tile last,
// when all its warps are free: twelve of them (three per TMEM lane quarter) add the pieces in pair order
// (deterministic) and write y.  Both CTAs of a pair walk the same units, and each hands over and finishes its own rows.
// Every wait is bounded; on expiry the CTA sets a status bit, stops issuing work and still frees its TMEM.
#pragma once
#include "wf_gemm_core.cuh"

namespace wf {

constexpr int PAIR_BK = 64;                              // k per stage; a unit of the work split is 128 k, two stages
constexpr int PAIR_A_BYTES = GEMM_BN * PAIR_BK * 2;      // 16 KB: this CTA's weight rows
constexpr int PAIR_B_HALF = 128 * PAIR_BK * 2;           // 16 KB: this CTA's 128 of a half's 256 tokens
constexpr int PAIR_MAX_STAGES = 8;
inline __host__ __device__ int pair_stage_bytes(int halves) { return PAIR_A_BYTES + halves * PAIR_B_HALF; }

// A pair's share of the unit sequence, cut into segments: a segment is a run of k-blocks of one tile.
struct GemmSegment {
    int tile, kb0, kb1;  // k-blocks [kb0, kb1) of `tile`
};
__device__ __forceinline__ void pair_units(const GemmParams& p, int pair, int& u0, int& u1) {
    u0 = pair * p.unit_q + min(pair, p.unit_r);
    u1 = u0 + p.unit_q + (pair < p.unit_r ? 1 : 0);
}
// the segment that starts at unit u (u < u1)
__device__ __forceinline__ GemmSegment segment_at(const GemmParams& p, int u, int u1) {
    GemmSegment g;
    g.tile = u / p.k_blocks;
    g.kb0 = u - g.tile * p.k_blocks;
    g.kb1 = min(p.k_blocks, g.kb0 + (u1 - u));
    return g;
}

// Where a dequant warp's loads stand in the pair's units: they run a few units ahead of the conversions.  rank: which 128 of
// the tile's 256 rows; dq: 16-row tile of the 128.
template <int QT, int KBW> struct GemmLoadWalk {
    const GemmParams& p;
    int u, u1, tile, kb, row0;
    const uint8_t* row = nullptr;
    __device__ __forceinline__ GemmLoadWalk(const GemmParams& p_, int u0, int u1_, int rank, int dq)
        : p(p_), u(u0), u1(u1_), tile(u0 / p_.k_blocks), kb(u0 - tile * p_.k_blocks), row0(rank * (GEMM_BN / 16) + dq) {
        set_row();
    }
    __device__ __forceinline__ void set_row() {  // rows behind the buffer's last tile are computed and never stored
        const int64_t rt = min((int64_t)(tile / p.m_tiles) * (2 * GEMM_BN / 16) + row0, (int64_t)p.rt_last);
        row = p.tiles + rt * p.kt_w * (int64_t)Tile<QT>::BYTES;
    }
    __device__ __forceinline__ void next(DequantRegs<QT> (&regs)[2], int lane) {
        if (u >= u1) return;
        const uint8_t* t = row + (size_t)(kb / KBW) * Tile<QT>::BYTES;
        regs[0].load(t, kb % KBW, lane, 0);
        regs[1].load(t, kb % KBW, lane, 1);
        u++;
        if (++kb == p.k_blocks) {
            kb = 0;
            tile++;
            set_row();
        }
    }
};

__device__ __forceinline__ void tmem_alloc_pair(void* smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(g_smem_u32(smem_dst)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// arrive on the barrier at this offset in both CTAs once the MMAs issued so far have finished
__device__ __forceinline__ void tc_commit_pair(void* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(g_smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}

// smem: [0, 1024) barriers + tmem slot | stages x (A 16 KB | B halves x 16 KB), 1024-byte aligned
template <int QT>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_pair_kernel(const GemmParams p, const __grid_constant__ CUtensorMap xmap) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);           // [8] leader: both CTAs' operands of the stage are in place
    uint64_t* b_full = full + PAIR_MAX_STAGES;                    // [8] rank 1: its own TMA data has landed
    uint64_t* s_empty = b_full + PAIR_MAX_STAGES;                 // [8] stage consumed by the MMAs
    uint64_t* acc_full = s_empty + PAIR_MAX_STAGES;               // [2] one per accumulator
    uint64_t* acc_empty = acc_full + 2;                           // [2] leader: the epilogues of both CTAs have read it
    uint64_t* tail_full = acc_empty + 2;                          // the accumulators of the tile shared with the following pairs
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const bool wide = p.halves == 2;
    const int tile_tokens = p.halves * 256;
    const uint32_t stage_bytes = (uint32_t)pair_stage_bytes(p.halves);
    uint8_t* stage0 = smem + 1024;

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;
    const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    const int stages = p.stages;
    int u0, u1;
    pair_units(p, pair, u0, u1);
    constexpr int KBW = Tile<QT>::K / GEMM_BK;  // units per weight k-tile

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            g_mbar_init(&full[s], 2 * GEMM_DEQUANT_WARPS + 2);
            g_mbar_init(&b_full[s], 1);
            g_mbar_init(&s_empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            g_mbar_init(&acc_full[b], 1);
            g_mbar_init(&acc_empty[b], 8);  // four epilogue warps of either CTA
        }
        g_mbar_init(tail_full, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the other CTA's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    auto fail = [&]() {
        report_status(p.status, STATUS_GEMM_PIPE_TIMEOUT);
        *abort_flag = 1;
    };
    // 256-token halves of token tile mt that hold tokens
    auto halves_of = [&](int mt) { return wide && p.m - mt * 512 > 256 ? 2 : 1; };
    // Accumulators are TMEM columns 0 .. 255 and 256 .. 511: one per half of a tile, or by turns for tiles of one half (`local`
    // counts the segments).  used[acc] counts the uses so far.

    if (warp == 0) {
        // ------------------------------------------------ TMA producer: this CTA's tokens
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");  // the fp16 activations
            StageCursor at;
            for (int u = u0; u < u1 && !*abort_flag;) {
                const GemmSegment g = segment_at(p, u, u1);
                const int mt = g.tile % p.m_tiles, nh = halves_of(mt);
                for (int kb = 2 * g.kb0; kb < 2 * g.kb1; kb++, at.advance(stages)) {  // in stages
                    const int s = at.s;
                    if (!g_mbar_wait(&s_empty[s], at.phase ^ 1)) { fail(); break; }
                    uint8_t* b_stage = stage0 + (size_t)s * stage_bytes + PAIR_A_BYTES;
                    uint64_t* bar = leader ? &full[s] : &b_full[s];
                    g_mbar_expect_tx(bar, (uint32_t)nh * PAIR_B_HALF);
                    for (int h = 0; h < nh; h++)
                        tma_load_2d(b_stage + h * PAIR_B_HALF, &xmap, kb * PAIR_BK, mt * tile_tokens + h * 256 + (int)rank * 128, bar);
                }
                u += g.kb1 - g.kb0;
            }
        }
    } else if (warp == 1) {
        asm volatile("griddepcontrol.wait;" ::: "memory");  // no bounded wait starts while earlier kernels of the stream run
        if (leader) {
            // ------------------------------------------------ MMA issuer of the pair (the whole warp walks the loop)
            const uint32_t issue = elect_one();
            const uint64_t a_desc0 = smem_desc_sw128(g_smem_u32(stage0)), b_desc0 = smem_desc_sw128(g_smem_u32(stage0) + PAIR_A_BYTES);
            StageCursor at;
            int local = 0, used[2] = {0, 0};
            for (int u = u0; u < u1 && !*abort_flag; local++) {
                const GemmSegment g = segment_at(p, u, u1);
                const int nh = halves_of(g.tile % p.m_tiles);
                bool ok = true;
                for (int kb = 2 * g.kb0; kb < 2 * g.kb1 && ok; kb++) {
                    const int s = at.s;
                    if (!g_mbar_wait(&full[s], at.phase)) { fail(); ok = false; break; }
                    tc_fence_after();
                    const uint64_t off = (uint64_t)((uint32_t)s * stage_bytes >> 4);
                    for (int h = 0; h < nh; h++) {
                        const int acc = wide ? h : (local & 1);
                        if (kb == 2 * g.kb0 && used[acc] >= 1) {  // the epilogues must have drained this accumulator's previous tile
                            if (!g_mbar_wait(&acc_empty[acc], (used[acc] - 1) & 1)) { fail(); ok = false; break; }
                            tc_fence_after();
                        }
                        tc_mma_span<2>(tmem_base + (uint32_t)(acc * 256), a_desc0 + off, b_desc0 + off + (uint64_t)(h * (PAIR_B_HALF >> 4)), p.idesc,
                                       (uint32_t)(kb - 2 * g.kb0), issue);
                        if (kb == 2 * g.kb1 - 1) {
                            if (issue) tc_commit_pair(&acc_full[acc]);
                            used[acc]++;
                        }
                    }
                    if (!ok) break;
                    if (issue) tc_commit_pair(&s_empty[s]);
                    at.advance(stages);
                }
                if (!ok) break;
                if (issue && g.kb0 == 0 && g.kb1 < p.k_blocks) tc_commit_pair(tail_full);
                u += g.kb1 - g.kb0;
            }
        } else if (lane == 0) {
            // ------------------------------------------------ rank 1: pass the word on that its TMA data has landed
            const int n = 2 * (u1 - u0);
            StageCursor at;
            for (int it = 0; it < n && !*abort_flag; it++, at.advance(stages)) {
                if (!g_mbar_wait(&b_full[at.s], at.phase)) { fail(); break; }
                mbar_arrive_cluster(map_to_rank(g_smem_u32(&full[at.s]), 0));
            }
        }
    } else if (warp >= 4 && warp < 8) {
        // ------------------------------------------------ epilogue (TMEM lane quarter = warp % 4), this CTA's 128 rows.
        // Every segment except the tile this pair owns the beginning of and shares with the following pairs.
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        int local = 0, used[2] = {0, 0};
        bool dead = false;
        asm volatile("griddepcontrol.wait;" ::: "memory");  // the row scales; gen
        unsigned int launch_gen = ld_acquire_u32(p.gen) + 1u;  // this launch's generation: see GemmParams
        if (launch_gen == 0u) launch_gen = 1u;                 // 0 is what untouched flags hold
        float* mine = p.partial + (size_t)blockIdx.x * GEMM_PIECE_TOKENS * GEMM_BN;
        for (int u = u0; u < u1 && !*abort_flag && !dead; local++) {
            const GemmSegment g = segment_at(p, u, u1);
            const int nt = g.tile / p.m_tiles, mt = g.tile % p.m_tiles;
            const int n = nt * (2 * GEMM_BN) + (int)rank * GEMM_BN + row;
            const bool starts = g.kb0 == 0, ends = g.kb1 == p.k_blocks;
            if (starts && !ends) break;
            const int parts = halves_of(mt);
            for (int h = 0; h < parts; h++) {
                const int acc = wide ? h : (local & 1);
                if (!g_mbar_wait(&acc_full[acc], used[acc] & 1)) { if (lane == 0) fail(); dead = true; break; }
                tc_fence_after();
                used[acc]++;
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * 256);
                for (int c = 0; c < 256; c += 32) {
                    uint32_t r[32];
                    tmem_ld32(taddr + (uint32_t)c, r);
                    if (!starts) write_piece_chunk(mine, r, h * 256 + c, row);
                    else store_chunk(p.y, p.ldy, p.col0, p.row_unscale, r, mt * tile_tokens + h * 256 + c, p.m, n, p.rows);
                }
                tc_fence_before();  // the accumulator has been read: the MMA issuer may overwrite it
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(map_to_rank(g_smem_u32(&acc_empty[acc]), 0));
            }
            if (dead) break;
            if (!starts) {  // publish this warp's 32 rows of the piece
                __threadfence();
                __syncwarp();
                if (lane == 0) st_release_u32(p.ready + blockIdx.x * 4 + quarter, launch_gen);
            }
            u += g.kb1 - g.kb0;
        }
    } else {
        // ------------------------------------------------ dequant warps 2, 3, 8 ..: one 16-row tile each per stage
        const int dq = (warp < 4) ? warp - 2 : warp - 6;  // 16-row tile of the 128 rows
        const int dg = lane >> 2, dq4 = lane & 3;
        const uint32_t full0 = map_to_rank(g_smem_u32(full), 0);
        // store addresses: the chunks of the lane's group in rows dg and dg + 8
        uint8_t* const a_mine = stage0 + (dq * 16 + dg) * 128;
        uint32_t a_off[2];
#pragma unroll
        for (int j = 0; j < 2; j++) a_off[j] = (uint32_t)((stage_chunk(j, dq4) ^ dg) << 4);
        // convert first, wait for the stage then, so that only the stores lie between "released" and "full"
        StageCursor at;
        auto finish_step = [&](const auto& regs, auto sub) {
            const int s = at.s;
            uint4 out[2][2];
#pragma unroll
            for (int hh = 0; hh < 2; hh++) regs[hh].template pair<decltype(sub)::value>(out[hh][0], out[hh][1]);
            if (!g_mbar_wait(&s_empty[s], at.phase ^ 1)) {
                if (lane == 0) fail();
                return false;
            }
            uint8_t* a_stage = a_mine + (size_t)s * stage_bytes;
#pragma unroll
            for (int hh = 0; hh < 2; hh++)
#pragma unroll
                for (int j = 0; j < 2; j++) *reinterpret_cast<uint4*>(a_stage + hh * 1024 + a_off[j]) = out[hh][j];
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic writes -> visible to the tensor core
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(full0 + (uint32_t)s * 8);
            if (at.advance(stages)) asm volatile("griddepcontrol.wait;" ::: "memory");  // no bounded wait under earlier kernels
            return true;
        };
        constexpr int DEPTH = 3;  // register sets in turn, 128 k each
        DequantRegs<QT> r[DEPTH][2];
        GemmLoadWalk<QT, KBW> walk(p, u0, u1, (int)rank, dq);
#pragma unroll
        for (int d = 0; d < DEPTH - 1; d++) walk.next(r[d], lane);
        bool ok = true;
        for (int u = u0; u < u1 && ok && !*abort_flag; u += DEPTH) {
#pragma unroll
            for (int d = 0; d < DEPTH; d++) {
                if (u + d >= u1) break;
                walk.next(r[(d + DEPTH - 1) % DEPTH], lane);
                if (!finish_step(r[d], std::integral_constant<int, 0>{}) || !finish_step(r[d], std::integral_constant<int, 1>{})) { ok = false; break; }
            }
        }
    }

    // ------------------------------------------------ the tile whose beginning this pair owns and whose rest lies in the
    // following pairs: the last segment of the share.  Twelve warps (three per TMEM lane quarter) add the pieces of
    // this CTA's rows in pair order and write y.
    __syncwarp();
    if (u0 < u1 && warp < 12) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        unsigned int launch_gen = ld_acquire_u32(p.gen) + 1u;
        if (launch_gen == 0u) launch_gen = 1u;
        const int tile = (u1 - 1) / p.k_blocks;
        const int kb0 = max(u0, tile * p.k_blocks) - tile * p.k_blocks, kb1 = u1 - tile * p.k_blocks;
        if (kb0 == 0 && kb1 < p.k_blocks) {
            const int quarter = warp & 3, slice = warp >> 2;
            const int row = quarter * 32 + lane;
            const int nt = tile / p.m_tiles, mt = tile % p.m_tiles;
            const int n = nt * (2 * GEMM_BN) + (int)rank * GEMM_BN + row;
            int local = 0;  // number of this segment
            for (int u = u0; u < u1; local++) {
                const GemmSegment g = segment_at(p, u, u1);
                if (g.tile == tile) break;
                u += g.kb1 - g.kb0;
            }
            const uint32_t col0 = wide ? 0u : (uint32_t)((local & 1) * 256);
            int last_pair = pair;
            bool ok = !*abort_flag;
            const int tile_end = (tile + 1) * p.k_blocks;
            for (int c = pair + 1; c < pairs && ok; c++) {
                int c0, c1;
                pair_units(p, c, c0, c1);
                if (c0 >= tile_end) break;
                last_pair = c;  // no share is empty
                int spins = 0;
                while (ld_acquire_u32(p.ready + (2 * c + (int)rank) * 4 + quarter) != launch_gen && ++spins < GEMM_POLL_SPINS) __nanosleep(64);
                if (spins >= GEMM_POLL_SPINS) ok = false;
            }
            // A barrier of its own: warps other than the epilogue's have not followed the phases of acc_full, and may get
            // here while it is still two phases behind, where a parity wait would take the older phase for this one.
            if (ok && !g_mbar_wait(tail_full, 0)) ok = false;
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (!ok && lane == 0) fail();
            tc_fence_after();
            const int chunks = halves_of(mt) * 8;  // of 32 tokens, dealt to the three warps of a quarter
            float4 v[8];
            auto fetch = [&](int cc, int ci) { load_piece_chunk(p.partial + (size_t)(2 * cc + (int)rank) * GEMM_PIECE_TOKENS * GEMM_BN, v, ci * 32, row); };
            if (ok && slice < chunks) fetch(pair + 1, slice);  // the next pair always holds a piece
            for (int ci = slice; ci < chunks && ok; ci += 3) {
                uint32_t r[32];
                tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + col0 + (uint32_t)(ci * 32), r);
                add_piece_chunk(r, v);
                for (int cc = pair + 2; cc <= last_pair; cc++) {  // pieces in pair order
                    fetch(cc, ci);
                    add_piece_chunk(r, v);
                }
                if (ci + 3 < chunks) fetch(pair + 1, ci + 3);  // under the stores of this one
                store_chunk(p.y, p.ldy, p.col0, p.row_unscale, r, mt * tile_tokens + ci * 32, p.m, n, p.rows);
            }
        }
    }

    // ------------------------------------------------ teardown: neither CTA leaves (or frees TMEM) while the other may still
    // arrive on its barriers or the pair's MMAs may still read its operands
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1 && *abort_flag) drain_after_abort();  // operands and MMAs that nobody waited for, in either CTA
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
    if (threadIdx.x == 0) {  // the last CTA out closes the generation
        asm volatile("griddepcontrol.wait;" ::: "memory");
        __threadfence();
        if (atomicAdd(p.gen + 1, 1u) == gridDim.x - 1) {
            p.gen[1] = 0u;
            __threadfence();
            const unsigned int g = ld_acquire_u32(p.gen) + 1u;
            st_release_u32(p.gen, g == 0u ? 1u : g);
        }
    }
}

}  // namespace wf
