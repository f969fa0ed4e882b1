// Prefill GEMM for many tokens and tiles (chosen by estimated cost from 65 tokens on, see gemm_launch): y[m, rows] =
// x[m, K] . W[rows, K]^T on pairs of CTAs (tcgen05 cta_group::2).
//
// A pair computes 256 weight rows x up to 256 tokens: one tcgen05.mma of M = 256 spans both SMs, each SM holding its own 128 rows of A
// (dequantized weights, fp16, in TMEM behind the accumulator), HALF of the tokens of B and its own 128 accumulator rows.
// With A in TMEM the MMAs keep the tensor core's pace, 1024 cycles per 128 k and 256 tokens, and take 64 bytes of shared memory a
// cycle of the 128 it can.  (A in shared memory, tiles of 512 tokens with eight dequantization warps: 109 bytes a cycle, 1300 -
// 1500 cycles per 128 k and 256 tokens.)  What bounds it now: in long loops the power cap; in one call, 4 us until the first MMA, 3 - 6
// us behind the last one.
// us a call, tiles of 512 or 256 tokens with A in shared memory / this: Q4_0 [11008 x 4096] 2048 tokens 150 / 139, Q4_K [14336 x 4096]
// 512 tokens 56 / 54, 700 tokens 85 / 76, [3584 x 8192] 1024 tokens 63 / 57, Q8_0 [8192 x 8192] 1024 tokens
// 110 / 109, 2000 tokens 210 / 202.
//
// Warp roles in each CTA (704 threads):
//   warp 0      TMA producer: this CTA's half of a tile's tokens, two spans of 64 k a stage, 128-byte swizzle
//   warp 1      leader (rank 0): issues the pair's MMAs and commits to the barriers of both CTAs;
//               rank 1: one thread tells the leader's `full` barrier that its own TMA data has landed
//   warps 4-7   epilogue of this CTA's 128 rows
//   warps 2,3,8-21  dequantization of this CTA's 128 rows, in two sets that take the stages (128 k) by turns
// One `full` barrier per stage, in the leader: the leader's TMA, a set of dequantization warps of either CTA and rank 1's word
// for its TMA arrive on it.  Everything the MMAs release (`s_empty`, `acc_full`) is committed to both CTAs by multicast.
//
// Work split ("stream-K"): all (tile, k-block) units form one sequence in tile order, cut into equal contiguous shares,
// one per pair, so every SM does the same number of MMA steps whatever the tile count.  Where the weight is larger than what the L2 keeps, each
// pair takes whole tiles first, in step with its neighbours (pair_waves), and the units of what is left are dealt.  A tile cut by a share boundary is
// finished by the pair that holds its first k-block: the pairs holding the rest reach their piece before that (it is the
// head of their share), write it to a scratch buffer and publish the launch number; the owner reaches the tile last,
// when all its warps are free: twelve of them (three per TMEM lane quarter) add the pieces in pair order
// (deterministic) and write y.  Both CTAs of a pair walk the same units, and each hands over and finishes its own rows.
// Every wait is bounded; on expiry the CTA sets a status bit, stops issuing work and still frees its TMEM.
#pragma once
#include "wf_gemm_core.cuh"

namespace wf {

constexpr int PAIR_TOKENS = 256;                         // of a tile, at most
constexpr int PAIR_COLS = 16;                            // tokens that a warp takes out of the accumulator at a time
constexpr int PAIR_SPAN = 128 * 64 * 2;                  // 16 KB: this CTA's 128 of a tile's tokens x 64 k
constexpr int PAIR_STAGE = 2 * PAIR_SPAN;                // 128 k, a unit of the work split
constexpr int PAIR_STAGES = 3;                           // of activations, and of weights in TMEM (64 columns each behind the accumulator)
constexpr int PAIR_SPILL = PAIR_TOKENS * GEMM_BN * 4;    // 128 KB: a segment's sums on their way to memory
constexpr size_t PAIR_SMEM = 1024 + (size_t)PAIR_STAGES * PAIR_STAGE + PAIR_SPILL;

// A pair's units: with WAVES those of p.waves whole tiles (tile w * pairs + pair) first, then its share of the units of the tiles behind the
// waves.  One counter runs over them: it has the number among those units in the share, [v0, v1), and begins waves * k_blocks below v0.
// They are walked in segments: a segment is a run of k-blocks of one tile.
__device__ __forceinline__ int share_begin(const GemmParams& p, int pair) { return pair * p.unit_q + min(pair, p.unit_r); }
struct GemmSegment {
    int tile, kb0, kb1;  // k-blocks [kb0, kb1) of `tile`
};
// the segment that starts at unit u (u < u1) of this pair, whose counter began at u0
template <bool WAVES> __device__ __forceinline__ GemmSegment segment_at(const GemmParams& p, int u, int u0, int u1) {
    GemmSegment g;
    if (WAVES && u - u0 < p.waves * p.k_blocks) {
        g.tile = (u - u0) / p.k_blocks * (int)(gridDim.x >> 1) + (int)(blockIdx.x >> 1);
        g.kb0 = 0;
        g.kb1 = p.k_blocks;
        return g;
    }
    g.tile = u / p.k_blocks;
    g.kb0 = u - g.tile * p.k_blocks;
    g.kb1 = min(p.k_blocks, g.kb0 + (u1 - u));
    if (WAVES) g.tile += p.waves * (int)(gridDim.x >> 1);
    return g;
}

// Where a dequant warp's loads stand in the pair's units: they run a few units ahead of the conversions.  rank: which 128 of
// the tile's 256 rows; dq: 16-row tile of the 128.
template <int QT, int KBW, bool WAVES> struct GemmLoadWalk {
    const GemmParams& p;
    int u, u1, tile, kb, row0, waves;  // waves: whole tiles to come, with the present one
    const uint8_t* row = nullptr;
    __device__ __forceinline__ GemmLoadWalk(const GemmParams& p_, int u0, int u1_, int set, int rank, int dq)
        : p(p_), u(u0 + set), u1(u1_), row0(rank * (GEMM_BN / 16) + dq), waves(WAVES ? p_.waves : 0) {
        if (WAVES) {
            tile = (int)(blockIdx.x >> 1);
            kb = set;
            if (kb >= p.k_blocks) advance();
        } else {
            tile = u / p.k_blocks;
            kb = u - tile * p.k_blocks;
        }
        set_row();
    }
    __device__ __forceinline__ void advance() {  // to the tile that kb lies in
        for (; kb >= p.k_blocks; kb -= p.k_blocks) {
            if (!WAVES || waves == 0) {
                tile++;
            } else if (--waves > 0) {
                tile += (int)(gridDim.x >> 1);
            } else {
                const int v0 = share_begin(p, (int)(blockIdx.x >> 1)), t = v0 / p.k_blocks;
                tile = p.waves * (int)(gridDim.x >> 1) + t;
                kb += v0 - t * p.k_blocks;
            }
        }
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
        u += GEMM_SETS;
        kb += GEMM_SETS;
        if (kb < p.k_blocks) return;
        advance();
        set_row();
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

// smem: [0, 1024) barriers + tmem slot | PAIR_STAGES stages, 1024-byte aligned | a segment's sums, PAIR_SPILL
template <int QT, bool WAVES>
__global__ void __launch_bounds__(768, 1) gemm_pair_kernel(const GemmParams p, const __grid_constant__ CUtensorMap xmap) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);           // [3] leader: both CTAs' operands of the stage are in place
    uint64_t* b_full = full + PAIR_STAGES;                        // [3] rank 1: its own TMA data has landed
    uint64_t* s_empty = b_full + PAIR_STAGES;                     // [3] stage consumed by the MMAs
    uint64_t* acc_full = s_empty + PAIR_STAGES;                   // the accumulator holds a segment
    uint64_t* acc_empty = acc_full + 1;                           // leader: the epilogues of both CTAs have read it
    uint64_t* tail_full = acc_empty + 1;                          // the accumulator of the tile shared with the following pairs
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint8_t* stage0 = smem + 1024;

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;
    const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    const int v0 = share_begin(p, pair), u0 = v0 - (WAVES ? p.waves * p.k_blocks : 0), u1 = share_begin(p, pair + 1);
    constexpr int KBW = Tile<QT>::K / GEMM_BK;  // units per weight k-tile

    // Dequantization warps: the first weights are requested before all set-up; which warp takes what: see the cluster kernel.
    const bool dequant = warp >= 8 || warp == 2 || warp == 3;
    const int nth = warp < 4 ? 0 : (warp - 8 - (warp & 3)) / 4 + ((warp & 3) >> 1);
    const int set = nth >> 1, dq = 2 * (warp & 3) + (nth & 1);
    constexpr int DEPTH = 2;  // units a warp holds: one is converted while the other loads
    DequantRegs<QT> r[DEPTH][2];
    GemmLoadWalk<QT, KBW, WAVES> walk(p, u0, u1, set, (int)rank, dq);
    if (dequant) {
#pragma unroll
        for (int d = 0; d < DEPTH; d++) walk.next(r[d], lane);
    }
    if (warp == 0) {  // a barrier per lane
        if (lane == 0) {
            prefetch_tensormap(&xmap);
            *abort_flag = 0;
        }
        // full: two TMA producers, eight dequantization warps of either CTA; acc_empty: four epilogue warps of either CTA
        if (lane < 3 * PAIR_STAGES + 3) g_mbar_init(full + lane, lane < PAIR_STAGES ? 2 * GEMM_DEQUANT_WARPS + 2 : lane == 3 * PAIR_STAGES + 1 ? 8 : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the other CTA's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot, a_tmem = tmem_base + PAIR_TOKENS;

    auto fail = [&]() {
        report_status(p.status, STATUS_GEMM_PIPE_TIMEOUT);
        *abort_flag = 1;
    };
    if (warp == 0) {
        // ------------------------------------------------ TMA producer: this CTA's tokens
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");  // the fp16 activations
            StageCursor at;
            for (int u = u0; u < u1 && !*abort_flag;) {
                const GemmSegment g = segment_at<WAVES>(p, u, u0, u1);
                const int tok0 = (g.tile % p.m_tiles) * p.bm + (int)rank * (p.bm >> 1);
                for (int kb = g.kb0; kb < g.kb1; kb++, at.advance(PAIR_STAGES)) {
                    const int s = at.s;
                    if (!g_mbar_wait(&s_empty[s], at.phase ^ 1)) { fail(); break; }
                    uint8_t* b_stage = stage0 + (size_t)s * PAIR_STAGE;
                    uint64_t* bar = leader ? &full[s] : &b_full[s];
                    g_mbar_expect_tx(bar, (uint32_t)p.bm * 128);
                    tma_load_2d(b_stage, &xmap, kb * GEMM_BK, tok0, bar);
                    tma_load_2d(b_stage + PAIR_SPAN, &xmap, kb * GEMM_BK + 64, tok0, bar);
                }
                u += g.kb1 - g.kb0;
            }
        }
    } else if (warp == 1) {
        asm volatile("griddepcontrol.wait;" ::: "memory");  // no bounded wait starts while earlier kernels of the stream run
        if (leader) {
            // ------------------------------------------------ MMA issuer of the pair (the whole warp walks the loop)
            const uint32_t issue = elect_one();
            const uint64_t b_desc0 = smem_desc_sw128(g_smem_u32(stage0));
            StageCursor at;
            int local = 0;
            for (int u = u0; u < u1 && !*abort_flag; local++) {
                const GemmSegment g = segment_at<WAVES>(p, u, u0, u1);
                bool ok = true;
                // the epilogues must have read the segment before this one
                if (local > 0 && !g_mbar_wait(acc_empty, (local - 1) & 1)) { fail(); break; }
                tc_fence_after();
                for (int kb = g.kb0; kb < g.kb1; kb++) {
                    const int s = at.s;
                    if (!g_mbar_wait(&full[s], at.phase)) { fail(); ok = false; break; }
                    tc_fence_after();
                    const uint64_t bd = b_desc0 + (uint64_t)(s * (PAIR_STAGE >> 4));
                    const uint32_t ad = a_tmem + (uint32_t)(s * 64);
                    tc_mma_span<2>(tmem_base, ad, bd, p.idesc, (uint32_t)(kb - g.kb0), issue);
                    tc_mma_span<2>(tmem_base, ad + 32, bd + (PAIR_SPAN >> 4), p.idesc, 1u, issue);
                    if (issue) tc_commit_pair(&s_empty[s]);
                    at.advance(PAIR_STAGES);
                }
                if (!ok) break;
                if (issue) {
                    tc_commit_pair(acc_full);
                    if (g.kb0 == 0 && g.kb1 < p.k_blocks) tc_commit_pair(tail_full);
                }
                u += g.kb1 - g.kb0;
            }
        } else if (lane == 0) {
            // ------------------------------------------------ rank 1: pass the word on that its TMA data has landed
            const int n = u1 - u0;
            StageCursor at;
            for (int it = 0; it < n && !*abort_flag; it++, at.advance(PAIR_STAGES)) {
                if (!g_mbar_wait(&b_full[at.s], at.phase)) { fail(); break; }
                mbar_arrive_cluster(map_to_rank(g_smem_u32(&full[at.s]), 0));
            }
        }
    } else if (warp >= 4 && warp < 8) {
        // ------------------------------------------------ epilogue (TMEM lane quarter = warp % 4), this CTA's 128 rows.
        // Every segment except the tile this pair owns the beginning of and shares with the following pairs.
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        int local = 0;
        asm volatile("griddepcontrol.wait;" ::: "memory");  // the row scales; gen
        unsigned int launch_gen = ld_acquire_u32(p.gen) + 1u;  // this launch's generation: see GemmParams
        if (launch_gen == 0u) launch_gen = 1u;                 // 0 is what untouched flags hold
        float* mine = p.partial + (size_t)blockIdx.x * GEMM_PIECE_TOKENS * GEMM_BN;
        uint4* const spill = reinterpret_cast<uint4*>(stage0 + PAIR_STAGES * PAIR_STAGE) + row;  // [tokens / 4][128 rows]
        for (int u = u0; u < u1 && !*abort_flag; local++) {
            const GemmSegment g = segment_at<WAVES>(p, u, u0, u1);
            const int nt = g.tile / p.m_tiles, mt = g.tile % p.m_tiles;
            const int n = nt * (2 * GEMM_BN) + (int)rank * GEMM_BN + row;
            const bool starts = g.kb0 == 0, ends = g.kb1 == p.k_blocks;
            if (starts && !ends) break;
            if (!g_mbar_wait(acc_full, local & 1)) { if (lane == 0) fail(); break; }
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
            // Through shared memory, so that the MMAs of the next segment wait for no store to global memory (this CTA's sums straight from
            // the accumulator to memory: 5500 cycles a segment; [11008 x 4096] Q4_0 2048 tokens 145 -> 136 us a call).
            const int cols = min(p.bm, p.m - mt * p.bm);
            for (int c = 0; c < cols; c += 32) {
                uint32_t v[32];
                tmem_ld32(taddr + (uint32_t)c, v);
#pragma unroll
                for (int j = 0; j < 8; j++) spill[(c / 4 + j) * GEMM_BN] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            }
            tc_fence_before();  // the accumulator has been read: the MMA issuer may overwrite it
            __syncwarp();
            // nobody waits for the last segment's word, which could come after the leader has left
            if (lane == 0 && u + g.kb1 - g.kb0 < u1) mbar_arrive_cluster(map_to_rank(g_smem_u32(acc_empty), 0));
            for (int c = 0; c < cols; c += PAIR_COLS) {  // a lane reads what it wrote
                uint32_t v[PAIR_COLS];
#pragma unroll
                for (int j = 0; j < PAIR_COLS / 4; j++) {
                    const uint4 q = spill[(c / 4 + j) * GEMM_BN];
                    v[4 * j] = q.x, v[4 * j + 1] = q.y, v[4 * j + 2] = q.z, v[4 * j + 3] = q.w;
                }
                if (!starts) write_piece_chunk(mine, v, c, row);
                else store_chunk(p.y, p.ldy, p.col0, p.row_unscale, v, mt * p.bm + c, p.m, n, p.rows);
            }
            if (!starts) {  // publish this warp's 32 rows of the piece
                __threadfence();
                __syncwarp();
                if (lane == 0) st_release_u32(p.ready + blockIdx.x * 4 + quarter, launch_gen);
            }
            u += g.kb1 - g.kb0;
        }
    } else {
        // ------------------------------------------------ dequantization warps (a stage: see the cluster kernel)
        const uint32_t full0 = map_to_rank(g_smem_u32(full), 0), a_mine = a_tmem + ((uint32_t)(dq * 16) << 16);
        StageCursor at;
        bool lapped = false;  // from the second lap on a wait is bounded by what earlier kernels let this one do
        auto advance = [&]() { lapped |= at.advance(PAIR_STAGES); };
        auto convert = [&](const DequantRegs<QT> (&regs)[2], auto sub, uint4 (&out)[2][2]) {
#pragma unroll
            for (int hh = 0; hh < 2; hh++) regs[hh].template pair<decltype(sub)::value>(out[hh][0], out[hh][1]);
        };
        auto finish_step = [&](const DequantRegs<QT> (&regs)[2]) {
            uint4 out[2][2];
            convert(regs, std::integral_constant<int, 0>{}, out);
            if (lapped) {
                asm volatile("griddepcontrol.wait;" ::: "memory");
                lapped = false;
            }
            if (!g_mbar_wait(&s_empty[at.s], at.phase ^ 1)) {
                if (lane == 0) fail();
                return false;
            }
            tc_fence_after();
            const uint32_t to = a_mine + (uint32_t)(at.s * 64);
            tmem_st_span(to, out[0][0], out[0][1], out[1][0], out[1][1]);
            convert(regs, std::integral_constant<int, 1>{}, out);
            tmem_st_span(to + 32, out[0][0], out[0][1], out[1][0], out[1][1]);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(full0 + (uint32_t)at.s * 8);
            advance();
            return true;
        };
        if (set > 0) advance();
        bool ok = true;
        for (int u = u0 + set; u < u1 && ok && !*abort_flag; u += GEMM_SETS * DEPTH) {
#pragma unroll
            for (int d = 0; d < DEPTH; d++) {
                if (u + d * GEMM_SETS >= u1) break;
                ok = finish_step(r[d]);
                if (!ok) break;
                walk.next(r[d], lane);
                advance();  // over the other set's stage
            }
        }
    }

    // ------------------------------------------------ the tile whose beginning this pair owns and whose rest lies in the
    // following pairs: the last segment of the share.  Twelve warps (three per TMEM lane quarter) add the pieces of
    // this CTA's rows in pair order and write y.
    __syncwarp();
    if (v0 < u1 && warp < 12) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        unsigned int launch_gen = ld_acquire_u32(p.gen) + 1u;
        if (launch_gen == 0u) launch_gen = 1u;
        const int t = (u1 - 1) / p.k_blocks, tile = t + (WAVES ? p.waves * pairs : 0);  // t: among the tiles behind the waves
        const int kb0 = max(v0, t * p.k_blocks) - t * p.k_blocks, kb1 = u1 - t * p.k_blocks;
        if (kb0 == 0 && kb1 < p.k_blocks) {
            const int quarter = warp & 3, slice = warp >> 2;
            const int row = quarter * 32 + lane;
            const int nt = tile / p.m_tiles, mt = tile % p.m_tiles;
            const int n = nt * (2 * GEMM_BN) + (int)rank * GEMM_BN + row;
            int last_pair = pair;
            bool ok = !*abort_flag;
            const int tile_end = (t + 1) * p.k_blocks;
            for (int c = pair + 1; c < pairs && ok; c++) {
                if (share_begin(p, c) >= tile_end) break;
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
            const int chunks = (min(p.bm, p.m - mt * p.bm) + PAIR_COLS - 1) / PAIR_COLS;  // dealt to the three warps of a quarter
            float4 v[PAIR_COLS / 4];
            auto fetch = [&](int cc, int ci) { load_piece_chunk(p.partial + (size_t)(2 * cc + (int)rank) * GEMM_PIECE_TOKENS * GEMM_BN, v, ci * PAIR_COLS, row); };
            if (ok && slice < chunks) fetch(pair + 1, slice);  // the next pair always holds a piece
            for (int ci = slice; ci < chunks && ok; ci += 3) {
                uint32_t a[PAIR_COLS];
                tmem_ld16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ci * PAIR_COLS), a);
                add_piece_chunk(a, v);
                for (int cc = pair + 2; cc <= last_pair; cc++) {  // pieces in pair order
                    fetch(cc, ci);
                    add_piece_chunk(a, v);
                }
                if (ci + 3 < chunks) fetch(pair + 1, ci + 3);  // under the stores of this one
                store_chunk(p.y, p.ldy, p.col0, p.row_unscale, a, mt * p.bm + ci * PAIR_COLS, p.m, n, p.rows);
            }
        }
    }

    // ------------------------------------------------ teardown: neither CTA leaves (or frees TMEM) while the other may still
    // arrive on its barriers or the pair's MMAs may still read its operands
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1 && *abort_flag) drain_after_abort();  // operands and MMAs that nobody waited for, in either CTA
    __syncwarp();
    // relaxed: what either CTA did in the other's shared memory has been waited for, and nobody waits here for stores of y
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
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
