// GEMM for few tokens, few tiles, or fp32 tokens: y[m, rows] = x[m, K] . W[rows, K]^T, one tile of 128 weight rows x BM
// (at most 128) tokens per cluster of S CTAs, which split its K.
//
// What bounds these calls is latency: a [4096 x 4096] weight has 32 tiles for 148 SMs, so K has to be split, and then the
// time goes into putting the parts together.  As stream-K shares whose pieces travel through global memory to the one
// CTA that owns the tile (write, fence, flag, poll, read up to four pieces) that took 8 - 14 us of 16 - 25 us.  Here every
// CTA sends each token of its accumulator to the rank that finishes it, by asynchronous stores straight into that CTA's
// shared memory which count themselves on its barrier; each rank adds its tokens' S parts in rank order (deterministic)
// and stores them.  No CTA has more to finish than another, and nothing goes through L2.
// Measured, 64 tokens, Q4_0 [4096 x 4096]: 14.2 us a call, 16.8 us as stream-K shares; 33 tokens of [1000 x 1024]: 7.5 us.
//
// Warp roles (448 threads):
//   warp 0      TMA producer: activation spans [BM tokens x 64 k], 128-byte swizzle
//   warp 1      MMA issuer; owns TMEM
//   warps 4-7   epilogue (TMEM lane quarter = warp % 4): accumulator -> the ranks' exchange buffers -> y
//   warps 2,3,8-13  dequantization: quantized tiles from global memory -> fp16 rows in the swizzled A stage
// A stage is 64 k.  The accumulator is double buffered in TMEM, so a tile is put together while the next one is computed.
// Every wait is bounded; on expiry the CTA sets a status bit, stops issuing work and still frees its TMEM.  Warps leave their
// loops on their own, so there is no barrier between some of them: they meet on mbarriers, whose waits are bounded, and
// all together at the end.
//
// PIECES 1, PLANES 1: bf16 tokens, weights rounded once to fp16.
// PIECES 2, PLANES 3: fp32 tokens.  Every weight is two fp16 (its value, and what rounding left), every token value three,
//   x = x0 + x1 + x2, so the products carry what fp32 would: D += hi . x0 and, in a second accumulator so that the small
//   terms do not pass through the rounding of the large sum, E += hi . x1 + hi . x2 + lo . x0 + lo . x1 (lo . x2 is below
//   2^-33 of the product).  The tensor core cuts each partial sum off at fp32 (about 1e-8 of the sum per addition, always
//   towards zero), so the accumulators are drained every FLUSH units and summed in fp32 with rounding: 6e-7 of the result
//   at any K, 2.4e-6 at K = 4096 without.
#pragma once
#include "wf_gemm_core.cuh"

namespace wf {

constexpr int SPLIT_MAX_STAGES = 8, SPLIT_MAX_RANKS = 8, SPLIT_MAX_TOKENS = 128;
constexpr int SPLIT_FLUSH = 4;  // units of 128 k the accumulators of a PIECES 2 kernel take before they are drained

inline __host__ __device__ int split_stage_bytes(int pieces, int planes, int bm) { return pieces * GEMM_BN * 128 + planes * bm * 128; }
// exchange buffer: [S][groups of four tokens a rank finishes][128 rows] float4 | token scales [4 epilogue warps][64]
inline __host__ __device__ int split_groups(int bm, int ranks) { return (bm / 4 + ranks - 1) / ranks; }
inline __host__ __device__ int split_exchange_bytes(int bm, int ranks) { return ranks == 1 ? 0 : ranks * split_groups(bm, ranks) * GEMM_BN * 16 + 1024; }

// smem: [0, 1024) barriers, tmem slot | stages x (A | B), 1024-byte aligned | exchange buffer
template <int QT, int PIECES, int PLANES>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_split_kernel(const GemmParams p, const __grid_constant__ CUtensorMap xmap) {
    constexpr int ACCS = PIECES;
    constexpr int FLUSH = PIECES == 1 ? 1 << 30 : SPLIT_FLUSH;
    constexpr int KBW = Tile<QT>::K / GEMM_BK;  // units per weight k-tile
    constexpr uint32_t A_BYTES = PIECES * GEMM_BN * 128;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* b_full = reinterpret_cast<uint64_t*>(smem);        // [8] activations landed
    uint64_t* a_full = b_full + SPLIT_MAX_STAGES;                // [8] weights dequantized
    uint64_t* s_empty = a_full + SPLIT_MAX_STAGES;               // [8] stage consumed by the MMAs
    uint64_t* acc_full = s_empty + SPLIT_MAX_STAGES;             // [2]
    uint64_t* acc_empty = acc_full + 2;                          // [2]
    uint64_t* ex_full = acc_empty + 2;                           // the parts of this rank's tokens have arrived
    uint64_t* ex_empty = ex_full + 1;                            // every rank has read its exchange buffer
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ex_empty + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t span_bytes = (uint32_t)p.bm * 128;  // 64 k of bm tokens
    const uint32_t stage_bytes = A_BYTES + PLANES * span_bytes;
    const int stages = p.stages, S = p.ranks;
    uint8_t* stage0 = smem + 1024;
    float4* ex = reinterpret_cast<float4*>(stage0 + (size_t)stages * stage_bytes);
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % S, cluster = (int)blockIdx.x / S, clusters = (int)gridDim.x / S;
    const int tiles = p.n_tiles * p.m_tiles;
    const int kb0 = rank * p.k_blocks / S, kb1 = (rank + 1) * p.k_blocks / S;  // this rank's units of every tile; S <= k_blocks
    const int my_tiles = (tiles - cluster + clusters - 1) / clusters;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; s++) {
            g_mbar_init(&b_full[s], 1);
            g_mbar_init(&a_full[s], GEMM_DEQUANT_WARPS);
            g_mbar_init(&s_empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            g_mbar_init(&acc_full[b], 1);
            g_mbar_init(&acc_empty[b], 4);  // four epilogue warps
        }
        g_mbar_init(ex_full, 1);
        g_mbar_init(ex_empty, 4 * S);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    if (S > 1) cluster_sync();  // the other ranks' barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    auto fail = [&]() {
        report_status(p.status, STATUS_GEMM_PIPE_TIMEOUT);
        *abort_flag = 1;
    };

    if (warp == 0) {
        // ------------------------------------------------ TMA producer (activations)
        if (lane == 0) {
            // The next call's conversion, 32 registers a thread, fits beside a CTA of 128 and waits there, and the next GEMM takes each
            // SM as it becomes free (a call of [5003 x 2784], 77 tokens, Q4_0: 12.7 -> 11.6 us; 64 tokens of [4096 x 4096], where shared
            // memory has no room for it beside, 12.7 -> 11.3 all the same).  Placed when the CTA begins its last tile: a conversion
            // that waits beside longer delays clusters of several tiles ([11008 x 4096], 128 tokens, two tiles each: 27.6 us
            // without, 28.9 placed at the start, 27.8 here).  fp32 tokens, whose conversion does not fit: 93 -> 98.
            auto last_tile = [&](int tile) {
                if (PIECES == 1 && tile + clusters >= tiles) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            };
            last_tile(cluster);
            asm volatile("griddepcontrol.wait;" ::: "memory");  // the fp16 activations
            StageCursor at;
            for (int tile = cluster; tile < tiles && !*abort_flag; tile += clusters) {
                const int tok0 = (tile % p.m_tiles) * p.bm;
                if (tile != cluster) last_tile(tile);
                for (int st = 2 * kb0; st < 2 * kb1; st++, at.advance(stages)) {
                    const int s = at.s;
                    if (!g_mbar_wait(&s_empty[s], at.phase ^ 1)) { fail(); break; }
                    uint8_t* b_stage = stage0 + (size_t)s * stage_bytes + A_BYTES;
                    g_mbar_expect_tx(&b_full[s], PLANES * span_bytes);
#pragma unroll
                    for (int pl = 0; pl < PLANES; pl++) tma_load_2d(b_stage + pl * span_bytes, &xmap, st * 64, pl * p.m + tok0, &b_full[s]);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        asm volatile("griddepcontrol.wait;" ::: "memory");  // no bounded wait starts while earlier kernels of the stream run
        const uint32_t issue = elect_one();
        const uint64_t a_desc0 = smem_desc_sw128(g_smem_u32(stage0)), b_desc0 = smem_desc_sw128(g_smem_u32(stage0) + A_BYTES);
        const uint64_t span = span_bytes >> 4;
        StageCursor at;
        int local = 0;
        bool ok = true;
        for (int tile = cluster; tile < tiles && ok && !*abort_flag; tile += clusters) {
            for (int g0 = kb0; g0 < kb1 && ok; local++) {  // groups of units that share an accumulator
                const int g1 = min(kb1, g0 + min(FLUSH, kb1 - g0)), buf = local & 1;
                if (local >= 2 && !g_mbar_wait(&acc_empty[buf], ((local >> 1) - 1) & 1)) { fail(); ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * ACCS * p.bm), e_tmem = d_tmem + (uint32_t)p.bm;
                for (int st = 2 * g0; st < 2 * g1; st++) {
                    const int s = at.s;
                    if (!g_mbar_wait(&b_full[s], at.phase) || !g_mbar_wait(&a_full[s], at.phase)) { fail(); ok = false; break; }
                    tc_fence_after();
                    const uint64_t off = (uint64_t)((uint32_t)s * stage_bytes >> 4);
                    const uint64_t ad = a_desc0 + off, bd = b_desc0 + off;
                    const uint32_t acc = (uint32_t)(st - 2 * g0);
                    tc_mma_span<1>(d_tmem, ad, bd, p.idesc, acc, issue);
                    if (PIECES == 2) {
                        const uint64_t lo = ad + (GEMM_BN * 128 >> 4);
                        tc_mma_span<1>(e_tmem, lo, bd, p.idesc, acc, issue);
                        tc_mma_span<1>(e_tmem, ad, bd + span, p.idesc, 1u, issue);
                        tc_mma_span<1>(e_tmem, lo, bd + span, p.idesc, 1u, issue);
                        tc_mma_span<1>(e_tmem, ad, bd + 2 * span, p.idesc, 1u, issue);
                    }
                    if (issue) tc_commit(&s_empty[s]);  // frees the stage when these MMAs have read it
                    at.advance(stages);
                }
                if (ok && issue) tc_commit(&acc_full[buf]);
                g0 = g1;
            }
        }
    } else if (warp >= 4 && warp < 8) {
        // ------------------------------------------------ epilogue
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;  // weight row inside the 128-row block
        const int groups = p.bm >> 2, per = split_groups(p.bm, S);  // groups of four tokens; rank r finishes [r * per, (r + 1) * per)
        // A rank without tokens to finish leaves ex_full alone: with nothing to arrive, its phases would complete at once and
        // run ahead of the warps that wait for them.
        const int mine = max(0, min(per, groups - rank * per));
        const uint32_t ex_addr = g_smem_u32(ex) + (uint32_t)(rank * per * GEMM_BN + row) * 16, bar_addr = g_smem_u32(ex_full);
        float* const scale = reinterpret_cast<float*>(ex + (size_t)S * per * GEMM_BN) + quarter * 64;
        int local = 0, round = 0;
        asm volatile("griddepcontrol.wait;" ::: "memory");  // the row scales; no bounded wait before
        float* sums = p.partial + (size_t)blockIdx.x * SPLIT_MAX_TOKENS * GEMM_BN;
        bool ok = true;
        for (int tile = cluster; tile < tiles && ok && !*abort_flag; tile += clusters, round++) {
            const int nt = tile / p.m_tiles, tok0 = (tile % p.m_tiles) * p.bm;
            const int n = nt * GEMM_BN + row;
            // what this rank finishes of the tile: tokens [first, first + left), at most 64 of them (S > 1); their scales go to
            // the warp's own place, so that it shares nothing with the others (in registers they cost up to 5 %)
            const int first = tok0 + rank * per * 4, left = min(mine * 4, p.m - first);
            if (S > 1) {
#pragma unroll
                for (int j = 0; j < 2; j++) scale[32 * j + lane] = 32 * j + lane < left ? p.row_unscale[first + 32 * j + lane] : 0.f;
                if (threadIdx.x == 128 && mine > 0) g_mbar_expect_tx(ex_full, (uint32_t)(S * mine * GEMM_BN * 16));
                if (round > 0 && !g_mbar_wait(ex_empty, (round - 1) & 1)) { if (lane == 0) fail(); break; }
            } else if (8 * lane < p.bm && tok0 + 8 * lane < p.m) {  // brought into the L1 while the tile is multiplied
                asm volatile("" ::"f"(p.row_unscale[tok0 + 8 * lane]));
            }
            uint32_t to = 0, in = 0;  // rank and place there of the next group of four tokens
            uint32_t to_addr = map_to_rank(ex_addr, 0), to_bar = map_to_rank(bar_addr, 0);
            for (int g0 = kb0; g0 < kb1; local++) {
                const int g1 = min(kb1, g0 + min(FLUSH, kb1 - g0)), buf = local & 1;
                const bool last = g1 == kb1;
                if (!g_mbar_wait(&acc_full[buf], (local >> 1) & 1)) { if (lane == 0) fail(); ok = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * ACCS * p.bm);
                for (int c = 0; c < p.bm; c += 32) {  // 32 columns at a time (also past a BM that is not a multiple of 32)
                    uint32_t r[32];
                    tmem_ld_accs<ACCS>(taddr + (uint32_t)c, p.bm, r);
                    if (PIECES == 2 && g0 > kb0) {  // what earlier groups of the tile came to
                        float4 v[8];
                        load_piece_chunk(sums, v, c, row);
                        add_piece_chunk(r, v);
                    }
                    if (PIECES == 2 && !last) {
                        write_piece_chunk(sums, r, c, row);
                    } else if (S == 1) {
                        store_chunk(p.y, p.ldy, p.col0, p.row_unscale, r, tok0 + c, p.m, n, p.rows);
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const int gr = (c >> 2) + j;
                            if (gr < groups) {
                                st_async_16(to_addr + in * (GEMM_BN * 16), r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3], to_bar);
                                if (++in == (uint32_t)per && gr + 1 < groups) {
                                    in = 0;
                                    to++;
                                    to_addr = map_to_rank(ex_addr, to);
                                    to_bar = map_to_rank(bar_addr, to);
                                }
                            }
                        }
                    }
                }
                tc_fence_before();  // the accumulator has been read: the MMA issuer may overwrite it
                __syncwarp();
                if (lane == 0) g_mbar_arrive(&acc_empty[buf]);
                g0 = g1;
            }
            if (!ok) break;
            if (S > 1) {  // this rank's tokens: the ranks' parts in rank order
                if (mine > 0 && !g_mbar_wait(ex_full, round & 1)) { if (lane == 0) fail(); break; }
                float* yp = p.y + (int64_t)first * p.ldy + p.col0 + n;
#pragma unroll 2
                for (int gi = 0; gi * 4 < left; gi++) {
                    float4 v = ex[(size_t)gi * GEMM_BN + row];
                    for (int src = 1; src < S; src++) {
                        const float4 w = ex[(size_t)(src * per + gi) * GEMM_BN + row];
                        v.x += w.x, v.y += w.y, v.z += w.z, v.w += w.w;
                    }
                    const float4 u = *reinterpret_cast<const float4*>(scale + gi * 4);
                    const float o[4] = {v.x * u.x, v.y * u.y, v.z * u.z, v.w * u.w};
                    if (n < p.rows) {
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            if (gi * 4 + e < left) yp[(int64_t)(gi * 4 + e) * p.ldy] = o[e];
                    }
                }
                __syncwarp();
                if (lane < S) mbar_arrive_cluster(map_to_rank(g_smem_u32(ex_empty), (uint32_t)lane));
            }
        }
    } else {
        // ------------------------------------------------ dequant warps 2, 3, 8..: one 16-row tile each per stage
        const int dq = (warp < 4) ? warp - 2 : warp - 6;  // 16-row tile of the 128 rows
        const int dg = lane >> 2, dq4 = lane & 3;
        uint8_t* const a_mine = stage0 + (dq * 16 + dg) * 128;
        uint32_t a_off[2];  // 16-byte chunks of the swizzled row
#pragma unroll
        for (int j = 0; j < 2; j++) a_off[j] = (uint32_t)((stage_chunk(j, dq4) ^ dg) << 4);
        // One step: convert registers loaded earlier into fp16 rows (still in registers), wait for the stage, store them and
        // hand the stage over.  Converting before the wait keeps the arithmetic off the path between "the MMAs have
        // released the stage" and "the stage is full again".  (Both stages of a unit in one step: 7 - 14 % slower.)
        StageCursor at;
        auto finish_step = [&](const DequantRegs<QT> (&regs)[2], auto sub) {
            const int s = at.s;
            uint4 out[2][2 * PIECES];
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                if constexpr (PIECES == 1) regs[hh].template pair<decltype(sub)::value>(out[hh][0], out[hh][1]);
                else regs[hh].template pair2<decltype(sub)::value>(out[hh][0], out[hh][1], out[hh][2], out[hh][3]);
            }
            if (!g_mbar_wait(&s_empty[s], at.phase ^ 1)) {
                if (lane == 0) fail();
                return false;
            }
            uint8_t* a_stage = a_mine + (size_t)s * stage_bytes;
#pragma unroll
            for (int hh = 0; hh < 2; hh++)
#pragma unroll
                for (int j = 0; j < 2 * PIECES; j++)
                    *reinterpret_cast<uint4*>(a_stage + (j >> 1) * (GEMM_BN * 128) + hh * 1024 + a_off[j & 1]) = out[hh][j];
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic writes -> visible to the tensor core
            __syncwarp();
            if (lane == 0) g_mbar_arrive(&a_full[s]);
            if (at.advance(stages)) asm volatile("griddepcontrol.wait;" ::: "memory");  // no bounded wait under earlier kernels
            return true;
        };
        // DEPTH register sets in turn (128 k each): the loads of the following DEPTH - 1 units are in flight while one is
        // converted, across the ends of tiles.
        constexpr int DEPTH = 3;
        DequantRegs<QT> r[DEPTH][2];
        int ltile = cluster, lkb = kb0;
        const uint8_t* lrow = nullptr;
        auto set_row = [&]() { lrow = p.tiles + ((int64_t)(ltile / p.m_tiles) * (GEMM_BN / 16) + dq) * p.kt_w * (int64_t)Tile<QT>::BYTES; };
        set_row();
        auto load_next = [&](DequantRegs<QT> (&regs)[2]) {
            if (ltile >= tiles) return;
            const uint8_t* t = lrow + (size_t)(lkb / KBW) * Tile<QT>::BYTES;
            regs[0].load(t, lkb % KBW, lane, 0);
            regs[1].load(t, lkb % KBW, lane, 1);
            if (++lkb == kb1) {
                lkb = kb0;
                ltile += clusters;
                if (ltile < tiles) set_row();
            }
        };
#pragma unroll
        for (int d = 0; d < DEPTH - 1; d++) load_next(r[d]);
        const int units = my_tiles * (kb1 - kb0);
        bool ok = true;
        for (int u = 0; u < units && ok && !*abort_flag; u += DEPTH) {
#pragma unroll
            for (int d = 0; d < DEPTH; d++) {
                if (u + d >= units) break;
                load_next(r[(d + DEPTH - 1) % DEPTH]);
                ok = finish_step(r[d], std::integral_constant<int, 0>{});
                if (ok) ok = finish_step(r[d], std::integral_constant<int, 1>{});
                if (!ok) break;
            }
        }
    }

    // ------------------------------------------------ teardown: no rank leaves while another may still store into its exchange
    // buffer or arrive on its barriers; TMEM is freed on every path
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (S > 1) cluster_sync();
    if (warp == 1) {
        if (*abort_flag) drain_after_abort();  // operands, MMAs and other ranks' parts that nobody waited for
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace wf
