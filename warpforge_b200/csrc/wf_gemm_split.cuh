// GEMM for few tokens, few tiles, or fp32 tokens: y[m, rows] = x[m, K] . W[rows, K]^T, one tile of 128 weight rows x BM
// (at most 128) tokens per cluster of S CTAs, which split its K.
//
// What bounds these calls is latency: a [4096 x 4096] weight has 32 tiles for 148 SMs, so K has to be split, and then the
// time goes into putting the parts together.  As stream-K shares whose pieces travel through global memory to the one
// CTA that owns the tile (write, fence, flag, poll, read up to four pieces) that took 8 - 14 us of 16 - 25 us.  Here every
// CTA sends each token of its accumulator to the rank that finishes it, by asynchronous stores straight into that CTA's
// shared memory which count themselves on its barrier; each rank adds its tokens' S parts in rank order (deterministic)
// and stores them.  No CTA has more to finish than another, and nothing goes through L2.
// Measured, 64 tokens, Q4_0 [4096 x 4096]: 9.3 us a call (16.8 as stream-K shares); 33 tokens of Q4_1 [1000 x 1024]: 6.2 us.
//
// A lies in TMEM, not in shared memory: the weights' fragment order is that of a 16x256b store, so a dequantizing lane's registers go
// there as they are, without addresses, bank conflicts or a proxy fence; the tensor core keeps its pace at any token count
// (tc_mma_span), and shared memory is left to the activations, which for fp32 tokens bounded the kernel (416 KB per 128 k and
// 96 tokens, 3250 cycles, where the products take 1900).  Two sets of eight dequantizing warps instead of one.  us a call,
// with A in shared memory and eight warps / so: Q4_0 [16384 x 2048] 128 tokens 16.4 / 13.1, Q8_0 [4096 x 11008] 96 tokens 28.7 /
// 25.0, Q4_1 [11008 x 4096] 96 fp32 tokens 44.4 / 39.0.
//
// Warp roles (704 threads):
//   warp 0      TMA producer: activation spans [BM tokens x 64 k], 128-byte swizzle
//   warp 1      MMA issuer; owns TMEM
//   warps 4-7   epilogue (TMEM lane quarter = warp % 4): accumulator -> the ranks' exchange buffers -> y
//   warps 2,3,8-21  dequantization: quantized tiles from global memory -> fp16 rows of A in TMEM, in two sets of eight warps
// TMEM: the accumulators (double buffered, so a tile is put together while the next one is computed), behind them the ring of
// A stages.
// Stages.  bf16 tokens: 128 k of weights and activations together, four of them, so that the MMA warp has one barrier to wait for and
// one commit per 128 k.  With stages of 64 k and barriers of their own for weights and activations the kernel took 664 cycles
// per 128 k even with dequantization left out, whatever the number of tokens: the MMA warp's waits (75 - 90 cycles each,
// though nothing had to be waited for) and commits, between the instructions of the five warps that share its scheduler (33 tokens,
// Q4_0 [16384 x 2048] 11.8 -> 9.6 us a call, [4096 x 4096] 9.3 -> 8.1, Q5_0 [5003 x 2784] 77 tokens 11.7 -> 10.8).  fp32
// tokens, whose MMAs take 960 cycles per 64 k: 64 k, weights and activations apart.
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

inline __host__ __device__ int split_stage_bytes(int planes, int bm) { return (planes == 1 ? 2 : planes) * bm * 128; }  // of activations
// Stages of weights that TMEM has room for: 4 of 128 k, or 2 - 6 of 64 k for fp32 tokens, an even number.
inline __host__ __device__ int split_a_stages(int pieces, int bm) { return pieces == 1 ? 4 : min((512 - 4 * bm) / 64, SPLIT_MAX_STAGES) & ~1; }
// exchange buffer: [S][groups of four tokens a rank finishes][128 rows] float4, where there are several ranks | token scales [4
// epilogue warps][128] | fp32 tokens: sums of the groups of units so far, [groups of four tokens][128 rows] float4
inline __host__ __device__ int split_groups(int bm, int ranks) { return (bm / 4 + ranks - 1) / ranks; }
inline __host__ __device__ int split_exchange_bytes(int pieces, int bm, int ranks) {
    return (ranks == 1 ? 0 : ranks * split_groups(bm, ranks) * GEMM_BN * 16) + 4 * SPLIT_MAX_TOKENS * 4 + (pieces == 1 ? 0 : bm * GEMM_BN * 4);
}

// smem: [0, 1024) barriers, tmem slot | stages of activations, 1024-byte aligned | exchange buffer
// Registers: 80 a thread, what the hardware has for 24 warps (it counts in fours); 22 are launched.
template <int QT, int PIECES, int PLANES>
__global__ void __launch_bounds__(768, 1) gemm_split_kernel(const GemmParams p, const __grid_constant__ CUtensorMap xmap) {
    constexpr int ACCS = PIECES;
    constexpr int FLUSH = PIECES == 1 ? 1 << 30 : SPLIT_FLUSH;
    constexpr int KBW = Tile<QT>::K / GEMM_BK;  // units per weight k-tile
    constexpr uint32_t A_COLS = 64;             // TMEM columns of an A stage: two spans of 64 k, or both pieces of one
    constexpr bool JOINT = PIECES == 1;         // weights and activations share stages and barriers (b_full, b_empty)
    constexpr int SPANS = JOINT ? 2 : 1;        // of 64 k per stage
    // The two sets of dequantization warps take units by turns (bf16), or a stage each of every unit (fp32: there may be no more than two
    // stages, and a set that came back to one only after the other set's turn could not tell by the barrier's parity whether that
    // turn is over).
    constexpr int TURN = PIECES == 1 ? GEMM_SETS : 1;
    using Regs = std::conditional_t<PIECES == 1, DequantRegs<QT>, DequantHalf<QT>>;
    constexpr int DEPTH = 2;  // units a dequantization warp holds: one is converted while the other loads
    constexpr int COLS = PIECES == 1 ? 32 : 16; // that an epilogue warp takes at a time
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t* b_full = reinterpret_cast<uint64_t*>(smem);        // [8] activations landed (JOINT: and weights dequantized)
    uint64_t* b_empty = b_full + SPLIT_MAX_STAGES;               // [8] read by the MMAs
    uint64_t* a_full = JOINT ? b_full : b_empty + SPLIT_MAX_STAGES;    // [8] weights dequantized
    uint64_t* a_empty = JOINT ? b_empty : a_full + SPLIT_MAX_STAGES;   // [8] read by the MMAs
    uint64_t* acc_full = b_full + 4 * SPLIT_MAX_STAGES;          // [2]
    uint64_t* acc_empty = acc_full + 2;                          // [2]
    uint64_t* ex_full = acc_empty + 2;                           // the parts of this rank's tokens have arrived
    uint64_t* ex_empty = ex_full + 1;                            // every rank has read its exchange buffer
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ex_empty + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t span_bytes = (uint32_t)p.bm * 128;  // 64 k of bm tokens
    const uint32_t stage_bytes = (JOINT ? 2 : PLANES) * span_bytes;
    const int stages = p.stages, a_stages = JOINT ? stages : split_a_stages(PIECES, p.bm), S = p.ranks;
    uint8_t* stage0 = smem + 1024;
    float4* ex = reinterpret_cast<float4*>(stage0 + (size_t)stages * stage_bytes);
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = (int)cluster_rank(), cluster = (int)cluster_id(), clusters = (int)cluster_count();
    const int tiles = p.n_tiles * p.m_tiles;
    const int kb0 = rank * p.unit_q + min(rank, p.unit_r), kb1 = kb0 + p.unit_q + (rank < p.unit_r ? 1 : 0);  // this rank's units of every tile
    const int my_tiles = p.tile_q + (cluster < p.tile_r ? 1 : 0);

    // Dequantization warps: their first weights, which depend on nothing, are requested before all set-up.  TMEM lanes 32 (warp % 4) ..
    // + 31 are all that a warp reaches: of the four of a quarter, two take the units of even number, two those of odd number, one
    // each of the quarter's two 16-row tiles.
    const bool dequant = warp >= 8 || warp == 2 || warp == 3;
    const int nth = warp < 4 ? 0 : (warp - 8 - (warp & 3)) / 4 + ((warp & 3) >> 1);  // of its quarter
    const int set = nth >> 1, dq = 2 * (warp & 3) + (nth & 1);                       // dq: 16-row tile of the 128 rows
    Regs r[DEPTH][2];
    const int units = my_tiles * (kb1 - kb0);
    const int unit0 = PIECES == 1 ? set : 0;
    int ltile = cluster, lkb = kb0, lunit = unit0;
    const uint8_t* lrow = nullptr;
    auto row_of = [&](int tile) { return p.m_tiles == 1 ? tile : tile / p.m_tiles; };
    auto set_row = [&]() { lrow = p.tiles + ((int64_t)row_of(ltile) * (GEMM_BN / 16) + dq) * p.kt_w * (int64_t)Tile<QT>::BYTES; };
    auto skip = [&](int n) {
        lkb += n;
        if (lkb < kb1) return;
        for (; lkb >= kb1; lkb -= kb1 - kb0) ltile += clusters;
        set_row();  // an address only, behind the last tile
    };
    auto load_next = [&](Regs (&regs)[2]) {
        if (lunit >= units) return;
        const uint8_t* t = lrow + (size_t)(lkb / KBW) * Tile<QT>::BYTES;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if constexpr (PIECES == 1) regs[h].load(t, lkb % KBW, lane, h);
            else regs[h].load(t, lkb % KBW, set, lane, h);
        }
        lunit += TURN;
        skip(TURN);
    };
    if (dequant) {
        set_row();
        skip(unit0);
#pragma unroll
        for (int d = 0; d < DEPTH; d++) load_next(r[d]);
    }

    // Everything up to the first MMA runs once and is fetched cold, so it is kept short: a barrier per lane, no divisions
    // (1.9 -> 1.4 us from the CTA's start to the end of the set-up).
    if (warp == 0) {
        if (lane == 0) {
            prefetch_tensormap(&xmap);
            *abort_flag = 0;
        }
        g_mbar_init(b_full + lane, lane >> 3 == 2 ? GEMM_DEQUANT_WARPS : JOINT && lane < 8 ? GEMM_DEQUANT_WARPS + 1 : 1);  // the rings
        // acc_full, acc_empty (the four epilogue warps), ex_full, ex_empty
        if (lane < 6) g_mbar_init(acc_full + lane, lane == 2 || lane == 3 ? 4 : lane == 5 ? 4 * S : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    if (S > 1) cluster_sync();  // the other ranks' barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot, a_tmem = tmem_base + (uint32_t)(2 * ACCS * p.bm);

    auto fail = [&]() {
        report_status(p.status, STATUS_GEMM_PIPE_TIMEOUT);
        *abort_flag = 1;
    };

    if (warp == 0) {
        // ------------------------------------------------ TMA producer (activations)
        if (lane == 0) {
            // The next call's conversion waits on SMs that are idle meanwhile, and the next GEMM takes each SM as it becomes free (a call of
            // [5003 x 2784], 77 tokens, Q4_0: 12.7 -> 11.6 us; 64 tokens of [4096 x 4096], 12.7 -> 11.3).  Placed when the CTA
            // begins its last tile: a conversion that waits longer delays clusters of several tiles ([11008 x 4096], 128
            // tokens, two tiles each: 27.6 us without, 28.9 placed at the start, 27.8 here).  p.early: where it pays (gemm_launch).
            auto last_tile = [&](int tile) {
                if (p.early && tile + clusters >= tiles) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            };
            last_tile(cluster);
            asm volatile("griddepcontrol.wait;" ::: "memory");  // the fp16 activations
            StageCursor at;
            for (int tile = cluster; tile < tiles && !*abort_flag; tile += clusters) {
                const int tok0 = (tile % p.m_tiles) * p.bm;
                if (tile != cluster) last_tile(tile);
                for (int st = 2 * kb0; st < 2 * kb1; st += SPANS, at.advance(stages)) {
                    const int s = at.s;
                    if (!g_mbar_wait(&b_empty[s], at.phase ^ 1)) { fail(); break; }
                    uint8_t* b_stage = stage0 + (size_t)s * stage_bytes;
                    g_mbar_expect_tx(&b_full[s], stage_bytes);
                    if (JOINT) {
                        tma_load_2d(b_stage, &xmap, st * 64, tok0, &b_full[s]);
                        tma_load_2d(b_stage + span_bytes, &xmap, st * 64 + 64, tok0, &b_full[s]);
                    } else {
#pragma unroll
                        for (int pl = 0; pl < PLANES; pl++) tma_load_2d(b_stage + pl * span_bytes, &xmap, st * 64, pl * p.m + tok0, &b_full[s]);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        asm volatile("griddepcontrol.wait;" ::: "memory");  // no bounded wait starts while earlier kernels of the stream run
        const uint32_t issue = elect_one();
        const uint64_t b_desc0 = smem_desc_sw128(g_smem_u32(stage0));
        const uint64_t span = span_bytes >> 4;
        StageCursor at, a_at;
        int local = 0;
        bool ok = true;
        for (int tile = cluster; tile < tiles && ok && !*abort_flag; tile += clusters) {
            for (int g0 = kb0; g0 < kb1 && ok; local++) {  // groups of units that share an accumulator
                const int g1 = min(kb1, g0 + min(FLUSH, kb1 - g0)), buf = local & 1;
                if (local >= 2 && !g_mbar_wait(&acc_empty[buf], ((local >> 1) - 1) & 1)) { fail(); ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * ACCS * p.bm), e_tmem = d_tmem + (uint32_t)p.bm;
                for (int st = 2 * g0; st < 2 * g1; st += SPANS) {
                    const int s = at.s;
                    if (!g_mbar_wait(&b_full[s], at.phase) || (!JOINT && !g_mbar_wait(&a_full[a_at.s], a_at.phase))) { fail(); ok = false; break; }
                    tc_fence_after();
                    const uint64_t bd = b_desc0 + (uint64_t)((uint32_t)s * stage_bytes >> 4);
                    const uint32_t hi = a_tmem + (uint32_t)(JOINT ? s : a_at.s) * A_COLS, lo = hi + 32;
                    const uint32_t acc = (uint32_t)(st - 2 * g0);
                    tc_mma_span<1>(d_tmem, hi, bd, p.idesc, acc, issue);
                    if (JOINT) {
                        tc_mma_span<1>(d_tmem, lo, bd + span, p.idesc, 1u, issue);
                    } else {
                        tc_mma_span<1>(e_tmem, lo, bd, p.idesc, acc, issue);
                        tc_mma_span<1>(e_tmem, hi, bd + span, p.idesc, 1u, issue);
                        tc_mma_span<1>(e_tmem, lo, bd + span, p.idesc, 1u, issue);
                        tc_mma_span<1>(e_tmem, hi, bd + 2 * span, p.idesc, 1u, issue);
                    }
                    if (issue) {  // frees the stages when these MMAs have read them
                        if (!JOINT) tc_commit(&a_empty[a_at.s]);
                        tc_commit(&b_empty[s]);
                    }
                    at.advance(stages);
                    if (!JOINT) a_at.advance(a_stages);
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
        // a copy for each warp, so that it shares nothing with the others (in registers they cost up to 5 %)
        float* const scale = reinterpret_cast<float*>(ex + (S == 1 ? 0 : (size_t)S * per * GEMM_BN)) + quarter * SPLIT_MAX_TOKENS;
        int local = 0, round = 0;
        // (in global memory each 16 tokens waited for the L2 behind the last MMA: 38 shapes 0.98 x, Q8_0 [3000 x 6016] 96 tokens 23.7 -> 22.4 us)
        float4* const sums = ex + (S == 1 ? 0 : (size_t)S * per * GEMM_BN) + 4 * SPLIT_MAX_TOKENS / 4 + row;
        asm volatile("griddepcontrol.wait;" ::: "memory");  // the row scales; no bounded wait before
        bool ok = true;
        for (int tile = cluster; tile < tiles && ok && !*abort_flag; tile += clusters, round++) {
            const int nt = row_of(tile), tok0 = (tile - nt * p.m_tiles) * p.bm;
            const int n = nt * GEMM_BN + row;
            // what this rank finishes of the tile: tokens [first, first + left), all of them where it is the only one
            const int first = tok0 + rank * per * 4, left = min(mine * 4, p.m - first);
            __syncwarp();
            for (int j = lane; j < mine * 4; j += 32) scale[j] = j < left ? p.row_unscale[first + j] : 0.f;
            __syncwarp();
            if (S > 1) {
                if (threadIdx.x == 128 && mine > 0) g_mbar_expect_tx(ex_full, (uint32_t)(S * mine * GEMM_BN * 16));
                if (round > 0 && !g_mbar_wait(ex_empty, (round - 1) & 1)) { if (lane == 0) fail(); break; }
            }
            uint32_t to = 0, in = 0;  // rank and place there of the next group of four tokens
            uint32_t to_addr = map_to_rank(ex_addr, 0), to_bar = map_to_rank(bar_addr, 0);
            for (int g0 = kb0; g0 < kb1; local++) {
                const int g1 = min(kb1, g0 + min(FLUSH, kb1 - g0)), buf = local & 1;
                const bool last = g1 == kb1;
                if (!g_mbar_wait(&acc_full[buf], (local >> 1) & 1)) { if (lane == 0) fail(); ok = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * ACCS * p.bm);
                for (int c = 0; c < p.bm; c += COLS) {  // 32 columns at a time (also past a BM that is not a multiple of 32), or 16
                    uint32_t v[COLS];
                    tmem_ld_accs(taddr + (uint32_t)c, p.bm, v);
                    if (PIECES == 2 && g0 > kb0) {  // what earlier groups of the tile came to
                        float4 e[COLS / 4];
#pragma unroll
                        for (int j = 0; j < COLS / 4; j++) e[j] = sums[((c >> 2) + j) * GEMM_BN];
                        add_piece_chunk(v, e);
                    }
                    if (PIECES == 2 && !last) {
#pragma unroll
                        for (int j = 0; j < COLS / 4; j++)
                            sums[((c >> 2) + j) * GEMM_BN] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
                    } else if (S == 1) {
                        store_chunk(p.y, p.ldy, p.col0, scale - tok0, v, tok0 + c, p.m, n, p.rows);
                    } else {
#pragma unroll
                        for (int j = 0; j < COLS / 4; j++) {
                            const int gr = (c >> 2) + j;
                            if (gr < groups) {
                                st_async_16(to_addr + in * (GEMM_BN * 16), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3], to_bar);
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
                constexpr int AT_ONCE = 4;  // groups whose parts are read together (one by one: 0.25 us each)
                for (int gi = 0; gi * 4 < left; gi += AT_ONCE) {
                    float4 v[AT_ONCE];
                    const float4* const mine0 = ex + (size_t)gi * GEMM_BN + row;
                    const int last = min(AT_ONCE, mine - gi) - 1;
#pragma unroll
                    for (int u = 0; u < AT_ONCE; u++) v[u] = mine0[min(u, last) * GEMM_BN];
                    for (int src = 1; src < S; src++) {
                        float4 w[AT_ONCE];
#pragma unroll
                        for (int u = 0; u < AT_ONCE; u++) w[u] = mine0[(src * per + min(u, last)) * GEMM_BN];
#pragma unroll
                        for (int u = 0; u < AT_ONCE; u++) v[u].x += w[u].x, v[u].y += w[u].y, v[u].z += w[u].z, v[u].w += w[u].w;
                    }
                    if (n < p.rows) {
#pragma unroll
                        for (int u = 0; u < AT_ONCE; u++) {
                            const float4 by = *reinterpret_cast<const float4*>(scale + (gi + min(u, last)) * 4);
                            const float o[4] = {v[u].x * by.x, v[u].y * by.y, v[u].z * by.z, v[u].w * by.w};
#pragma unroll
                            for (int e = 0; e < 4; e++)
                                if ((gi + u) * 4 + e < left) yp[(int64_t)((gi + u) * 4 + e) * p.ldy] = o[e];
                        }
                    }
                }
                __syncwarp();
                if (tile + clusters < tiles && lane < S) mbar_arrive_cluster(map_to_rank(g_smem_u32(ex_empty), (uint32_t)lane));
            }
        }
    } else {
        // ------------------------------------------------ dequant warps
        // One step: convert registers loaded earlier (still in registers; the first of two spans), wait for the stage, store it and hand
        // it over.  Converting before the wait keeps arithmetic off the path between "the MMAs have released the stage" and "the
        // stage is full again".
        const uint32_t a_mine = a_tmem + ((uint32_t)(dq * 16) << 16);
        StageCursor at;
        bool lapped = false;  // from the second lap on a wait is bounded by what earlier kernels let this one do
        auto advance = [&]() { lapped |= at.advance(a_stages); };
        auto convert = [&](const Regs (&regs)[2], auto sub, uint4 (&out)[2][2 * PIECES]) {
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                if constexpr (JOINT) regs[hh].template pair<decltype(sub)::value>(out[hh][0], out[hh][1]);
                else regs[hh].pair2(out[hh][0], out[hh][1], out[hh][2], out[hh][3]);
            }
        };
        auto finish_step = [&](const Regs (&regs)[2]) {
            uint4 out[2][2 * PIECES];
            convert(regs, std::integral_constant<int, 0>{}, out);
            if (lapped) {
                asm volatile("griddepcontrol.wait;" ::: "memory");
                lapped = false;
            }
            if (!g_mbar_wait(&a_empty[at.s], at.phase ^ 1)) {
                if (lane == 0) fail();
                return false;
            }
            tc_fence_after();
            const uint32_t to = a_mine + (uint32_t)at.s * A_COLS;
            tmem_st_span(to, out[0][0], out[0][1], out[1][0], out[1][1]);
            if constexpr (JOINT) {
                convert(regs, std::integral_constant<int, 1>{}, out);
                tmem_st_span(to + 32, out[0][0], out[0][1], out[1][0], out[1][1]);
            } else {
                tmem_st_span(to + 32, out[0][2], out[0][3], out[1][2], out[1][3]);
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) g_mbar_arrive(&a_full[at.s]);
            advance();
            return true;
        };
        if (set > 0) advance();
        bool ok = true;
        for (int u = unit0; u < units && ok && !*abort_flag; u += TURN * DEPTH) {
#pragma unroll
            for (int d = 0; d < DEPTH; d++) {
                if (u + d * TURN >= units) break;
                ok = finish_step(r[d]);
                if (!ok) break;
                load_next(r[d]);
                advance();  // over the other set's stage
            }
        }
    }

    // ------------------------------------------------ teardown: no rank leaves while another may still store into its exchange
    // buffer or arrive on its barriers (what the others sent it has landed: relaxed, so that nobody waits for its stores of y); TMEM is
    // freed on every path.  The ranks leave together: let go one by one, they leave SMs in which the next call's clusters do
    // not find places side by side.
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (S > 1) {
        asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
    if (warp == 1) {
        if (*abort_flag) drain_after_abort();  // operands, MMAs and other ranks' parts that nobody waited for
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace wf
