// Decode GEMV, y[m, rows] = x[m, K] . W[rows, K]^T with W in the tiled quantized layout of wf_layout.cuh: the launch side
// and the one-token kernel.  HBM-bound: every weight byte is read exactly once, from global memory straight into
// the registers of the warp that multiplies it.
//   * one token, bf16 or fp32: gemv1_kernel below (integer MMAs on exact base-256 digits of the activations,
//     wf_gemv_stream.cuh);
//   * 2 .. 32 activation columns (bf16 tokens, or two and more fp32 tokens as three exact bf16 columns each): gemvn_kernel
//     (bf16 MMAs, k-sliced units, wf_gemv_multi.cuh); more tokens than that go through it in passes, or to the
//     tensor-core GEMM (wf_gemm.cu) where the caller routes them there.
//
// Replaces the fp32 batch_matmul_f32 launch of
// warpforge-backend-nvidia/src/main/java/io/surfworks/warpforge/backend/nvidia/ops/DotGeneralKernel.java:263-281
// (PTX at .../nvidia/cuda/CudaKernels.java:4423-4585) for quantized right-hand sides.
#include "wf_gemv_multi.cuh"

namespace wf {

// ---------------------------------------------------------------- one token
// Between the wait for the grid that writes x and the first tile lies a chain that nothing overlaps: request x, turn it into
// digits, find the warp's run.  Four warps per scheduler hide little of it, so what does not depend on x is done before
// the wait, and each input kind has its own kernel, whose staging is no call behind a switch (rms_norm, which reads the row twice, still
// calls its two passes): behind the wait it took 1000 cycles
// until the first element was requested, and 900 - 1700 from the staged row to the first tile.  With that, half the
// instructions per digit, digits without bank conflicts and the cut row-tiles added by both halves of a warp, a 32-layer step of
// the 7B shape went from 1097 to 1007 us, [4096 x 11008] from 7.8 to 7.2 (Q4_0).
// What the staging needs to know, in registers before the wait:
struct StageArgs {
    const void* x;
    const float* aux;
    int k, kp;
};
template <int KIND> __device__ __forceinline__ StageArgs pinned(StageArgs a) {
    if (KIND != XK_RMSNORM_F32) asm volatile("" : "+l"(a.x), "+r"(a.k), "+r"(a.kp));
    if (KIND == XK_SWIGLU_F32) asm volatile("" : "+l"(a.aux));
    return a;
}
template <class Stage> __device__ __forceinline__ void stage_row(const StageArgs& a, uint8_t* xd, uint8_t* recs, float inv = 1.f) {
    const int padded = ((a.kp >> 3) + 31) & ~31;
#pragma unroll 1
    for (int c0 = threadIdx.x; c0 < padded; c0 += GEMV_CONSUMERS * Stage::U) {  // warp-uniform trip counts
        Stage s;
        s.fetch(a.x, a.aux, a.k, c0, GEMV_CONSUMERS);
        s.put(xd, recs, a.kp, c0, GEMV_CONSUMERS, a.aux != nullptr, inv);
    }
}

// Integer MMAs on exact base-256 digits of the activations, every warp streaming its own run of tiles from
// global memory into registers (wf_gemv_stream.cuh).  512 threads, all of them consumers.
template <int QT, int KIND>
__global__ void __launch_bounds__(GEMV_CONSUMERS, 1) gemv1_kernel(const GemvParams p) {
    using T = Tile<QT>;
    using R = TileRegs<QT>;
    extern __shared__ __align__(128) uint8_t smem[];
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem);
    WsPiece* pieces = reinterpret_cast<WsPiece*>(smem + WS_CTRL_BYTES);
    uint8_t* recs = smem + WS_CTRL_BYTES + WS_PIECE_BYTES;
    const int kp = p.kt * T::K;
    uint8_t* xd = recs + (size_t)(kp >> 5) * 32;

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int bx = blockIdx.x;
    int t0, t1;
    ws_cta_share(bx, (int)gridDim.x, p.chunk_q, p.chunk_r, p.aligned, p.kt, t0, t1);
    auto stamp = [&](int i) {
        if (p.timing != nullptr && threadIdx.x == 0) {
            unsigned long long tm;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tm));
            p.timing[(size_t)blockIdx.x * 8 + i] = tm;
        }
    };
    // Programmatic stream serialization: this grid may start while the previous one drains, and what follows
    // griddepcontrol.wait sees all that it wrote.  The weights depend on nothing, so every warp requests the first tiles
    // of its run before that.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const WsShare share{p.tiles, t0, t1, p.kt, 0, {0, 0}};
    auto share_of = [&](int) { return share; };
    constexpr int DEPTH = WsGeom<QT, false>::DEPTH;
    R slots[DEPTH];
    WsCursor cur;
    WsNext next = ws_prime<QT, DEPTH, true>(slots, cur, share_of, 1, warp, lane);
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        ws_bars_init(smem);
    }
    ws_clear_digits(xd, kp, GEMV_CONSUMERS);
    const WsRun run = ws_open(share, warp);
    __syncthreads();
    const WsBars bar = ws_bars(smem);

    using Stage = StageQ8<R::BETA_INT, KIND>;
    const StageArgs args = pinned<KIND>(StageArgs{p.x, nullptr, p.k, kp});
    asm volatile("griddepcontrol.wait;" ::: "memory");
    stamp(0);
    stage_row<Stage>(args, xd, recs);
    __syncthreads();
    stamp(1);
    auto emit_row = [&](int n, float v) {
        if (n < p.rows) p.y[p.col0 + n] = v;
    };
    stamp(2);
    uint32_t seq = 0;
    ws_consume<QT, DEPTH, true>(share, run, p.chunk_q, p.chunk_r, warp, lane, slots, next, cur, bar, pieces, seq, smem_u32(xd), smem_u32(recs),
                   smem_u32(recs) + (uint32_t)(kp >> 5) * 16, p.scratch, p.status, smem_u32(const_cast<int*>(abort_flag)), share_of, 1,
                   emit_row);
    stamp(4);
    if (*abort_flag) {  // a wait ran out somewhere in this CTA
        if (lane == 0) report_status(p.status, STATUS_GEMV_FIXUP_TIMEOUT);
    }
    stamp(5);
}

// The same for a program: several weights, the fp32 operations before the projection in its staging, a residual in its store.
// Its own kernel, because what a plain call does not need it would fetch cold and jump over: 2 % of a 4 - 8 us call.
template <int QT, int KIND>
__global__ void __launch_bounds__(GEMV_CONSUMERS, 1) gemv1_group_kernel(const Gemv1GroupParams p) {
    using T = Tile<QT>;
    using R = TileRegs<QT>;
    extern __shared__ __align__(128) uint8_t smem[];
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem);
    WsPiece* pieces = reinterpret_cast<WsPiece*>(smem + WS_CTRL_BYTES);
    uint8_t* recs = smem + WS_CTRL_BYTES + WS_PIECE_BYTES;
    const int kp = p.kt * T::K;
    uint8_t* xd = recs + (size_t)(kp >> 5) * 32;

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int bx = blockIdx.x;
    int t0, t1;
    ws_cta_share(bx, (int)gridDim.x, p.chunk_q, p.chunk_r, p.aligned, p.kt, t0, t1);
    // start, waited, staged, done
    auto stamp = [&](int i) {
        if (p.timing != nullptr && threadIdx.x == 0) {
            unsigned long long tm;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tm));
            if (p.timing_at + i < 64) p.timing[(size_t)bx * 64 + p.timing_at + i] = tm;
        }
    };
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    stamp(0);
    auto share_of = [&](int o) {  // this CTA's part of weight o
        const int begin = p.op[o].rt_begin * p.kt, end = p.op[o].rt_end * p.kt;
        const int a = max(t0, begin), b = min(t1, end);
        return WsShare{p.op[o].tiles, a < b ? a - begin : 0, a < b ? b - begin : 0, p.kt, 0, {0, 0}};
    };
    constexpr int DEPTH = WsGeom<QT, true>::DEPTH;
    R slots[DEPTH];
    WsCursor cur;
    WsNext next = ws_prime<QT, DEPTH, true>(slots, cur, share_of, p.n_ops, warp, lane);
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        mbar_init(smem_u32(smem + 16), 1);
        ws_bars_init(smem);
    }
    ws_clear_digits(xd, kp, GEMV_CONSUMERS);
    // the first weight this CTA has tiles of, and the warp's run of them
    int o = 0;
    WsShare share = share_of(0);
    while (share.t0 == share.t1 && o + 1 < p.n_ops) share = share_of(++o);
    WsRun run = ws_open(share, warp);
    float* y = p.op[o].y;
    const float* residual = p.op[o].residual;
    int rows = p.op[o].rows;
    __syncthreads();
    const WsBars bar = ws_bars(smem);
    const StageArgs args = pinned<KIND>(StageArgs{p.x, p.aux, p.k, kp});
    asm volatile("" : "+l"(y), "+l"(residual), "+r"(rows));

    asm volatile("griddepcontrol.wait;" ::: "memory");
    stamp(1);
    if constexpr (KIND != XK_RMSNORM_F32) {
        stage_row<StageQ8<R::BETA_INT, KIND>>(args, xd, recs);
    } else if (p.x_bytes > 0) {  // two passes over x: from shared memory
        uint8_t* const xs = xd + (size_t)kp * 8;
        const float* const gamma = p.aux != nullptr ? reinterpret_cast<const float*>(xs + p.x_bytes) : nullptr;
        const uint32_t bar_x = smem_u32(smem + 16);
        if (threadIdx.x == 0) {
            mbar_expect_tx(bar_x, (uint32_t)(p.x_bytes * (gamma ? 2 : 1)));
            bulk_load(smem_u32(xs), p.x, (uint32_t)p.x_bytes, bar_x);
            if (gamma) bulk_load(smem_u32(gamma), p.aux, (uint32_t)p.x_bytes, bar_x);
        }
        mbar_wait_or_abort(bar_x, 0, smem_u32(const_cast<int*>(abort_flag)));
        const float inv = cta_rms_inv<true>(reinterpret_cast<const float*>(xs), p.k, p.eps, reinterpret_cast<float*>(smem + 192), GEMV_CONSUMERS);
        stage_x_q8<R::BETA_INT, XK_RMSNORM_F32, true>(xs, p.k, xd, recs, kp, GEMV_CONSUMERS, gamma, inv);
    } else {
        const float inv = cta_rms_inv(static_cast<const float*>(p.x), p.k, p.eps, reinterpret_cast<float*>(smem + 192), GEMV_CONSUMERS);
        stage_x_q8<R::BETA_INT, XK_RMSNORM_F32>(p.x, p.k, xd, recs, kp, GEMV_CONSUMERS, p.aux, inv);
    }
    __syncthreads();
    stamp(2);
    uint32_t seq = 0;
    while (true) {
        auto emit_row = [&](int n, float v) {
            if (n < rows) {
                if (residual != nullptr) v += __ldcg(residual + n);
                y[n] = v;
            }
        };
        ws_consume<QT, DEPTH, true>(share, run, p.chunk_q, p.chunk_r, warp, lane, slots, next, cur, bar, pieces, seq, smem_u32(xd), smem_u32(recs),
                       smem_u32(recs) + (uint32_t)(kp >> 5) * 16, p.scratch, p.status, smem_u32(const_cast<int*>(abort_flag)), share_of,
                       p.n_ops, emit_row);
        do {  // the next one, the same for the whole CTA
            if (++o >= p.n_ops) break;
            share = share_of(o);
        } while (share.t0 == share.t1);
        if (o >= p.n_ops) break;
        run = ws_open(share, warp);
        y = p.op[o].y;
        residual = p.op[o].residual;
        rows = p.op[o].rows;
    }
    // silu(gate) * up by the CTA that has stored both: in the staging of the projection that reads it every CTA would read all
    // of gate and up and take all sigmoids (11008 rows: 6.0 us of staging instead of 2.3)
    if (p.act != nullptr) {
        __syncthreads();
        const int row1 = min(t1 / p.kt * 16, p.op[0].rows);
        for (int n = t0 / p.kt * 16 + threadIdx.x; n < row1; n += GEMV_CONSUMERS) {
            const float f = p.op[0].y[n], sig = 1.0f / (1.0f + expf(-f));
            p.act[n] = (f * sig) * p.op[1].y[n];
        }
    }
    stamp(3);
    if (*abort_flag) {  // a wait ran out somewhere in this CTA
        if (lane == 0) report_status(p.status, STATUS_GEMV_FIXUP_TIMEOUT);
        drain_after_abort();  // the activations' copies
    }
}

// ---------------------------------------------------------------- host side
constexpr size_t GEMV_SMEM_LIMIT = 227 * 1024;

// Without a device to ask: a GPC's SMs are seldom a multiple of a cluster, so about a tenth of the SMs stay out of
// clusters of three and more.
static void gemvn_clusters_estimate(int sm_count, int* clusters) {
    for (int n = 1; n <= GEMVN_MAX_CLUSTER; n++) clusters[n] = n <= 2 ? sm_count / n : sm_count * 9 / (10 * n);
}

// How many clusters of each size the current device holds at a time (every instance of the kernel takes a whole SM), asked once.
static const int* gemvn_clusters(int sm_count) {
    struct Capacity {
        bool ready = false;
        int clusters[GEMVN_MAX_CLUSTER + 1] = {};
    };
    static Capacity devs[64];
    static std::mutex mu;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    Capacity& d = devs[dev & 63];
    if (d.ready) return d.clusters;
    gemvn_clusters_estimate(sm_count, d.clusters);
    const auto kernel = gemvn_kernel<WF_QTYPE_Q4_0, 1, WAY_CLUSTER, false>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMV_SMEM_LIMIT) == cudaSuccess) {
        for (int n = 2; n <= GEMVN_MAX_CLUSTER; n++) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)n);
            cfg.blockDim = dim3(GEMV_CONSUMERS);
            cfg.dynamicSmemBytes = GEMVN_SMEM;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)n;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int count = 0;
            // one fewer of the larger ones: a cluster that does not find its place in the first wave costs a whole round
            if (cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) == cudaSuccess) d.clusters[n] = n >= 3 && count > 16 ? count - 1 : count;
        }
        d.ready = true;
    }
    cudaGetLastError();  // a failed question leaves the estimate
    return d.clusters;
}

// The cut of a weight for `cols` activation columns, worked out once per weight (the search walks dozens of
// candidates: too slow for every call of a microsecond-scale kernel).
static GemvNPlan cached_plan(int sm_count, const Weight& w, int cols, bool x_f32) {
    Weight::Split& e = const_cast<Weight&>(w).split_cache[x_f32 ? 1 : 0][cols];
    if (e.slices < 0) {
        const GemvNPlan p = gemvn_plan(gemvn_clusters(sm_count), w.g.qtype, w.g.rt, w.g.kt, cols, x_f32);
        e.kc = (short)p.kc;
        e.batch = (short)p.batch;
        e.ctas = (short)p.ctas;
        e.ns = (float)p.ns;
        e.slices = (short)p.slices;
    }
    GemvNPlan p;
    p.slices = e.slices;
    p.kc = e.kc;
    p.batch = e.batch;
    p.ctas = e.ctas;
    p.ns = e.ns;
    p.part = p.slices > GEMVN_MAX_CLUSTER;
    return p;
}

// Activation columns one launch of the several-token kernel can take for this weight: at most 32, fewer when no slice of
// them fits, or the partial sums of more than eight slices would not fit their buffer.
static int gemvn_cols_per_pass(int sm_count, const Weight& w, bool x_f32) {
    for (int cols = GEMVN_MAX_COLS; cols >= (x_f32 ? 3 : 1); cols--)
        if (cached_plan(sm_count, w, cols, x_f32).slices > 0) return cols;
    return 0;
}

// Tokens per launch for a call of m tokens: as many as one launch can take, or 16 columns where the estimate says that
// several launches, which read the weight again, are quicker than one whose activations leave little room for batches of
// sums (a launch boundary costs about 2 us).  32 tokens: Q4_0 [28014 x 4992] 58.4 us in one launch, 50.3 in two; Q4_K
// [28672 x 8192] 122 and 105; [4096 x 4096] 10.0 and 13.4.
static int gemvn_tokens_per_pass(int sm_count, const Weight& w, bool x_f32, int64_t m) {
    const int per_tok = x_f32 ? 3 : 1;
    int best = 0;
    double best_ns = 0;
    for (int cols : {gemvn_cols_per_pass(sm_count, w, x_f32), 16}) {
        const int64_t most = cols / per_tok;
        if (most < 1 || (best > 0 && most >= best)) continue;
        const int64_t passes = (m + most - 1) / most, tokens = (m + passes - 1) / passes;
        const GemvNPlan p = cached_plan(sm_count, w, (int)tokens * per_tok, x_f32);
        if (p.slices < 1) continue;
        const double ns = (double)passes * (p.ns + 2000.0);
        if (best == 0 || ns < best_ns) {
            best_ns = ns;
            best = (int)tokens;
        }
    }
    return best;
}

// Largest number of tokens one launch can take (0: the weight does not fit any kernel).
int gemv_max_tokens_per_pass(const Weight& w, int x_dtype) {
    const bool f32 = x_dtype == WF_DTYPE_F32;
    const int cols = gemvn_cols_per_pass(w.ctx ? w.ctx->sm_count : 148, w, f32);
    const int n = f32 ? cols / 3 : cols;
    if (n == 0 && ws_fits((int)w.g.kt * tile_k(w.g.qtype), 0)) return 1;
    return n;
}

// grid 0: only make the kernel ready (its first use loads it, which can take milliseconds).
template <class Params>
static cudaError_t launch_one_token(void (*kernel)(const Params), bool (&attr_set)[64], const Params& p, int grid, size_t smem, cudaStream_t s) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMV_SMEM_LIMIT);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    if (grid == 0) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(GEMV_CONSUMERS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, p);
}
template <int QT, int KIND> static cudaError_t launch_one_token_of(const GemvParams& p, int grid, size_t smem, cudaStream_t s) {
    static bool attr_set[64] = {};
    return launch_one_token(gemv1_kernel<QT, KIND>, attr_set, p, grid, smem, s);
}
template <int QT, int KIND> static cudaError_t launch_one_token_of(const Gemv1GroupParams& p, int grid, size_t smem, cudaStream_t s) {
    static bool attr_set[64] = {};
    return launch_one_token(gemv1_group_kernel<QT, KIND>, attr_set, p, grid, smem, s);
}
template <int QT> static cudaError_t launch_one_token(const GemvParams& p, int grid, size_t smem, cudaStream_t s) {
    return p.x_f32 ? launch_one_token_of<QT, XK_F32>(p, grid, smem, s) : launch_one_token_of<QT, XK_BF16>(p, grid, smem, s);
}
template <int QT> static cudaError_t launch_one_token(const Gemv1GroupParams& p, int grid, size_t smem, cudaStream_t s) {
    switch (p.x_kind) {
        case XK_F32: return launch_one_token_of<QT, XK_F32>(p, grid, smem, s);
        case XK_RMSNORM_F32: return launch_one_token_of<QT, XK_RMSNORM_F32>(p, grid, smem, s);
        case XK_SWIGLU_F32: return launch_one_token_of<QT, XK_SWIGLU_F32>(p, grid, smem, s);
        default: return launch_one_token_of<QT, XK_BF16>(p, grid, smem, s);
    }
}
template <class Params> static cudaError_t launch_qt_one_token(int qt, const Params& p, int grid, size_t smem, cudaStream_t s) {
    return qt == WF_QTYPE_Q4_0   ? launch_one_token<WF_QTYPE_Q4_0>(p, grid, smem, s)
           : qt == WF_QTYPE_Q4_1 ? launch_one_token<WF_QTYPE_Q4_1>(p, grid, smem, s)
           : qt == WF_QTYPE_Q8_0 ? launch_one_token<WF_QTYPE_Q8_0>(p, grid, smem, s)
                                 : launch_one_token<WF_QTYPE_Q4_K>(p, grid, smem, s);
}

template <int QT, int NG, int WAY, bool GROUP>
static cudaError_t launch_several(const GemvNParams<GROUP ? GEMV_GROUP : 1>& p, int grid, size_t smem, cudaStream_t s) {
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && !attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(gemvn_kernel<QT, NG, WAY, GROUP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMV_SMEM_LIMIT);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    if (grid == 0) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(GEMV_CONSUMERS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.slices;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.cluster ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemvn_kernel<QT, NG, WAY, GROUP>, p);
}
template <int QT, int NG, bool GROUP>
static cudaError_t launch_way(const GemvNParams<GROUP ? GEMV_GROUP : 1>& p, int grid, size_t smem, cudaStream_t s) {
    if (!p.x_f32 && p.slices == 1) return launch_several<QT, NG, WAY_DIRECT, GROUP>(p, grid, smem, s);
    if constexpr (!GROUP) {
        if (p.x_f32 || !p.cluster) return launch_several<QT, NG, WAY_ANY, GROUP>(p, grid, smem, s);
    }
    return launch_several<QT, NG, WAY_CLUSTER, GROUP>(p, grid, smem, s);
}
template <int NG, bool GROUP>
static cudaError_t launch_qt_several(int qt, const GemvNParams<GROUP ? GEMV_GROUP : 1>& p, int grid, size_t smem, cudaStream_t s) {
    return qt == WF_QTYPE_Q4_0   ? launch_way<WF_QTYPE_Q4_0, NG, GROUP>(p, grid, smem, s)
           : qt == WF_QTYPE_Q4_1 ? launch_way<WF_QTYPE_Q4_1, NG, GROUP>(p, grid, smem, s)
           : qt == WF_QTYPE_Q8_0 ? launch_way<WF_QTYPE_Q8_0, NG, GROUP>(p, grid, smem, s)
                                 : launch_way<WF_QTYPE_Q4_K, NG, GROUP>(p, grid, smem, s);
}

// Allocates (once per stream) what the kernels of that stream exchange partial results through: the one-token
// kernel's scratch slots, the several-token kernel's partial sums and arrival counters.  Streams get their own
// so GEMVs on different streams may overlap.
int gemv_prepare_stream(Context* c, cudaStream_t s) {
    GemvScratch& sc = c->gemv_scratch[s];
    if (sc.ctas >= c->sm_count) return WF_OK;
    const int rc = refuse_allocation_while_recording(c, s, "the decode kernels' scratch");
    if (rc != WF_OK) return rc;
    sc.ctas = 0;
    WF_CUDA(c, make_shared_device(c, sc.d_slots, (size_t)c->sm_count * 128 * sizeof(uint2)));
    WF_CUDA(c, cudaMemset(sc.d_slots.get(), 0, (size_t)c->sm_count * 128 * sizeof(uint2)));
    WF_CUDA(c, make_shared_device(c, sc.d_part, GEMVN_PART_BYTES));
    WF_CUDA(c, make_shared_device(c, sc.d_count, (size_t)GEMVN_MAX_ROW_TILES * sizeof(int)));
    WF_CUDA(c, cudaMemset(sc.d_count.get(), 0, (size_t)GEMVN_MAX_ROW_TILES * sizeof(int)));
    sc.ctas = c->sm_count;
    return WF_OK;
}

struct GemvBuffers {
    uint2* slots;  // one-token kernel: [ctas][128] exchange slots
    float* part;   // several tokens: GEMVN_PART_BYTES of partial sums
    int* count;    // several tokens: [GEMVN_MAX_ROW_TILES] arrival counters
};

// One launch per pass of tokens.  clear: zero the exchange slots / arrival counters on the stream before every
// launch (for buffers that may hold leftovers of a failed call).
static int launch_passes(Context* c, const GemvCall& call, cudaStream_t s, const GemvBuffers& buf, bool clear,
                         unsigned long long* timing, const char* what) {
    const Weight& w = *call.w;
    const int qt = w.g.qtype;
    const int kp = (int)w.g.kt * tile_k(qt);
    const bool f32 = call.x_dtype == WF_DTYPE_F32;
    const size_t esz = f32 ? 4 : 2;
    if (call.m == 1 && ws_fits(kp, 0)) {  // one token (bf16 or fp32): the integer path, every warp streaming its own run
        const WsSplit one = ws_split(c->sm_count, w.g.rt, w.g.kt);
        GemvParams p{};
        p.tiles = w.d_tiles;
        p.x = call.d_x;
        p.y = call.d_y;
        p.scratch = buf.slots;
        p.status = c->d_status;
        p.timing = timing;
        p.ldy = call.ldy;
        p.col0 = call.col0;
        p.ldx = w.g.k;
        p.rows = (int)w.g.rows;
        p.k = (int)w.g.k;
        p.kt = (int)w.g.kt;
        p.rt = (int)w.g.rt;
        p.m = 1;
        p.x_f32 = f32;
        p.chunk_q = one.chunk_q;
        p.chunk_r = one.chunk_r;
        p.aligned = one.aligned;
        if (clear) WF_CUDA(c, cudaMemsetAsync(buf.slots, 0, (size_t)one.ctas * 128 * sizeof(uint2), s));
        cudaError_t e = launch_qt_one_token(qt, p, one.ctas, ws_smem(kp, 0), s);
        if (e != cudaSuccess) return cuda_status(c, e, what);
        c->launches++;
        return WF_OK;
    }
    const int per_tok = f32 ? 3 : 1;
    const int per_pass = gemvn_tokens_per_pass(c->sm_count, w, f32, call.m);
    if (per_pass < 1) return set_error(c, WF_ERR_TOO_LARGE, "weight [%lld x %lld] is beyond the decode kernels", (long long)w.g.rows, (long long)w.g.k);
    if (w.g.rt > GEMVN_MAX_ROW_TILES) return set_error(c, WF_ERR_TOO_LARGE, "%lld rows: more than %d row-tiles", (long long)w.g.rows, GEMVN_MAX_ROW_TILES);
    for (int64_t m0 = 0; m0 < call.m; m0 += per_pass) {
        GemvNParams<1> p{};
        p.w[0] = GemvNWeight{w.d_tiles, call.d_y + m0 * call.ldy + call.col0, call.ldy, (int)w.g.rows, (int)w.g.rt};
        p.n_w = 1;
        p.x = static_cast<const uint8_t*>(call.d_x) + (size_t)m0 * w.g.k * esz;
        p.part = buf.part;
        p.count = buf.count;
        p.status = c->d_status;
        p.timing = timing;
        p.timing_at = -1;
        p.ldx = w.g.k;
        p.k = (int)w.g.k;
        p.kt = (int)w.g.kt;
        p.rt = (int)w.g.rt;
        p.m = (int)std::min<int64_t>(call.m - m0, per_pass);
        p.x_f32 = f32;
        p.cols = p.m * per_tok;
        const GemvNPlan plan = cached_plan(c->sm_count, w, p.cols, f32);
        if (plan.slices < 1) return set_error(c, WF_ERR_TOO_LARGE, "no split of K=%lld fits %d activation columns", (long long)w.g.k, p.cols);
        p.slices = plan.slices;
        p.kc = plan.kc;
        p.batch = plan.batch;
        p.cluster = plan.slices > 1 && !plan.part;
        const int ng = (p.cols + 7) / 8;
        const int grid = plan.part ? c->sm_count : plan.ctas * plan.slices;
        const size_t smem = gemvn_smem(qt, p.kc, p.cols, f32, p.slices, p.batch, &p.sx, &p.piece_off, &p.ex_off);
        if (clear && plan.part) WF_CUDA(c, cudaMemsetAsync(buf.count, 0, (size_t)w.g.rt * sizeof(int), s));
        const cudaError_t e = ng == 1   ? launch_qt_several<1, false>(qt, p, grid, smem, s)
                              : ng == 2 ? launch_qt_several<2, false>(qt, p, grid, smem, s)
                              : ng == 3 ? launch_qt_several<3, false>(qt, p, grid, smem, s)
                                        : launch_qt_several<4, false>(qt, p, grid, smem, s);
        if (e != cudaSuccess) return cuda_status(c, e, what);
        c->launches++;
    }
    return WF_OK;
}

static int check_shape(Context* c, const Weight& w, int x_dtype) {
    if (gemv_max_tokens_per_pass(w, x_dtype) < 1)
        return set_error(c, WF_ERR_TOO_LARGE, "K=%lld needs more shared memory than one SM has", (long long)w.g.k);
    if (w.g.rt * w.g.kt >= (1LL << 31)) return set_error(c, WF_ERR_TOO_LARGE, "weight has too many tiles");
    return WF_OK;
}

int gemv_reserve(Context* c, const GemvCall& call, cudaStream_t s) {
    const int rc = check_shape(c, *call.w, call.x_dtype);
    return rc != WF_OK ? rc : gemv_prepare_stream(c, s);
}

int gemv_launch(Context* c, const GemvCall& call, cudaStream_t s) {
    const int rc = gemv_reserve(c, call, s);
    if (rc != WF_OK) return rc;
    if (call.w->g.rt * call.w->g.kt < 1) return WF_OK;
    const GemvScratch& sc = c->gemv_scratch[s];
    return launch_passes(c, call, s, GemvBuffers{sc.d_slots.get(), sc.d_part.get(), sc.d_count.get()}, false, c->salt >= 2 ? c->d_timing : nullptr, "gemv launch");
}

// ---------------------------------------------------------------- a program's launches
static cudaError_t launch_group(const GemvPrepared& g, int grid, cudaStream_t s);
static std::array<GemvNPlan, 2> program_ways(const int* clusters, int qt, int64_t rt, int64_t kt, int tokens) {
    std::array<GemvNPlan, 2> ways = {gemvn_plan(clusters, qt, rt, kt, tokens, false, GEMVN_ONE_SLICE), gemvn_plan(clusters, qt, rt, kt, tokens, false, GEMVN_CLUSTERS)};
    if (rt >= clusters[1]) ways[1].ns += GEMVN_CLUSTER_LATE_NS;
    return ways;
}
bool gemv_plan_groups(Context* c, std::vector<GemvGroup>& groups) {
    if (groups.empty() || groups[0].m < 2) return true;
    std::vector<std::array<GemvNPlan, 2>> ways;
    for (const GemvGroup& g : groups) {
        int64_t rt = 0;
        for (int i = 0; i < g.n; i++) rt += g.w[i]->g.rt;
        ways.push_back(program_ways(gemvn_clusters(c->sm_count), g.w[0]->g.qtype, rt, g.w[0]->g.kt, g.m));
    }
    std::vector<GemvNPlan> plans;
    if (!gemvn_plan_program(ways, &plans)) return false;
    for (size_t i = 0; i < groups.size(); i++) groups[i].plan = plans[i];
    return true;
}
bool gemv_prepare_group(Context* c, const GemvGroup& g, GemvPrepared* out) {
    if (g.n < 1 || g.n > GEMV_GROUP || g.m < 1 || g.m > 8) return false;
    const Weight& first = *g.w[0];
    const int qt = first.g.qtype, kt = (int)first.g.kt, kp = kt * tile_k(qt);
    int64_t rt = 0;
    for (int i = 0; i < g.n; i++) {
        if (g.w[i]->g.qtype != qt || g.w[i]->g.k != first.g.k) return false;
        rt += g.w[i]->g.rt;
    }
    if (rt * kt >= (1LL << 31) || rt > GEMVN_MAX_ROW_TILES) return false;
    out->qt = qt;
    out->m = g.m;
    if (g.m == 1) {
        if (!ws_fits(kp, 0)) return false;
        Gemv1GroupParams& p = out->one;
        p = {};
        int64_t end = 0;
        for (int i = 0; i < g.n; i++) {
            const int64_t begin = g.act != nullptr ? 0 : end;
            end = begin + g.w[i]->g.rt;
            p.op[i] = Gemv1Op{g.w[i]->d_tiles, g.y[i], g.residual[i], (int)g.w[i]->g.rows, (int)begin, (int)end};
        }
        p.n_ops = g.n;
        p.x = g.x;
        p.aux = g.aux;
        p.eps = g.eps;
        p.x_kind = g.x_kind;
        p.k = (int)first.g.k;
        p.kt = kt;
        if (g.n == 1) {
            const WsSplit sp = ws_split(c->sm_count, rt, kt);
            out->grid = sp.ctas;
            p.aligned = sp.aligned;
            p.chunk_q = sp.chunk_q;
            p.chunk_r = sp.chunk_r;
        } else if (g.act != nullptr) {
            const int64_t one = first.g.rt;
            out->grid = (int)std::min<int64_t>(c->sm_count, one);
            p.aligned = 1;
            p.chunk_q = (int)(one / out->grid);
            p.chunk_r = (int)(one % out->grid);
            p.act = g.act;
        } else {  // whole row-tiles of the list: nothing is finished between CTAs
            out->grid = (int)std::min<int64_t>(c->sm_count, rt);
            p.aligned = 1;
            p.chunk_q = (int)(rt / out->grid);
            p.chunk_r = (int)(rt % out->grid);
        }
        p.scratch = g.scratch;
        p.status = c->d_status;
        p.timing = g.timing;
        p.timing_at = g.timing_at;
        out->smem = ws_smem(kp, 0);
        if (g.x_kind == XK_RMSNORM_F32) {  // x and gamma as they are in memory behind the digits, where there is room
            const size_t rows = (size_t)p.k * 4 * (g.aux ? 2 : 1);
            if (out->smem + rows <= GEMV_SMEM_LIMIT) {
                p.x_bytes = p.k * 4;
                out->smem += rows;
            }
        }
        return launch_group(*out, 0, nullptr) == cudaSuccess;
    }
    if (g.x_kind != XK_BF16) return false;
    const GemvNPlan& plan = g.plan;
    if (plan.slices < 1 || plan.part) return false;
    GemvNParams<GEMV_GROUP>& p = out->several;
    p = {};
    int64_t end = 0;
    for (int i = 0; i < g.n; i++) {
        end += g.w[i]->g.rt;
        p.w[i] = GemvNWeight{g.w[i]->d_tiles, g.y[i], g.ldy[i], (int)g.w[i]->g.rows, (int)end};
    }
    p.n_w = g.n;
    p.x = g.x;
    p.status = c->d_status;
    p.timing = g.timing;
    p.timing_at = g.timing_at;
    p.ldx = first.g.k;
    p.k = (int)first.g.k;
    p.kt = kt;
    p.rt = (int)rt;
    p.m = p.cols = g.m;
    p.slices = plan.slices;
    p.kc = plan.kc;
    p.batch = plan.batch;
    p.cluster = plan.slices > 1;
    out->grid = plan.ctas * plan.slices;
    out->smem = gemvn_smem(qt, p.kc, p.cols, false, p.slices, p.batch, &p.sx, &p.piece_off, &p.ex_off);
    return launch_group(*out, 0, nullptr) == cudaSuccess;
}
static cudaError_t launch_group(const GemvPrepared& g, int grid, cudaStream_t s) {
    return g.m == 1 ? launch_qt_one_token(g.qt, g.one, grid, g.smem, s) : launch_qt_several<1, true>(g.qt, g.several, grid, g.smem, s);
}
cudaError_t gemv_launch_group(const GemvPrepared& g, cudaStream_t s) { return launch_group(g, g.grid, s); }

// ---------------------------------------------------------------- allocation-free variant
// What the kernels exchange partial results through lives, for wf_qlinear_noalloc, in these statically sized
// device arrays instead of memory obtained from cudaMalloc: the one-token kernel's slots (256 KiB), the
// several-token kernel's partial sums (8 MiB) and arrival counters (256 KiB).  Every GPU that loads the library
// carries them until the process exits.  One set per device is shared by all calls on that device.
constexpr int GEMV_NOALLOC_MAX_CTAS = 256;  // the kernel launches one CTA per SM
static __device__ __align__(256) uint2 g_noalloc_slots[GEMV_NOALLOC_MAX_CTAS * 128];
static __device__ __align__(256) float g_noalloc_part[GEMVN_PART_BYTES / sizeof(float)];
static __device__ __align__(256) int g_noalloc_count[GEMVN_MAX_ROW_TILES];

// In host code `g_noalloc_slots` is only a handle for the symbol, not an address the GPU can
// use; the device address is looked up once per device, with that device current.
static std::mutex g_noalloc_mu;
static GemvBuffers g_noalloc_ptr[64] = {};

static int noalloc_buffers_for_current_device(Context* c, GemvBuffers* out) {
    if (c->device < 0 || c->device >= 64) return set_error(c, WF_ERR_TOO_LARGE, "device index %d beyond 63", c->device);
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[c->device].slots) {
        GemvBuffers b{};
        cudaError_t e = cudaGetSymbolAddress((void**)&b.slots, g_noalloc_slots);
        if (e == cudaSuccess) e = cudaGetSymbolAddress((void**)&b.part, g_noalloc_part);
        if (e == cudaSuccess) e = cudaGetSymbolAddress((void**)&b.count, g_noalloc_count);
        if (e != cudaSuccess) return cuda_status(c, e, "cudaGetSymbolAddress(static GEMV work arrays)");
        g_noalloc_ptr[c->device] = b;
    }
    *out = g_noalloc_ptr[c->device];
    return WF_OK;
}

// Same kernels and the same work split as gemv_launch, but nothing is allocated: slots, partial sums and
// counters come from the static arrays above; slots and counters are cleared on the stream before every launch,
// because the arrays keep whatever the previous call (possibly a failed one) left in them.
int gemv_launch_noalloc(Context* c, const GemvCall& call, cudaStream_t s) {
    int rc = check_shape(c, *call.w, call.x_dtype);
    if (rc != WF_OK) return rc;
    if (c->sm_count > GEMV_NOALLOC_MAX_CTAS)
        return set_error(c, WF_ERR_TOO_LARGE, "device has %d SMs; the static fix-up array covers at most %d", c->sm_count,
                         GEMV_NOALLOC_MAX_CTAS);
    if (call.w->g.rt * call.w->g.kt < 1) return WF_OK;
    GemvBuffers buf{};
    rc = noalloc_buffers_for_current_device(c, &buf);
    if (rc != WF_OK) return rc;
    return launch_passes(c, call, s, buf, true, nullptr, "gemv launch (no-alloc)");
}

}  // namespace wf

extern "C" int wf_plan_several_tokens(int qtype, int64_t rows, int64_t k, int cols, int x_is_f32, int sm_count, int* slices,
                                      int* k_tiles_per_slice, int* team, int* uses_partial_sums, int64_t* smem_bytes) {
    using namespace wf;
    const int qt = device_qtype(qtype);
    if (qt != WF_QTYPE_Q4_0 && qt != WF_QTYPE_Q4_1 && qt != WF_QTYPE_Q8_0 && qt != WF_QTYPE_Q4_K) return WF_ERR_UNSUPPORTED_TYPE;
    if (rows < 1 || k < 1 || cols < 1 || cols > GEMVN_MAX_COLS || sm_count < 1 || !slices || !k_tiles_per_slice || !team) return WF_ERR_INVALID_ARGUMENT;
    const int64_t rt = (rows + 15) / 16, kt = (k + tile_k(qt) - 1) / tile_k(qt);
    int clusters[GEMVN_MAX_CLUSTER + 1];
    gemvn_clusters_estimate(sm_count, clusters);
    GemvNPlan p = gemvn_plan(clusters, qt, rt, kt, cols, x_is_f32 != 0);
    // sums that meet in clusters need no buffer: a cut whose sums come to more than it holds is not described here
    if (p.slices > 1 && gemvn_sum_bytes(p.slices, cols, rt) > GEMVN_PART_BYTES) p = GemvNPlan{};
    *slices = p.slices;
    *k_tiles_per_slice = p.kc;
    // the warps of a CTA cut its tiles evenly: about this many share a row-tile
    const int share = p.slices > 0 ? GEMV_WARPS / (int)std::min<int64_t>((rt + p.ctas - 1) / p.ctas, GEMV_WARPS) : 1;
    *team = share >= 16 ? 16 : share >= 8 ? 8 : share;
    if (uses_partial_sums) *uses_partial_sums = p.slices > 1 || x_is_f32 ? 1 : 0;
    if (smem_bytes) *smem_bytes = p.slices > 0 ? (int64_t)gemvn_smem(qt, p.kc, cols, x_is_f32 != 0, p.slices, p.batch, nullptr, nullptr, nullptr) : 0;
    return WF_OK;
}

// The cuts of a program's launches without a device (clusters as gemvn_clusters_estimate has them).
extern "C" int wf_plan_program(int qtype, int n, const int64_t* rows, const int64_t* k, int tokens, int sm_count, int* slices, int* k_tiles_per_slice) {
    using namespace wf;
    const int qt = device_qtype(qtype);
    if (qt != WF_QTYPE_Q4_0 && qt != WF_QTYPE_Q4_1 && qt != WF_QTYPE_Q8_0 && qt != WF_QTYPE_Q4_K) return WF_ERR_UNSUPPORTED_TYPE;
    if (n < 1 || n > (1 << 20) || !rows || !k || tokens < 2 || tokens > 8 || sm_count < 1 || !slices || !k_tiles_per_slice) return WF_ERR_INVALID_ARGUMENT;
    int clusters[GEMVN_MAX_CLUSTER + 1];
    gemvn_clusters_estimate(sm_count, clusters);
    std::vector<std::array<GemvNPlan, 2>> ways;
    for (int i = 0; i < n; i++) {
        if (rows[i] < 1 || k[i] < 1) return WF_ERR_INVALID_ARGUMENT;
        ways.push_back(program_ways(clusters, qt, (rows[i] + 15) / 16, (k[i] + tile_k(qt) - 1) / tile_k(qt), tokens));
    }
    std::vector<GemvNPlan> plans;
    if (!gemvn_plan_program(ways, &plans)) plans.assign(n, GemvNPlan{});
    for (int i = 0; i < n; i++) {
        slices[i] = plans[i].slices;
        k_tiles_per_slice[i] = plans[i].kc;
    }
    return WF_OK;
}
