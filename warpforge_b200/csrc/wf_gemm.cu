// Prefill GEMM: y[m, rows] = x[m, K] . W[rows, K]^T for many tokens, W in the tiled quantized
// layout of wf_layout.cuh, on the 5th-generation tensor cores:
//
//   D[weight rows x tokens] (fp32, in TMEM) += A[rows x 16] (fp16, in TMEM) * B[16 x tokens] (fp16, smem)
//
// A call is two kernels: convert_rows_kernel rewrites the activations as fp16 times a power of two per row, and one of
//   gemm_pair_kernel   (wf_gemm_pair.cuh)   pairs of CTAs on tiles of 256 rows x up to 256 tokens, stream-K
//   gemm_split_kernel  (wf_gemm_split.cuh)  clusters of CTAs that split the K of a tile of 128 rows x up to 128 tokens;
//                                           also the kernel of fp32 activations
// dequantizes the weights into TMEM and multiplies.  The launch side and the choice between them are here.
//
// bf16 activations: weights are rounded once to fp16 (at most 2^-11 of a weight) after the exact fp32 dequantization; products
// and sums are fp32 in the tensor core.  Replaces the host transpose + batch_matmul_f32 of
// warpforge-backend-nvidia/src/main/java/io/surfworks/warpforge/backend/nvidia/ops/DotGeneralKernel.java:169-298.
#include "wf_gather_route.h"
#include "wf_gemm_pair.cuh"
#include "wf_gemm_split.cuh"

namespace wf {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

constexpr size_t GEMM_SMEM_LIMIT = 227 * 1024;

bool gemm_supported(const Weight& w, int x_dtype, int64_t m, const void* d_x) {
    // K a multiple of 8 elements and a 16-byte aligned activation pointer: rows are read in 16-byte pieces, the TMA row
    // stride must be a multiple of 16 bytes.  Whole 128-row blocks exist for any row count: the weight buffer is padded
    // to 8 row-tiles with zero scales.
    // fp32 activations keep fp32's range: a weight with values beyond fp16's stays on the decode kernel.
    if (x_dtype == WF_DTYPE_F32 && w.beyond_fp16) return false;
    return many_tokens(x_dtype == WF_DTYPE_F32, m) && (w.g.k % 8) == 0 && (reinterpret_cast<uintptr_t>(d_x) & 15) == 0 && encode_tiled_fn() != nullptr;
}

// What the kernels of one format need to know about a device, found out once: how many clusters of each size it holds
// at a time (a pair's stream-K fix-up needs the whole grid resident; GPCs with an odd SM count hold fewer pairs than SMs / 2).
struct GemmDevice {
    bool ready = false;
    int pairs = 0;
    int clusters[SPLIT_MAX_RANKS + 1] = {};
};
template <class Kernel> static cudaError_t max_clusters(Kernel kernel, int size, int* out) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)size);
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = GEMM_SMEM_LIMIT;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(out, kernel, &cfg);
}
template <int QT> static cudaError_t gemm_prepare(int device, GemmDevice** out) {
    static GemmDevice devs[64];
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    GemmDevice& d = devs[device & 63];
    *out = &d;
    if (d.ready) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel<QT, 1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM_LIMIT);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_split_kernel<QT, 2, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM_LIMIT);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_pair_kernel<QT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM_LIMIT);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_pair_kernel<QT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM_LIMIT);
    if (e == cudaSuccess) e = max_clusters(gemm_pair_kernel<QT, false>, 2, &d.pairs);
    int waved = 0;
    if (e == cudaSuccess) e = max_clusters(gemm_pair_kernel<QT, true>, 2, &waved);
    d.pairs = std::min(d.pairs, waved);
    for (int n = 1; n <= SPLIT_MAX_RANKS && e == cudaSuccess; n++) {
        e = max_clusters(gemm_split_kernel<QT, 1, 1>, n, &d.clusters[n]);
        // one fewer than the device says: a cluster that does not find its place in the first wave costs a whole round
        if (n >= 3 && d.clusters[n] > 16) d.clusters[n]--;
    }
    d.ready = e == cudaSuccess;
    return e;
}

template <class Kernel>
static cudaError_t gemm_launch_one(Kernel kernel, const GemmParams& p, const CUtensorMap& map, int grid, int cluster, size_t smem, cudaStream_t s) {
    // Programmatic stream serialization: this kernel may start while the conversion of the activations (the previous launch
    // of the stream) is still running; what reads the conversion's output waits with griddepcontrol.wait, the rest
    // (barrier set-up, TMEM allocation, the first weight loads and conversions) runs under it.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, p, map);
}

// What a call costs in us by either kernel, fitted to measurements on one B200 (weights from HBM, calls back to back): 2200 calls of the
// split kernel (11 - 2048 tokens, weights from [600 x 6976] to [14336 x 8192], every number of ranks, token tiles of 64, 96 and
// 128), 61 shapes of the pair kernel.  Conversion, launch and start; a cost per unit of 128 k on the busiest CTA or pair, where the
// slower of dequantization and MMAs counts; the parts put together.  The fits are off by 9 % and 5 % (one standard deviation); of 495 calls
// of 40 - 2048 tokens the choice is 1.7 % off the best of the settings that promise most.
// Clusters of one, more than 32 units: the clock sinks and the weights come from memory, up to 0.56 us a unit at K = 8192 (without
// that term Q4_K [8192 x 8192] 256 tokens went to them, 42.7 us, pairs 40.2, three weights in turn 136 and 123; Q4_1 [9000 x 6976] 700
// tokens 91.8 and 75.7).
static double split_cost(int qt, int64_t rounds, int units, int ranks, int bm, int64_t m, bool f32) {
    const double b = bm / 128.0, t = (double)m / 256;
    if (f32) {
        const double dequant = qt == WF_QTYPE_Q4_0 ? 0.76 : qt == WF_QTYPE_Q4_1 ? 0.98 : qt == WF_QTYPE_Q8_0 ? 0.92 : 1.07;
        const double unit = std::max(dequant, 0.56 + 1.12 * b);
        return ranks == 1 ? 3.5 + 1.6 * t + (double)rounds * units * unit : 5.0 + 4.3 * t + (double)rounds * (units * unit + 0.6 * b);
    }
    const double dequant = qt == WF_QTYPE_Q4_0 ? 0.37 : qt == WF_QTYPE_Q4_1 ? 0.42 : qt == WF_QTYPE_Q8_0 ? 0.44 : 0.53;
    const double unit = std::max(dequant, 0.07 + 0.35 * b);
    if (ranks == 1) return 2.5 + 0.7 * t + (double)rounds * (units * (unit + 0.0008 * std::max(0, units - 32)) + 1.3 + 0.25 * b);
    return 3.8 + 1.5 * t + (double)rounds * (units * unit + 3.6 * b);
}
// share: units of the busiest pair; a tile of U units is put together from the pieces of U / share pairs
static double pair_cost(int qt, int64_t share, int k_blocks, int bm, int64_t m) {
    const double b = bm / 256.0, dequant = qt == WF_QTYPE_Q4_0 ? 0.45 : qt == WF_QTYPE_Q4_1 ? 0.5 : qt == WF_QTYPE_Q8_0 ? 0.62 : 0.6;
    return 14.4 + 2.0 * (double)m / 1024 + (double)share * std::max(dequant, 0.79 * b) + 1.6 * b * (double)k_blocks / (double)share;
}
// Where two ways are close, the one that the fits know better: smaller token tiles and clusters instead of pairs have to promise as much.
constexpr double SMALLER_TILES_GAIN = 0.92, CLUSTERS_GAIN = 0.97;

// Whole tiles that each pair takes before the units of the rest are dealt.  A weight is read once per token tile, and where its tiles lie in
// shares one behind the other, the pairs that read the same rows do so at different times: what does not stay in the L2 comes from
// memory each time (Q8_0 [8192 x 8192], 2000 tokens, 8 token tiles: 570 MB; 194 with waves, whose neighbours walk the same rows in step).
// The pieces of the rest meet at the very end then, and nothing hides that: it has to be 24 units a pair.  us without / with waves:
//   a larger weight: Q8_0 [8192 x 8192] 2048 tokens 236 / 209, 1024 tokens 115 / 110, 768 tokens (19 units left) 89.4 / 89.8, [28672 x 4096]
//   600 tokens 136 / 121, [12288 x 4096] 1024 tokens 86.5 / 85, Q4_0 [8192 x 8192] 2048 tokens (37.7 MB) 202 / 196
//   less of it, or less read again: Q8_0 [8192 x 4096] 1024 tokens (35.7 MB) 62.1 / 62.5, Q4_K [14336 x 4096] 1024 tokens (34 MB) 94 / 95,
//   Q8_0 [20000 x 2048] 1024 tokens (131 MB read again) 77.7 / 79.3
constexpr int64_t WAVES_WEIGHT_BYTES = 37000000, WAVES_BYTES_AGAIN = 132000000, WAVES_REST_UNITS = 24;
static int64_t pair_waves(int64_t tiles, int64_t workers, int k_blocks, int token_tiles, int64_t weight_bytes) {
    if (weight_bytes < WAVES_WEIGHT_BYTES || (token_tiles - 1) * weight_bytes < WAVES_BYTES_AGAIN) return 0;
    int64_t waves = tiles / workers;
    while (waves > 0 && (tiles - waves * workers) * k_blocks < WAVES_REST_UNITS * workers) waves--;
    return waves;
}

// CTAs per tile of the split kernel, the cheapest by split_cost.
static int split_ranks(const GemmDevice& d, int qt, int64_t tiles, int k_blocks, int bm, int64_t m, bool f32, double* cost) {
    int best = 1;
    *cost = 1e30;
    for (int n = 1; n <= SPLIT_MAX_RANKS && n <= k_blocks; n++) {
        if (d.clusters[n] < 1) continue;
        const int64_t rounds = (tiles + d.clusters[n] - 1) / d.clusters[n];
        const double t = split_cost(qt, rounds, (k_blocks + n - 1) / n, n, bm, m, f32);
        if (t < *cost) {
            *cost = t;
            best = n;
        }
    }
    return best;
}

// How a call is cut: which kernel, its tiles, and what share of them a CTA or pair has.
struct GemmChoice {
    bool pair;
    int bm, n_tiles, m_tiles, k_blocks;
    int cluster;      // CTAs of a cluster (the ranks that split K), 2 for pairs
    int groups;       // clusters or pairs
    int waves;        // pairs: whole tiles that each takes first
    int64_t rest;     // pairs: units behind the waves
    bool too_large;
};
static GemmChoice gemm_choose(const GemmDevice& d, const WeightGeom& g, int64_t m, bool f32) {
    GemmChoice c{};
    c.k_blocks = (int)((g.k + GEMM_BK - 1) / GEMM_BK);
    // Clusters on tiles of 128 rows x up to 128 tokens.  Token tiles are of one size, in steps of 32 where there are several (the
    // epilogue works on 32 tokens at a time and must not reach into a neighbour); fp32: 96, so that two stages and the
    // exchange buffer fit.
    c.n_tiles = (int)((g.rows + GEMM_BN - 1) / GEMM_BN);
    double cost = 1e30;
    for (int most = f32 ? 96 : SPLIT_MAX_TOKENS; most >= (f32 ? 96 : 64); most -= 32) {  // smaller tiles where they fill the device better
        const int64_t token_tiles = (m + most - 1) / most, grain = token_tiles > 1 ? 32 : 16;
        const int bm = (int)(((m + token_tiles - 1) / token_tiles + grain - 1) / grain * grain);
        const int m_tiles = (int)((m + bm - 1) / bm);
        double t = 0;
        const int ranks = split_ranks(d, g.qtype, (int64_t)c.n_tiles * m_tiles, c.k_blocks, bm, m, f32, &t);
        if (t >= SMALLER_TILES_GAIN * cost) continue;
        cost = t;
        c.bm = bm;
        c.m_tiles = m_tiles;
        c.cluster = ranks;
    }
    c.groups = (int)std::min<int64_t>(d.clusters[c.cluster], (int64_t)c.n_tiles * c.m_tiles);
    // Pairs of CTAs on tiles of 256 rows x up to 256 tokens (of one size, in steps of 32), stream-K shares.  A tile of U units shared by n
    // pairs costs about U / n units plus n - 1 pieces added by its owner, a piece costing about two units: no share is shorter
    // than sqrt(2 U) units, which bounds n for weights with few tiles.
    const int pair_n = (int)((g.rows + 2 * GEMM_BN - 1) / (2 * GEMM_BN)), pair_m = (int)((m + PAIR_TOKENS - 1) / PAIR_TOKENS);
    const int pair_bm = (int)(((m + pair_m - 1) / pair_m + 31) / 32 * 32);
    int min_units = 1;
    while ((int64_t)min_units * min_units < 2 * c.k_blocks) min_units++;
    const int64_t units = (int64_t)pair_n * pair_m * c.k_blocks;
    const int workers = (int)std::min<int64_t>(d.pairs, std::max<int64_t>(1, units / min_units));
    c.too_large = std::max(units, (int64_t)c.n_tiles * c.m_tiles * c.k_blocks) >= (1LL << 30);
    c.pair = !f32 && m > 64 && d.pairs > 0 && CLUSTERS_GAIN * pair_cost(g.qtype, (units + workers - 1) / workers, c.k_blocks, pair_bm, m) < cost;
    if (c.pair) {
        c.bm = pair_bm;
        c.n_tiles = pair_n;
        c.m_tiles = pair_m;
        c.cluster = 2;
        c.groups = workers;
        c.waves = (int)pair_waves((int64_t)pair_n * pair_m, workers, c.k_blocks, pair_m, g.bytes());
        c.rest = units - (int64_t)c.waves * workers * c.k_blocks;
    }
    return c;
}
static cudaError_t gemm_device(int qt, int device, GemmDevice** out) {
    return qt == WF_QTYPE_Q4_0   ? gemm_prepare<WF_QTYPE_Q4_0>(device, out)
           : qt == WF_QTYPE_Q4_1 ? gemm_prepare<WF_QTYPE_Q4_1>(device, out)
           : qt == WF_QTYPE_Q8_0 ? gemm_prepare<WF_QTYPE_Q8_0>(device, out)
                                 : gemm_prepare<WF_QTYPE_Q4_K>(device, out);
}

// The stream's scratch, grown on demand.
static int gemm_scratch(Context* c, cudaStream_t s, GemvScratch& sc, int64_t x16_bytes) {
    if (x16_bytes > sc.x16_bytes) {
        const int rc = refuse_allocation_while_recording(c, s, "the fp16 activation scratch");
        if (rc != WF_OK) return rc;
        sc.d_x16.reset();
        sc.x16_bytes = 0;
        WF_CUDA(c, make_shared_device(c, sc.d_x16, (size_t)x16_bytes));
        sc.x16_bytes = x16_bytes;
    }
    if (!sc.d_gemm_ready) {
        const int rc = refuse_allocation_while_recording(c, s, "the GEMM's piece buffers");
        if (rc != WF_OK) return rc;
        if (!sc.d_gemm_partial) WF_CUDA(c, make_shared_device(c, sc.d_gemm_partial, (size_t)c->sm_count * GEMM_PIECE_TOKENS * GEMM_BN * sizeof(float)));
        const size_t bytes = ((size_t)c->sm_count * 4 + 2) * sizeof(unsigned int);
        std::shared_ptr<unsigned int> ready;
        WF_CUDA(c, make_shared_device(c, ready, bytes));
        WF_CUDA(c, cudaMemsetAsync(ready.get(), 0, bytes, s));
        sc.d_gemm_ready = ready;
    }
    return WF_OK;
}

int gemm_prepare_stream(Context* c, cudaStream_t s) {
    int64_t most = 0;
    for (const auto& kv : c->gemv_scratch) most = std::max(most, kv.second.x16_bytes);
    return most > 0 ? gemm_scratch(c, s, c->gemv_scratch[s], most) : WF_OK;
}

// Bytes of a call's converted rows: the fp16 planes, and behind them (at *scales) the rows' scales.
static int64_t gemm_x16_bytes(const GemvCall& call, int planes, int64_t* scales) {
    const int64_t kx = (call.w->g.k + 63) & ~63LL;  // elements of a converted row
    *scales = (planes * call.m * kx * 2 + 255) & ~255LL;
    return *scales + ((call.m * 4 + 127) & ~127LL);
}

int qlinear_reserve(Context* c, const GemvCall& call, cudaStream_t s) {
    if (gemm_supported(*call.w, call.x_dtype, call.m, call.d_x)) {
        const bool f32 = call.x_dtype == WF_DTYPE_F32;
        int64_t scales;
        const int rc = gemm_scratch(c, s, c->gemv_scratch[s], gemm_x16_bytes(call, f32 ? 3 : 1, &scales));
        if (rc != WF_ERR_RECORDING || !f32) return rc;
    }
    return gemv_reserve(c, call, s);
}

int qlinear_launch(Context* c, const GemvCall& call, cudaStream_t s) {
    // many tokens: tensor-core GEMM; a few tokens: the HBM-bound GEMV
    if (!gemm_supported(*call.w, call.x_dtype, call.m, call.d_x)) return gemv_launch(c, call, s);
    const int rc = gemm_launch(c, call, s);
    // the decode kernels take fp32 tokens without more scratch than a recorded stream has
    return rc == WF_ERR_RECORDING && call.x_dtype == WF_DTYPE_F32 ? gemv_launch(c, call, s) : rc;
}

int gemm_launch(Context* c, const GemvCall& call, cudaStream_t s) {
    const Weight& w = *call.w;
    const int qt = w.g.qtype;
    const bool f32 = call.x_dtype == WF_DTYPE_F32;
    const int planes = f32 ? 3 : 1;
    GemmDevice* dev = nullptr;
    {
        const cudaError_t e = gemm_device(qt, c->device, &dev);
        if (e != cudaSuccess) return cuda_status(c, e, "gemm attributes");
    }
    // the last 128-row block may reach past the padded row-tiles: the weight buffer must cover it
    if ((w.g.rows + GEMM_BN - 1) / GEMM_BN * (GEMM_BN / 16) > w.g.rt_alloc)
        return set_error(c, WF_ERR_SHAPE, "weight buffer does not cover the last 128-row block");
    const GemmChoice ch = gemm_choose(*dev, w.g, call.m, f32);
    if (ch.too_large) return set_error(c, WF_ERR_TOO_LARGE, "GEMM has too many tile steps");
    const bool pair = ch.pair;
    GemmParams p{};
    p.tiles = w.d_tiles;
    p.y = call.d_y;
    p.status = c->d_status;
    p.ldy = call.ldy;
    p.col0 = call.col0;
    p.rows = (int)w.g.rows;
    p.kt_w = (int)w.g.kt;
    p.rt_last = (int)w.g.rt_alloc - 1;
    p.m = (int)call.m;
    p.k_blocks = ch.k_blocks;
    p.bm = ch.bm;
    p.n_tiles = ch.n_tiles;
    p.m_tiles = ch.m_tiles;
    const int cluster = ch.cluster, grid = ch.groups * ch.cluster;
    size_t stage_bytes, exchange = 0;
    if (pair) {
        p.waves = ch.waves;
        p.unit_q = (int)(ch.rest / ch.groups);
        p.unit_r = (int)(ch.rest % ch.groups);
        stage_bytes = PAIR_STAGE;
    } else {
        p.ranks = ch.cluster;
        // The conversion of fp32 rows takes more registers than a GEMM's CTA leaves, so it waits on idle SMs and keeps the next GEMM's
        // clusters from them.  Few rows are worth it: 14 shapes of 11 - 32 tokens 0.95 x (worst 1.02), 26 of 40 - 256 tokens 1.03 x
        // (worst 1.14).
        p.early = !f32 || call.m <= 32;
        p.unit_q = p.k_blocks / p.ranks;
        p.unit_r = p.k_blocks % p.ranks;
        p.tile_q = p.n_tiles * p.m_tiles / ch.groups;
        p.tile_r = p.n_tiles * p.m_tiles % ch.groups;
        stage_bytes = (size_t)split_stage_bytes(planes, p.bm);
        exchange = (size_t)split_exchange_bytes(f32 ? 2 : 1, p.bm, cluster);
    }
    p.stages = (int)std::min<size_t>((GEMM_SMEM_LIMIT - 1024 - exchange) / stage_bytes, pair ? PAIR_STAGES : f32 ? 8 : split_a_stages(1, p.bm));
    // A = fp16 weights, B = fp16 activations, D = fp32; both operands K-major
    p.idesc = (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(p.bm >> 3) << 17) | ((uint32_t)((pair ? 2 * GEMM_BN : GEMM_BN) >> 4) << 24);

    // the activations' fp16 planes and row scales
    const int64_t kx = (w.g.k + 63) & ~63LL;
    int64_t x16_plane;
    const int64_t x16_bytes = gemm_x16_bytes(call, planes, &x16_plane);
    GemvScratch& sc = c->gemv_scratch[s];
    {
        const int rc = gemm_scratch(c, s, sc, x16_bytes);
        if (rc != WF_OK) return rc;
    }
    p.partial = sc.d_gemm_partial.get();
    p.ready = sc.d_gemm_ready.get();
    p.gen = p.ready + (size_t)c->sm_count * 4;
    __half* x16 = reinterpret_cast<__half*>(sc.d_x16.get());
    float* unscale = reinterpret_cast<float*>(sc.d_x16.get() + x16_plane);
    p.row_unscale = unscale;

    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)kx, (cuuint64_t)(call.m * planes)};
    const cuuint64_t strides[1] = {(cuuint64_t)kx * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)(pair ? p.bm / 2 : p.bm)};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_tiled_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x16, dims, strides, box, estr,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(c, WF_ERR_CUDA_BASE + 1, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)call.m);
        cfg.blockDim = dim3(CONVERT_THREADS);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const bool longer = w.g.k > CONVERT_KEEP_SHORT * CONVERT_THREADS * 8;
        const auto convert = f32      ? convert_rows_kernel<3, 2>
                             : longer ? convert_rows_kernel<1, CONVERT_KEEP_LONG>
                                      : convert_rows_kernel<1, CONVERT_KEEP_SHORT>;
        WF_CUDA(c, cudaLaunchKernelEx(&cfg, convert, call.d_x, x16, unscale, (int)call.m, (int)w.g.k));
    }
    c->launches++;
    const size_t smem = pair ? PAIR_SMEM : 1024 + (size_t)p.stages * stage_bytes + exchange;
    auto launch = [&](auto tag) {
        constexpr int QT = decltype(tag)::value;
        return pair  ? gemm_launch_one(p.waves > 0 ? gemm_pair_kernel<QT, true> : gemm_pair_kernel<QT, false>, p, map, grid, cluster, smem, s)
               : f32 ? gemm_launch_one(gemm_split_kernel<QT, 2, 3>, p, map, grid, cluster, smem, s)
                     : gemm_launch_one(gemm_split_kernel<QT, 1, 1>, p, map, grid, cluster, smem, s);
    };
    const cudaError_t e = qt == WF_QTYPE_Q4_0   ? launch(std::integral_constant<int, WF_QTYPE_Q4_0>{})
                          : qt == WF_QTYPE_Q4_1 ? launch(std::integral_constant<int, WF_QTYPE_Q4_1>{})
                          : qt == WF_QTYPE_Q8_0 ? launch(std::integral_constant<int, WF_QTYPE_Q8_0>{})
                                                : launch(std::integral_constant<int, WF_QTYPE_Q4_K>{});
    if (e != cudaSuccess) return cuda_status(c, e, "gemm launch");
    c->launches++;
    return WF_OK;
}

}  // namespace wf

extern "C" int wf_plan_many_tokens(int64_t ctx, int qtype, int64_t rows, int64_t k, int64_t tokens, int x_is_f32, int* pairs, int* tile_tokens,
                                   int* ctas, int* groups, int* waves) {
    using namespace wf;
    Context* c = get_context(ctx);
    if (!c) return WF_ERR_INVALID_HANDLE;
    ScopedLock lk(c);
    if (!lk.ok) return WF_ERR_BUSY;
    WF_CUDA(c, cudaSetDevice(c->device));
    WeightGeom g{};
    g.qtype = device_qtype(qtype);
    if (g.qtype != WF_QTYPE_Q4_0 && g.qtype != WF_QTYPE_Q4_1 && g.qtype != WF_QTYPE_Q8_0 && g.qtype != WF_QTYPE_Q4_K) return WF_ERR_UNSUPPORTED_TYPE;
    if (rows < 1 || k < 1 || k % block_k(qtype) || !many_tokens(x_is_f32 != 0, tokens) || !pairs || !tile_tokens || !ctas || !groups || !waves)
        return WF_ERR_INVALID_ARGUMENT;
    g.rows = rows;
    g.k = k;
    g.rt = (rows + TILE_ROWS - 1) / TILE_ROWS;
    g.kt = (k + tile_k(g.qtype) - 1) / tile_k(g.qtype);
    g.rt_alloc = (g.rt + 7) / 8 * 8;
    GemmDevice* dev = nullptr;
    const cudaError_t e = gemm_device(g.qtype, c->device, &dev);
    if (e != cudaSuccess) return cuda_status(c, e, "gemm attributes");
    const GemmChoice ch = gemm_choose(*dev, g, tokens, x_is_f32 != 0);
    if (ch.too_large) return WF_ERR_TOO_LARGE;
    *pairs = ch.pair ? 1 : 0;
    *tile_tokens = ch.bm;
    *ctas = ch.cluster;
    *groups = ch.groups;
    *waves = ch.waves;
    return WF_OK;
}
