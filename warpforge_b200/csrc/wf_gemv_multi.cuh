// Decode GEMV for several tokens (2 .. 32 activation columns): y[m, rows] = x[m, K] . W[rows, K]^T, memory-bound.
//
// Every warp loads its tiles from global memory straight into registers (the tile layout is the MMA's fragment
// order) and multiplies them on mma.m16n8k16 with exact bf16 operands and fp32 accumulation: the 4-bit codes of a
// 32-k block become A fragments once (unpack8) and meet NG = 1 .. 4 groups of eight activation columns, so the
// integer work per weight byte does not grow with the number of tokens.  fp32 activations enter as three exact
// bf16 columns per token (x = hi + mid + lo), as in the one-pass ring kernel this replaces.
//
// Work split.  K is cut into S slices of kc k-tiles so that a slice of the activations (all columns) fits in shared memory
// and, where a weight has few rows, so that every SM gets some of it.  A unit is one row-tile (16 rows) times one slice.
// A CTA owns consecutive units of one slice; its 16 warps cut the run of their tiles into 16 equal runs, wherever that
// falls: a warp keeps its sums in registers while it stays inside a unit and leaves them in shared memory (a "piece") when
// it leaves the unit or its run ends.  After a barrier the warps add each unit's pieces in warp order.  Units are taken in
// batches as large as the pieces' shared memory allows: mostly one; the first tiles of the next batch are requested before
// a batch is added up.
//
// Slices.  With S = 1 the sums are y.  With S = 2 .. 8 the CTAs of the S slices form a cluster that shares its row-tiles
// out: each CTA sends the sums of a unit to the CTA that owns the row-tile (st.async into its shared memory, counted by an
// mbarrier there), which adds the slices in order and stores y.  Only a K too long for eight slices (32 columns beyond
// 16384, 24 beyond 22528, 16 beyond 40960) goes through memory: partial sums [row-tile][slice], an arrival counter per row-tile, and the
// warp that finds all other slices already counted adds them, in slice order, and puts the counter back to zero.  Nowhere
// does the result depend on who comes last, and nobody waits for a CTA outside its cluster.
//
// What bounds it: at few columns the weight bytes; at 9 and more the instructions (per 32-k block and eight columns a
// 16-byte and an 8-byte shared load, two MMAs, four FMAs); on small shards the chain launch - activations - tiles - sums.
// Teams of warps per row-tile and partial
// sums in memory for every S > 1 took, 16 columns, Q4_K: 1024 x 8192 10.1 us, 3584 x 8192 15.8, 1024 x 28672 19.3; the even
// cut and the clusters take 5.8, 11.9 and 13.0.  4096 x 4096 Q4_0, one slice: 5.5 -> 4.6 at 4 columns, 9.2 -> 6.7 at 16,
// 17.0 -> 9.9 at 32.
//
// Replaces, for up to 32 tokens, the fp32 batch_matmul_f32 launch of
// warpforge-backend-nvidia/src/main/java/io/surfworks/warpforge/backend/nvidia/ops/DotGeneralKernel.java:263-281.
#pragma once
#include <array>

#include "wf_gemv_stream.cuh"

namespace wf {

constexpr int GEMVN_MAX_COLS = 32;
constexpr int GEMVN_MAX_SLICES = 64;
constexpr int GEMVN_MAX_CLUSTER = 8;  // slices that meet in a cluster (the largest portable size)
constexpr int GEMVN_MAX_BATCH = 64;   // units a CTA adds up at a time
// Shared memory that a plan may fill.  bf16 tokens: what wf_plan_several_tokens has always kept to.  fp32 tokens, whose rows
// are three columns, need more of it for their sums: with all there is, the units of a CTA are mostly one batch (ten tokens,
// Q4_0 [6704 x 9728]: 34.7 -> 31.8 us).
constexpr size_t GEMVN_SMEM = 200 * 1024, GEMVN_SMEM_F32 = 227 * 1024;
constexpr size_t GEMVN_PART_BYTES = 8u << 20;  // partial sums a launch may use (the static array of the no-alloc entry is this large)
constexpr int GEMVN_MAX_ROW_TILES = 1 << 16;   // arrival counters

struct GemvNWeight {
    const uint8_t* tiles;
    float* y;  // its first row of the first token
    int64_t ldy;
    int rows, rt_end;  // rt_end: row-tiles of the launch's weights up to and with this one
};
template <int GROUP> struct GemvNParams {
    GemvNWeight w[GROUP];  // one weight, or several of the same K that read the same activations, as one list of row-tiles
    int n_w;
    const void* x;
    float* part;  // [rt][slices][column pairs][8] float4, used beyond GEMVN_MAX_CLUSTER slices
    int* count;   // [rt] arrivals per row-tile, zero between launches
    int* status;
    int64_t ldx;
    int k, kt, rt;
    int m, x_f32, cols;     // cols = activation columns = m (bf16) or 3 m (fp32)
    int slices, kc, batch;  // k-slices; k-tiles per slice (the last slice may have fewer); units added up at a time
    int cluster;            // the slices of a row-tile are the CTAs of a cluster
    int sx;                 // bytes per staged activation row
    int piece_off, ex_off;  // byte offsets in shared memory: pieces; sums on their way to y
    unsigned long long* timing;  // optional globaltimer stamps: [ctas][8], or a program's [ctas][64]
    int timing_at;               // -1, or this launch's first stamp in a program's row
};

struct GemvNPlan {
    int slices = 0, kc = 0, batch = 0;  // slices == 0: no plan fits
    int ctas = 0;                       // CTAs (per slice, where the slices form clusters)
    bool part = false;                  // partial sums go through memory
    double ns = 0;                      // the estimate
};

// A program's launch: weights of one type and K that read the same activations.
struct GemvGroup {
    int n = 0, m = 1;
    const Weight* w[GEMV_GROUP] = {};
    float* y[GEMV_GROUP] = {};
    int64_t ldy[GEMV_GROUP] = {};
    const float* residual[GEMV_GROUP] = {};
    const void* x = nullptr;
    int x_kind = 0;
    const float* aux = nullptr;
    float eps = 0.f;
    float* act = nullptr;  // two weights, a gate and an up projection: silu(gate) * up goes here as well
    uint2* scratch = nullptr;
    unsigned long long* timing = nullptr;
    int timing_at = -1;
    GemvNPlan plan;  // several tokens: gemv_plan_groups
};
struct GemvPrepared {
    int qt = 0, m = 1, grid = 0;
    size_t smem = 0;
    Gemv1GroupParams one;
    GemvNParams<GEMV_GROUP> several;
};
bool gemv_plan_groups(Context* c, std::vector<GemvGroup>& groups);  // a program's launches in their order; false: beyond the kernels
bool gemv_prepare_group(Context* c, const GemvGroup& g, GemvPrepared* out);  // false: beyond the kernels
cudaError_t gemv_launch_group(const GemvPrepared& g, cudaStream_t s);

template <int QT, int NG> struct GemvNGeom {
    // tiles a warp holds in registers while it multiplies: what 128 registers per thread leave room for
    static constexpr int DEPTH = (QT == WF_QTYPE_Q4_0) ? (NG >= 3 ? 3 : 4) : (QT == WF_QTYPE_Q4_1) ? 3 : (QT == WF_QTYPE_Q8_0 && NG == 1) ? 3 : 2;
};

// Shared memory: control 128 | start values [kc * TK / 32][NG][4] float2 | staged x [cols][sx] | pieces [batch + 15][NG][32]
// float4 | sums of the CTA's own row-tiles [slices][ceil(batch / slices)][NG][32] float4 (a cluster's exchange, or fp32
// tokens, whose three columns meet there).
inline size_t gemvn_smem(int qt, int kc, int cols, bool x_f32, int slices, int batch, int* sx_out, int* piece_off_out, int* ex_off_out) {
    const int kslice = kc * tile_k(qt), ng = (cols + 7) / 8;
    const int sx = kslice * 2 + 64;  // +64: consecutive rows start 16 banks apart
    if (sx_out) *sx_out = sx;
    size_t b = 128 + (size_t)(kslice / 32) * ng * 32 + (size_t)cols * sx;
    b = (b + 127) & ~(size_t)127;
    if (piece_off_out) *piece_off_out = (int)b;
    b += (size_t)(batch + GEMV_WARPS - 1) * ng * 512;
    if (ex_off_out) *ex_off_out = (int)b;
    if (slices <= GEMVN_MAX_CLUSTER && (slices > 1 || x_f32)) b += (size_t)slices * ((batch + slices - 1) / slices) * ng * 512;
    return b;
}

inline size_t gemvn_sum_bytes(int slices, int cols, int64_t rt) { return (size_t)slices * ((cols + 1) & ~1) * rt * 16 * 4; }

// clusters[S]: how many clusters of S CTAs the device holds at a time (S = 1: SMs).  The cheapest cut by an estimate in
// nanoseconds: the busiest warp's tiles, the staging of the slice, and per batch the way of its sums to y.  The constants
// are a fit to 78 measured weights from 128 x 8192 to 28014 x 2496 with 2 .. 32 columns, each at every S up to 8.  In calls of
// more than 13 us clusters of 3, 5 and 7 take longer than that by 8 % and 4 %, and 20 % on devices whose GPCs hold an odd
// number of 7s.  On 130 other weights, up to 32000 x 8192, the choices are 1.4 % slower than the best S on average and 14 % at
// worst (2.4 % and 32 % without that correction).  Memory is the way where eight slices do not fit (against a cluster of the
// same S it measured 1 - 4 us more on small weights, up to twice the time on tall ones).
// ways: which cuts are considered.
constexpr int GEMVN_ONE_SLICE = 1, GEMVN_CLUSTERS = 2, GEMVN_MEMORY = 4, GEMVN_ANY = 7;
inline GemvNPlan gemvn_plan(const int* clusters, int qt, int64_t rt, int64_t kt, int cols, bool x_f32, int ways = GEMVN_ANY) {
    GemvNPlan best;
    const int ng = (cols + 7) / 8, tk = tile_k(qt), sms = clusters[1];
    const double per_group = 15.9 + (qt == WF_QTYPE_Q4_1 ? 3.3 : qt == WF_QTYPE_Q8_0 ? 16.3 : qt == WF_QTYPE_Q4_K ? 5.0 : 0.0);
    const double tile_ns = (tk / 128) * (17.3 + per_group * ng);  // one SM's time per tile
    double best_ns = 0;
    int last_kc = 0;
    for (int s = 1; s <= GEMVN_MAX_SLICES && s <= kt && s <= sms; s++) {
        const int kc = (int)((kt + s - 1) / s), slices = (int)((kt + kc - 1) / kc);
        if (kc == last_kc) continue;
        last_kc = kc;
        const bool part = slices > GEMVN_MAX_CLUSTER;
        if (!(ways & (slices == 1 ? GEMVN_ONE_SLICE : part ? GEMVN_MEMORY : GEMVN_CLUSTERS))) continue;
        if (part && gemvn_sum_bytes(slices, cols, rt) > GEMVN_PART_BYTES) continue;
        const int64_t room = part ? sms / slices : clusters[slices];  // CTAs a slice gets, at least
        if (room < 1) continue;
        const int64_t units = (rt + std::min(room, rt) - 1) / std::min(room, rt);  // of the busiest CTA
        int batch = (int)std::min<int64_t>(units, GEMVN_MAX_BATCH);
        while (batch >= 1 && gemvn_smem(qt, kc, cols, x_f32, slices, batch, nullptr, nullptr, nullptr) > (x_f32 ? GEMVN_SMEM_F32 : GEMVN_SMEM)) batch--;
        if (batch < 1) continue;
        double ns = (double)cols * kc * tk * 2 / (x_f32 ? 27.2 : 87.3);
        for (int64_t left = units; left > 0; left -= batch) {
            const int nb = (int)std::min<int64_t>(batch, left), own = (nb + slices - 1) / slices;
            ns += ((nb * kc + GEMV_WARPS - 1) / GEMV_WARPS) * GEMV_WARPS * tile_ns;
            ns += 847.0 + (x_f32 ? 270.0 : 223.0) * ((nb * ng + GEMV_WARPS - 1) / GEMV_WARPS);
            if (part) ns += 1313.0 + 119.4 * nb * ng + 145.2 * slices;
            else if (slices > 1) ns += 616.0 + slices * (6.1 + 32.1 * ((own * ng + GEMV_WARPS - 1) / GEMV_WARPS));
            if (x_f32 && !part) ns += 31.1 * slices * ((own * (cols / 3) * 16 + GEMV_CONSUMERS - 1) / GEMV_CONSUMERS);
        }
        if (!part && ns > 13000.0) ns *= slices == 3 || slices == 7 ? 1.1 : slices == 5 ? 1.05 : 1.0;
        if (best.slices == 0 || ns < best_ns) {
            best_ns = ns;
            best.slices = slices;
            best.kc = kc;
            best.batch = batch;
            best.ctas = (int)std::min(room, rt);
            best.part = part;
            best.ns = ns;
        }
    }
    return best;
}

// The cuts of a program's launches, which follow each other again and again: ways[i] = the cheapest cut of launch i into one slice and
// into clusters (sums through memory are not for them; slices == 0: does not fit).  The estimates come from calls of one kind in a
// row.  In a program a launch of one slice takes each SM half a microsecond before the launch in front of it ends, but behind
// clusters, which need several SMs at once, it starts 1 us after that end, as clusters do themselves.  So a change from clusters to
// one slice is charged, and clusters where one slice has work for every SM; what is least is the sum over the circle of
// launches.  Measured: 204 programs (Q4_0, Q4_1, Q8_0, Q4_K; 2 - 8 tokens; decoder layers of d 1024 to 4096) at nine settings of
// the two charges, and 14 programs of like launches.  Without them layers take 1.9 % more than with the best setting of each, up to
// 21 % ([2816 x 7680] Q4_K); 1.5 us on every launch of clusters and nothing else: 0.2 %, up to 4 %, but programs of like launches
// with few rows 9 %, up to 33 % ([1024 x 9216] Q4_K, four tokens).
constexpr double GEMVN_CHANGE_NS = 700.0, GEMVN_CLUSTER_LATE_NS = 800.0;
inline bool gemvn_plan_program(const std::vector<std::array<GemvNPlan, 2>>& ways, std::vector<GemvNPlan>* out) {
    const size_t n = ways.size();
    constexpr double NEVER = 1e30;
    const auto cost = [&](size_t i, int w) { return ways[i][w].slices > 0 ? ways[i][w].ns : NEVER; };
    const auto change = [](int from, int to) { return from == 1 && to == 0 ? GEMVN_CHANGE_NS : 0.0; };
    double best = NEVER;
    for (int first = 0; first < 2; first++) {  // the first launch's way, which the last one's successor has as well
        std::vector<std::array<int, 2>> from(n);
        double sum[2] = {first == 0 ? cost(0, 0) : NEVER, first == 1 ? cost(0, 1) : NEVER};
        for (size_t i = 1; i < n; i++) {
            double next[2];
            for (int w = 0; w < 2; w++) {
                from[i][w] = sum[1] + change(1, w) < sum[0] + change(0, w);
                next[w] = sum[from[i][w]] + change(from[i][w], w) + cost(i, w);
            }
            sum[0] = next[0];
            sum[1] = next[1];
        }
        int last = sum[1] + change(1, first) < sum[0] + change(0, first);
        const double total = sum[last] + change(last, first);
        if (total >= best) continue;
        best = total;
        out->assign(n, GemvNPlan{});
        for (size_t i = n; i-- > 0; last = from[i][last]) (*out)[i] = ways[i][last];
    }
    return best < NEVER;
}

// Stage this CTA's k-slice [k_lo, k_lo + kslice) of every token: bf16 rows of kslice elements (zero beyond k) and,
// per 32-k block, group of eight columns and column pair q, the float2 {beta X(2q), beta X(2q+1)} with X the fp32
// sum of the block's 32 activations of that column (the start values of rows g and g+8 alike).
//
// bf16 activations: the rows are copied verbatim, one bulk asynchronous copy per token straight into shared
// memory (no registers, no per-thread load latency; `bar` is an initialised mbarrier with one arrival pending),
// and the block sums are taken from shared memory afterwards, one (column, block) per thread, in the association
// ((s0 + s1) + (s2 + s3)) of four eight-element runs.
template <class Params> static __device__ void stage_x_slice_bulk(const Params& p, uint8_t* xs, float* cinit, int k_lo, int kslice, int ng, float beta,
                                          int nthreads, uint32_t bar, uint32_t abort32) {
    const int valid = max(0, min(kslice, p.k - k_lo));  // elements of the slice that exist
    if (threadIdx.x < 32) {  // one token per lane
        if (threadIdx.x == 0) mbar_expect_tx(bar, (uint32_t)(p.m * valid * 2));
        __syncwarp();
        const int t = threadIdx.x;
        if (t < p.m && valid > 0)
            bulk_load(smem_u32(xs + (size_t)t * p.sx), static_cast<const uint16_t*>(p.x) + (size_t)t * p.ldx + k_lo, (uint32_t)valid * 2, bar);
    }
    if (valid < kslice) {  // K ends inside the slice: zeros behind it (k is a multiple of 32, so whole 16-byte pieces)
        const int pieces = (kslice - valid) >> 3;
        for (int i = threadIdx.x; i < p.m * pieces; i += nthreads) {
            const int t = i / pieces, c = i - t * pieces;
            *reinterpret_cast<uint4*>(xs + (size_t)t * p.sx + (size_t)(valid + c * 8) * 2) = make_uint4(0u, 0u, 0u, 0u);
        }
        __syncthreads();
    }
    mbar_wait_or_abort(bar, 0, abort32);
    // Neighbouring threads take neighbouring tokens of one block: their rows start 16 banks apart, so every second one
    // meets the banks of the first, and each such pair starts at another of the block's four 16-byte runs (taken
    // through an exclusive or, which leaves the pairs of the final additions what they are).
    const int nblk = kslice >> 5;
    for (int i = threadIdx.x; i < p.m * nblk; i += nthreads) {
        const int b = i / p.m, t = i - b * p.m, rot = (threadIdx.x >> 1) & 3;
        const uint4* src = reinterpret_cast<const uint4*>(xs + (size_t)t * p.sx + (size_t)b * 64);
        float part[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint4 v = src[j ^ rot];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            float sum = 0.f;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                sum += __uint_as_float(w[e] << 16);
                sum += __uint_as_float(w[e] & 0xFFFF0000u);
            }
            part[j] = sum;
        }
        const float v = beta * ((part[0] + part[1]) + (part[2] + part[3]));
        cinit[(size_t)b * ng * 8 + t] = v;  // [block][group][q] float2 = [block][column]
    }
}

// fp32 activations (three bf16 columns per token), through registers.
template <class Params> static __device__ void stage_x_slice(const Params& p, uint8_t* xs, float* cinit, int k_lo, int kslice, int ng, float beta,
                                     int nthreads) {
    const int groups = kslice >> 3;  // 8 elements per thread step; a multiple of 4
    const int total = p.m * groups;
    const int padded = (total + 31) & ~31;
    // Every CTA of a slice reads the same activations: each starts at another place of the list (a multiple of 32
    // items, so warps and the four threads of a block stay together), or all of them would ask the same L2 lines at
    // the same moment.
    const int rot = (int)(((int64_t)(blockIdx.x / p.slices) * 2654435761LL) % (padded >> 5)) << 5;
    auto item = [&](int raw) {
        const int i = raw + rot;
        return i >= padded ? i - padded : i;
    };
    // block sums: 4 consecutive threads hold one 32-element block (groups is a multiple of 4, so they belong to one token)
    auto block_sums = [&](float (&sum)[3], bool live, int t, int c8) {
#pragma unroll
        for (int s = 0; s < 3; s++) {
            sum[s] += __shfl_xor_sync(0xFFFFFFFFu, sum[s], 1);
            sum[s] += __shfl_xor_sync(0xFFFFFFFFu, sum[s], 2);
        }
        if (live && (threadIdx.x & 3) == 0) {
            float* blk = cinit + (size_t)(c8 >> 2) * ng * 8;  // [group][q] float2 = [column]
            const int parts = p.x_f32 ? 3 : 1;
            for (int s = 0; s < parts; s++) blk[p.x_f32 ? 3 * t + s : t] = beta * sum[s];
        }
    };
    // four items' loads in flight: one after the other, each paid a trip to the L2
    constexpr int AHEAD = 4;
    for (int raw0 = threadIdx.x; raw0 < padded; raw0 += AHEAD * nthreads) {  // warp-uniform trip counts
        float4 va[AHEAD], vb[AHEAD];
#pragma unroll
        for (int j = 0; j < AHEAD; j++) {
            const int raw = raw0 + j * nthreads, idx = raw < padded ? item(raw) : total;
            const int t = idx < total ? idx / groups : 0, c8 = idx - t * groups, kk = k_lo + c8 * 8;
            va[j] = vb[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (idx < total && kk < p.k) {
                const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(p.x) + (size_t)t * p.ldx + kk);
                va[j] = __ldcg(src);
                vb[j] = __ldcg(src + 1);
            }
        }
#pragma unroll
        for (int j = 0; j < AHEAD; j++) {
            const int raw = raw0 + j * nthreads;
            if (raw >= padded) break;
            const int idx = item(raw);
            const bool live = idx < total;
            const int t = live ? idx / groups : 0, c8 = live ? idx - t * groups : 0;
            float sum[3] = {0.f, 0.f, 0.f};
            const float f[8] = {va[j].x, va[j].y, va[j].z, va[j].w, vb[j].x, vb[j].y, vb[j].z, vb[j].w};
            uint32_t hi[4], mid[4], lo[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float x0 = f[2 * i], x1 = f[2 * i + 1];
                const float h0 = __uint_as_float(__float_as_uint(x0) & 0xFFFF0000u);
                const float h1 = __uint_as_float(__float_as_uint(x1) & 0xFFFF0000u);
                const float r0 = x0 - h0, r1 = x1 - h1;
                const float m0 = __uint_as_float(__float_as_uint(r0) & 0xFFFF0000u);
                const float m1 = __uint_as_float(__float_as_uint(r1) & 0xFFFF0000u);
                const float l0 = r0 - m0, l1 = r1 - m1;  // at most 8 significant bits left: exact in bf16
                hi[i] = pack_bf16_trunc(h0, h1);
                mid[i] = pack_bf16_trunc(m0, m1);
                lo[i] = pack_bf16_trunc(l0, l1);
                sum[0] += h0 + h1;
                sum[1] += m0 + m1;
                sum[2] += l0 + l1;
            }
            if (live) {
                *reinterpret_cast<uint4*>(xs + (size_t)(3 * t) * p.sx + c8 * 16) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(xs + (size_t)(3 * t + 1) * p.sx + c8 * 16) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
                *reinterpret_cast<uint4*>(xs + (size_t)(3 * t + 2) * p.sx + c8 * 16) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            block_sums(sum, live, t, c8);
        }
    }
}

// What lies between a unit's sums and y.  Its own kernel for each of the two ways that most calls take: the code after the
// last tile runs once and is fetched from the L2, so the branches it would jump over cost a small call 0.4 us.
enum GemvNWay {
    WAY_DIRECT,   // one slice, bf16 tokens: straight to y
    WAY_CLUSTER,  // the slices of bf16 tokens meet in a cluster
    WAY_ANY       // fp32 tokens, or partial sums in memory
};

template <int QT, int NG, int WAY, bool GROUP>
__global__ void __launch_bounds__(GEMV_CONSUMERS, 1) gemvn_kernel(const GemvNParams<GROUP ? GEMV_GROUP : 1> p) {
    using T = Tile<QT>;
    using R = TileRegs<QT>;
    constexpr int DEPTH = GemvNGeom<QT, NG>::DEPTH;
    constexpr uint32_t XSTEP = T::K * 2, CSTEP = (T::K / 32) * NG * 32;  // staged bytes per tile
    extern __shared__ __align__(128) uint8_t smem[];

    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int S = WAY == WAY_DIRECT ? 1 : p.slices, slice = (int)blockIdx.x % S, idx = (int)blockIdx.x / S;  // slice = rank in the cluster
    const int ctas = ((int)gridDim.x - slice + S - 1) / S;                                                    // CTAs working on this slice
    const int k0t = slice * p.kc, kcs = min(p.kc, p.kt - k0t);
    const int u0 = (int)((unsigned)(idx * p.rt) / (unsigned)ctas), nu = (int)((unsigned)((idx + 1) * p.rt) / (unsigned)ctas) - u0;  // its units
    const bool cluster = WAY == WAY_CLUSTER || (WAY == WAY_ANY && p.cluster), f32 = WAY == WAY_ANY && p.x_f32;

    auto stamp = [&](int i) {
        if (p.timing != nullptr && threadIdx.x == 0) {
            unsigned long long tm;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(tm));
            if (!GROUP || p.timing_at < 0) {
                p.timing[(size_t)blockIdx.x * 8 + i] = tm;
            } else {  // a program's op: start, waited, staged, done
                const int at = p.timing_at + (i == 3 ? 0 : i == 4 ? 3 : i + 1);
                if (at < 64) p.timing[(size_t)blockIdx.x * 64 + at] = tm;
            }
        }
    };
    // Programmatic stream serialization, as in the one-token kernel: the weights depend on nothing, so the first
    // tiles are requested before the wait for the previous grid.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    stamp(3);
    // A batch: its units and tiles, this warp's run of them [lo, lo + nt), the unit and k-tile the run starts in.
    int nb = 0, total = 0, nt = 0, unit = 0, kk = 0;
    R slots[DEPTH];
    const uint8_t* lptr = nullptr;
    int lkk = 0, lrem = 0;
    int lw = 0, lleft = 0;  // GROUP: the weight being requested from and its row-tiles from here on
    auto load_next = [&](R& slot) {
        if (lrem > 0) {
            slot.load_global_n(lptr, lane);
            lrem--;
            lptr += T::BYTES;
            if (++lkk == kcs) {  // next unit: the same k-tiles of the next row-tile
                lkk = 0;
                lptr += (size_t)(p.kt - kcs) * T::BYTES;
                if (GROUP && --lleft == 0 && lw + 1 < p.n_w) {
                    lw++;
                    lleft = p.w[lw].rt_end - p.w[lw - 1].rt_end;
                    lptr = p.w[lw].tiles + (size_t)k0t * T::BYTES;
                }
            }
        }
    };
    auto open_batch = [&](int b0) {
        nb = min(p.batch, nu - b0);
        total = nb * kcs;
        // 16 equal runs; one tile for each of the first warps where there are fewer
        const bool each = total < GEMV_WARPS;
        const int lo = each ? min(warp, total) : (int)((unsigned)(warp * total) / GEMV_WARPS);
        nt = (each ? min(warp + 1, total) : (int)((unsigned)((warp + 1) * total) / GEMV_WARPS)) - lo;
        unit = (int)((unsigned)lo / (unsigned)kcs);
        kk = lkk = lo - unit * kcs;
        lrem = nt;
        int u = u0 + b0 + unit;
        if (GROUP) {
            for (lw = 0; lw + 1 < p.n_w && u >= p.w[lw].rt_end; lw++) {}
            lleft = p.w[lw].rt_end - u;
            u -= lw > 0 ? p.w[lw - 1].rt_end : 0;
        }
        lptr = p.w[GROUP ? lw : 0].tiles + ((size_t)u * p.kt + k0t + kk) * T::BYTES;
        static_for<DEPTH>([&](auto J) { load_next(slots[decltype(J)::value]); });
    };
    open_batch(0);
    // control words: mbarrier of the activation copies at 0, abort word at 8, mbarrier of the cluster's sums at 16, the units
    // that this CTA completed: their number at 24, they at 32 .. 95
    const uint32_t abort32 = smem_u32(smem + 8), sums_bar = smem_u32(smem + 16);
    if (threadIdx.x == 0) {
        *reinterpret_cast<volatile int*>(smem + 8) = 0;
        mbar_init(smem_u32(smem), 1);
        mbar_init(sums_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // the others may send sums here from now on; waited for before the first ones are sent
    if (cluster) asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");

    float* cinit = reinterpret_cast<float*>(smem + 128);  // [kslice / 32][NG][4] float2
    const int kslice = kcs * T::K;
    uint8_t* xs = reinterpret_cast<uint8_t*>(cinit + (size_t)(p.kc * T::K / 32) * NG * 8);
    float4* const pieces = reinterpret_cast<float4*>(smem + p.piece_off);  // [unit of the batch + warp][NG][32]
    float4* const sums = reinterpret_cast<float4*>(smem + p.ex_off);       // [slice][own unit][NG][32]

    asm volatile("griddepcontrol.wait;" ::: "memory");
    stamp(0);
    if (f32) stage_x_slice(p, xs, cinit, k0t * T::K, kslice, NG, R::BETA, GEMV_CONSUMERS);
    else stage_x_slice_bulk(p, xs, cinit, k0t * T::K, kslice, NG, R::BETA, GEMV_CONSUMERS, smem_u32(smem), abort32);
    __syncthreads();
    stamp(1);
    if (*reinterpret_cast<volatile int*>(smem + 8)) {  // the copies did not land in time: y will be garbage, the status says so
        if (threadIdx.x == 0) report_status(p.status, STATUS_GEMV_FIXUP_TIMEOUT);
        drain_after_abort();
    }

    // dead columns read the last live row: their results are computed and never stored
    uint32_t xg[NG];
#pragma unroll
    for (int gi = 0; gi < NG; gi++) xg[gi] = smem_u32(xs) + (uint32_t)min(8 * gi + g, p.cols - 1) * p.sx + q * 16;
    const uint32_t c32 = smem_u32(cinit) + q * 8;
    const int pairs = (p.cols + 1) >> 1;  // live column pairs: a lane's float4 is one of them in two rows

    // a unit's sums of eight columns, as the lanes hold them, to y (bf16 tokens)
    auto store_y = [&](int u, int gi, const float4& v) {
        int at = 0;
        if (GROUP) {
            while (at + 1 < p.n_w && u >= p.w[at].rt_end) at++;
            u -= at > 0 ? p.w[at - 1].rt_end : 0;
        }
        const GemvNWeight& w = p.w[at];
        const int r0 = u * 16 + g, r1 = r0 + 8, col = 8 * gi + 2 * q;
        float* const y = w.y + (int64_t)col * w.ldy + r0;
        if (col < p.cols) {
            if (r0 < w.rows) y[0] = v.x;
            if (r1 < w.rows) y[8] = v.z;
        }
        if (col + 1 < p.cols) {
            if (r0 < w.rows) y[w.ldy] = v.y;
            if (r1 < w.rows) y[w.ldy + 8] = v.w;
        }
    };
    // place of (column, row) among a unit's float4s, in floats
    auto place = [](int col, int row) { return ((col >> 3) * 32 + (row & 7) * 4 + ((col & 7) >> 1)) * 4 + (row >> 3) * 2 + (col & 1); };

    for (int b0 = 0, round = 0; b0 < nu; b0 += p.batch, round++) {
        float acc[NG][4];
#pragma unroll
        for (int gi = 0; gi < NG; gi++) acc[gi][0] = acc[gi][1] = acc[gi][2] = acc[gi][3] = 0.f;
        for (int g0 = 0; g0 < nt; g0 += DEPTH) {
            static_for<DEPTH>([&](auto J) {
                constexpr int j = decltype(J)::value;
                if (g0 + j < nt) {
                    slots[j].template compute_n<NG>(acc, xg, (uint32_t)kk * XSTEP, c32 + (uint32_t)kk * CSTEP);
                    load_next(slots[j]);
                    if (++kk == kcs || g0 + j + 1 == nt) {  // the piece's place is its own: unit + warp grows along the run
                        float4* const to = pieces + (size_t)(unit + warp) * NG * 32 + lane;
#pragma unroll
                        for (int gi = 0; gi < NG; gi++) {
                            to[gi * 32] = make_float4(acc[gi][0], acc[gi][1], acc[gi][2], acc[gi][3]);
                            acc[gi][0] = acc[gi][1] = acc[gi][2] = acc[gi][3] = 0.f;
                        }
                        unit++;
                        kk = 0;
                    }
                }
            });
        }
        const int bn = nb, btotal = total;
        const bool more = b0 + p.batch < nu;
        if (more) open_batch(b0 + p.batch);
        if (b0 == 0) stamp(4);
        // the warps whose runs, [w total / runs, (w + 1) total / runs), meet the tiles of unit i
        int w0 = 0, w1 = 0;
        const int runs = min(btotal, GEMV_WARPS);
        auto holders = [&](int i) {
            w0 = (int)((unsigned)((i * kcs + 1) * runs - 1) / (unsigned)btotal);
            w1 = (int)((unsigned)((i + 1) * kcs * runs - 1) / (unsigned)btotal);
        };
        if (warp < bn * NG) holders(warp / NG);
        __syncthreads();  // the batch's pieces are there
        if (cluster) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        const int per_rank = (p.batch + S - 1) / S;                              // places for own units in `sums`
        const int own = slice < bn ? (bn - slice + S - 1) / S : 0;               // units whose row-tiles this rank stores
        if (cluster && own > 0 && threadIdx.x == 0) mbar_expect_tx(sums_bar, (uint32_t)(S * own * NG * 512));

        for (int it = warp; it < bn * NG; it += GEMV_WARPS) {
            const int i = it / NG, gi = it % NG;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int w = w0; w <= w1; w += 4) {  // four pieces in flight
                float4 a[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    a[j] = w + j <= w1 ? pieces[((size_t)(i + w + j) * NG + gi) * 32 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    v.x += a[j].x;
                    v.y += a[j].y;
                    v.z += a[j].z;
                    v.w += a[j].w;
                }
            }
            if (cluster) {
                const uint32_t to = smem_u32(sums + ((size_t)(slice * per_rank + i / S) * NG + gi) * 32 + lane);
                st_async_16(map_to_rank(to, (uint32_t)(i % S)), __float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z),
                            __float_as_uint(v.w), map_to_rank(sums_bar, (uint32_t)(i % S)));
            } else if (S > 1) {
                float4* const to = reinterpret_cast<float4*>(p.part) + (((size_t)(u0 + b0 + i) * S + slice) * pairs + 4 * gi + q) * 8 + g;
                if (4 * gi + q < pairs) __stcg(to, v);
            } else if (f32) {
                sums[((size_t)i * NG + gi) * 32 + lane] = v;
            } else {
                store_y(u0 + b0 + i, gi, v);
            }
            if (it + GEMV_WARPS < bn * NG) holders((it + GEMV_WARPS) / NG);
        }

        if (WAY == WAY_DIRECT) {
            // done
        } else if (S == 1 || cluster) {
            if (cluster) {
                if (own > 0) mbar_wait_or_abort(sums_bar, round & 1, abort32);
            } else if (f32) {
                __syncthreads();
            }
            if (f32) {  // columns 3t, 3t + 1, 3t + 2 are the hi / mid / lo parts of token t
                for (int e = threadIdx.x; e < own * p.m * 16; e += GEMV_CONSUMERS) {
                    const int row = e & 15, j = (e >> 4) / p.m, t = (e >> 4) - j * p.m, r = (u0 + b0 + slice + j * S) * 16 + row;
                    const int hi = place(3 * t, row), mid = place(3 * t + 1, row), lo = place(3 * t + 2, row);
                    float v = 0.f;
                    for (int s = 0; s < S; s++) {
                        const float* const f = reinterpret_cast<const float*>(sums + (size_t)(s * per_rank + j) * NG * 32);
                        v += (f[lo] + f[mid]) + f[hi];
                    }
                    if (r < p.w[0].rows) p.w[0].y[(int64_t)t * p.w[0].ldy + r] = v;
                }
            } else if (cluster) {
                for (int it = warp; it < own * NG; it += GEMV_WARPS) {
                    const int j = it / NG, gi = it % NG;
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int s = 0; s < S; s++) {
                        const float4 a = sums[((size_t)(s * per_rank + j) * NG + gi) * 32 + lane];
                        v.x += a.x;
                        v.y += a.y;
                        v.z += a.z;
                        v.w += a.w;
                    }
                    store_y(u0 + b0 + slice + j * S, gi, v);
                }
            }
        } else {
            // count the units in, list those that this CTA completed, then add their slices
            int* const listed = reinterpret_cast<int*>(smem + 24);
            __syncthreads();
            if (warp == 0) {
                int n = 0;
                for (int i = lane; i - lane < bn; i += 32) {
                    int old = 0, *const count = p.count + u0 + b0 + i;
                    if (i < bn) asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(old) : "l"(count) : "memory");
                    const bool last = i < bn && old == S - 1;
                    const unsigned all = __ballot_sync(0xFFFFFFFFu, last);
                    if (last) {
                        *count = 0;  // nobody else touches it again in this launch
                        smem[32 + n + __popc(all & ((1u << lane) - 1))] = (uint8_t)i;
                    }
                    n += __popc(all);
                }
                if (lane == 0) *listed = n;
            }
            __syncthreads();
            for (int e = threadIdx.x; e < *listed * p.m * 16; e += GEMV_CONSUMERS) {
                const int j = e / (p.m * 16), row = e & 15, t = (e - j * p.m * 16) >> 4, u = u0 + b0 + smem[32 + j];
                // [column pair][row & 7] float4 of {pair} x {row, row + 8}
                auto at = [&](int col) { return ((col >> 1) * 8 + (row & 7)) * 4 + (row >> 3) * 2 + (col & 1); };
                const float* const base = p.part + (size_t)u * S * pairs * 32;
                float v = 0.f;
#pragma unroll 4
                for (int s = 0; s < S; s++) {
                    const float* const f = base + (size_t)s * pairs * 32;
                    v += f32 ? (__ldcg(f + at(3 * t + 2)) + __ldcg(f + at(3 * t + 1))) + __ldcg(f + at(3 * t)) : __ldcg(f + at(t));
                }
                if (u * 16 + row < p.w[0].rows) p.w[0].y[(int64_t)t * p.w[0].ldy + u * 16 + row] = v;
            }
        }
        if (more) {  // this batch's pieces and sums are read
            __syncthreads();
            if (cluster) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        }
    }
    if (*reinterpret_cast<volatile int*>(smem + 8)) {  // a wait ran out: stay until the others' sums have landed
        if (lane == 0) report_status(p.status, STATUS_GEMV_FIXUP_TIMEOUT);
        if (cluster) {
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        }
        drain_after_abort();
    }
}

}  // namespace wf
