// Building blocks of the tensor-core GEMM kernels: tcgen05 / TMA / mbarrier wrappers, the conversion of the activations, the
// epilogue's stores and the dequantization of weight tiles to fp16.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "wf_common.cuh"

namespace wf {

constexpr int GEMM_BN = 128;             // weight rows per CTA and tile (UMMA M per CTA)
constexpr int GEMM_BK = 128;             // k per unit of the work split
constexpr int GEMM_DEQUANT_WARPS = 8;    // of a set: a 16-row weight tile each
constexpr int GEMM_SETS = 2;             // sets, which take units by turns
constexpr int GEMM_THREADS = (6 + GEMM_SETS * GEMM_DEQUANT_WARPS) * 32;  // TMA, MMA, 4 epilogue, dequantization warps
constexpr int GEMM_WAIT_SPINS = 1 << 20;    // of an mbarrier wait, which suspends the thread for microseconds per try
constexpr int GEMM_POLL_SPINS = 1 << 22;    // of a poll of global memory
constexpr int GEMM_PIECE_TOKENS = 256;   // tokens a stream-K piece can hold

struct GemmParams {
    const uint8_t* tiles;
    float* y;
    const float* row_unscale;  // [m] power of two that undoes the scaling of token row m (convert_rows_kernel)
    int* status;
    int64_t ldy, col0;
    int rows, kt_w;      // kt_w: weight k-tiles per row-tile stripe (tile_k of the format)
    int rt_last;         // last row-tile in the weight buffer
    int m;               // tokens
    int bm;              // tokens of a tile (UMMA N: multiple of 16, pairs of 32, <= 256)
    int n_tiles, m_tiles, k_blocks;  // k_blocks = ceil(k / 128)
    int stages;          // split kernel
    int ranks;           // split kernel: CTAs of a cluster, which share a tile's K
    int early;           // split kernel: let the next kernel be placed while this one runs
    uint32_t idesc;
    // pair kernel: `waves` whole tiles a pair, then stream-K: the (tile, k-block) units behind form one sequence, pair b owns [b*q + min(b,r), ...)
    // split kernel: rank b owns those k-blocks of every tile, cluster c takes tile_q tiles, one more below tile_r
    int unit_q, unit_r, tile_q, tile_r, waves;
    float* partial;        // [ctas][GEMM_PIECE_TOKENS][128] fp32: a CTA's piece of a tile that begins in an earlier pair
    unsigned int* ready;   // [ctas][4] generation whose piece (per 32-row quarter) is complete in `partial`
    unsigned int* gen;     // [0] generations completed so far, [1] CTAs that have left the current launch: the kernel
                           // numbers its own launches, so a launch recorded in a CUDA graph is a new generation on every replay
                           // (read after griddepcontrol.wait, when the previous launch's closing store is visible)
};

// ---------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ uint32_t g_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void g_mbar_init(void* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(g_smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void g_mbar_arrive(void* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(g_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void g_mbar_expect_tx(void* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(g_smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool g_mbar_wait(void* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        ".reg .u32 n;\n\t"
        "mov.u32 n, 0;\n\t"
        "WFG_WAIT_%=:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra WFG_DONE_%=;\n\t"
        "add.u32 n, n, 1;\n\t"
        "setp.lt.u32 q, n, %3;\n\t"
        "@q bra WFG_WAIT_%=;\n\t"
        "WFG_DONE_%=:\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(g_smem_u32(bar)), "r"(parity), "r"((uint32_t)GEMM_WAIT_SPINS)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_id() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_count() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// Arrives on a barrier of another CTA of the cluster (its address there: map_to_rank).  Default semantics (release at CTA scope): weights that
// are handed over lie in the sender's TMEM, where tcgen05.wait::st has seen them arrive, and the fences before_thread_sync in front of the arrive
// and after_thread_sync behind the wait put the MMAs behind them; a TMA's data has landed when its own barrier says so; an exchange buffer that is given
// back has been read into registers.  `.release.cluster` costs a fence that waits for the thread's loads in flight, 0.9 us per stage.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, void* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            g_smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(g_smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tmem_alloc(void* smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(g_smem_u32(smem_dst)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(void* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(g_smem_u32(bar)) : "memory");
}
// One 64-k span of a tile: four MMAs of 16 k, A in TMEM (eight columns each), B 32 bytes (two descriptor units) apart in the swizzled
// rows.  Issued by the thread whose `issue` is non-zero; the whole warp comes here with the same operands, which therefore sit in
// uniform registers.  (Issued from a branch of one lane, every operand had to be moved there, and at about 200 cycles per MMA
// the issuing thread, not the tensor core with its 128, set the pace.)  accumulate: 0 = the first MMA starts from zero.
// With A in TMEM the tensor core reads only B from shared memory, and keeps its pace for any N from 32 on (cycles per MMA of 128 rows x 16 k, A in shared memory / in TMEM, measured: N = 16: 39 / 11, 48: 44 / 24,
// 96: 56 / 48, 128: 64 / 64).
template <int GROUP> __device__ __forceinline__ void tc_mma_span(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t issue) {
#define WF_MMA_SPAN(G)                                                                 \
    asm volatile(                                                                         \
        "{\n\t.reg .pred p, e, t;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"  \
        "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"      \
        "add.s32 a1, %1, 8;\n\tadd.s32 a2, %1, 16;\n\tadd.s32 a3, %1, 24;\n\t"            \
        "add.s64 b1, %2, 2;\n\tadd.s64 b2, %2, 4;\n\tadd.s64 b3, %2, 6;\n\t"              \
        "@e tcgen05.mma.cta_group::" G ".kind::f16 [%0], [%1], %2, %3, p;\n\t"           \
        "@e tcgen05.mma.cta_group::" G ".kind::f16 [%0], [a1], b1, %3, t;\n\t"           \
        "@e tcgen05.mma.cta_group::" G ".kind::f16 [%0], [a2], b2, %3, t;\n\t"           \
        "@e tcgen05.mma.cta_group::" G ".kind::f16 [%0], [a3], b3, %3, t;\n\t}" ::"r"(d_tmem), \
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(issue)                  \
        : "memory")
    if (GROUP == 1) WF_MMA_SPAN("1");
    else WF_MMA_SPAN("2");
#undef WF_MMA_SPAN
}
// 16 rows x 64 k of fp16 into 16 lanes x 32 columns of TMEM.  A lane holds rows g = lane / 4 (r0) and g + 8 (r1), of either 32-k block the
// eight elements 8 q .. 8 q + 7 (q = lane % 4): of each 16-byte piece the first half goes into the columns of one MMA, the
// second into those of the next (order of k: span_piece).
__device__ __forceinline__ void tmem_st_span(uint32_t taddr, const uint4& r0b0, const uint4& r0b1, const uint4& r1b0, const uint4& r1b1) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(r0b0.x), "r"(r0b0.y), "r"(r1b0.x), "r"(r1b0.y), "r"(r0b0.z), "r"(r0b0.w), "r"(r1b0.z), "r"(r1b0.w),
        "r"(r0b1.x), "r"(r0b1.y), "r"(r1b1.x), "r"(r1b1.y), "r"(r0b1.z), "r"(r0b1.w), "r"(r1b1.z), "r"(r1b1.w)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e;
}
__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u32(unsigned int* p, unsigned int v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Place in the ring of stages.  A consumer waits for parity `phase`, a producer for `phase ^ 1`: a barrier that has completed
// nothing yet lets the first lap pass.  (Stage and lap from a step count by division cost 50 of the 170 instructions of a
// dequantization step.)
struct StageCursor {
    int s = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ bool advance(int stages) {  // true at the start of a lap
        if (++s < stages) return false;
        s = 0;
        phase ^= 1;
        return true;
    }
};
// K-major operand, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);   // start address
    d |= (uint64_t)1 << 16;                    // leading byte offset (unused with swizzle), 16 B
    d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1 << 46;                    // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;                    // SWIZZLE_128B
    return d;
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// N columns of one accumulator (32), or of the sum of two that lie bm columns apart (16).
__device__ __forceinline__ void tmem_ld_accs(uint32_t taddr, int, uint32_t (&r)[32]) { tmem_ld32(taddr, r); }
__device__ __forceinline__ void tmem_ld_accs(uint32_t taddr, int bm, uint32_t (&r)[16]) {
    uint32_t e[16];
    tmem_ld16(taddr, r);
    tmem_ld16(taddr + (uint32_t)bm, e);
#pragma unroll
    for (int j = 0; j < 16; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(e[j]));
}

// ---------------------------------------------------------------- the order of k inside a span
// 64 k are four MMAs of 16.  What tmem_st_span does with the weights makes elements 8 q + 4 h .. + 3 of 32-k block j the q-th quarter of
// the 16 k of MMA 2 j + h, so a row of activations has them, as 8-byte pieces of its 128 bytes, at piece 4 (2 j + h) + q (the sum
// does not care).
__host__ __device__ inline int span_piece(int j, int q, int h) { return 4 * (2 * j + h) + q; }

// ---------------------------------------------------------------- activations to fp16
// x16 = fp16(x * 2^s) with s chosen so that the largest magnitude of the row lands in [2^14, 2^15), or 126
// where that would take more (magnitudes below 2^-112, down to subnormal ones); 2^-s undoes it behind the MMAs.
//   bf16 (PLANES 1): exact whenever the scaled value is a normal fp16.
//   fp32 (PLANES 3): v = hi + mid + lo, each the fp16 nearest to what is left: exact down to 2^-39 of the largest
//   (below that, what fp32 rounding leaves of a sum that the largest takes part in).
// Rows are padded to whole spans of 64 k (zeros) and lie in the spans' order of k.
template <int PLANES> struct RowGroup {  // eight elements of a row
    uint4 a, b;                          // b: fp32 only
    __device__ __forceinline__ void load(const void* row, int i) {
        const uint4* src = static_cast<const uint4*>(row) + (size_t)i * (PLANES == 1 ? 1 : 2);
        a = src[0];
        if (PLANES > 1) b = src[1];
    }
    // The largest magnitude so far: for bf16 of either half of the words, which is enough unless there is an Inf or a NaN (0x7F80
    // and up); for fp32 the bits of the largest exponent, Inf and NaN aside.
    __device__ __forceinline__ uint32_t largest(uint32_t m) const {
        if (PLANES == 1) return __vmaxu2(__vmaxu2(m, __vmaxu2(a.x & 0x7FFF7FFFu, a.y & 0x7FFF7FFFu)), __vmaxu2(a.z & 0x7FFF7FFFu, a.w & 0x7FFF7FFFu));
        return max(m, (uint32_t)exponent() << 23);
    }
    __device__ __forceinline__ int exponent() const {  // largest biased exponent; Inf and NaN do not drive the scale
        int e = 0;
        auto one = [&](uint32_t v) { e = max(e, v == 0xFFu ? 0 : (int)v); };
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < (PLANES == 1 ? 4 : 8); i++) {
            one((w[i] >> 23) & 0xFFu);
            if (PLANES == 1) one((w[i] >> 7) & 0xFFu);
        }
        return e;
    }
    // store(plane, eight fp16)
    template <class Store> __device__ __forceinline__ void convert(float scale, Store store) const {
        float f[8];
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            f[2 * e] = (PLANES == 1 ? __uint_as_float(w[e] << 16) : __uint_as_float(w[2 * e])) * scale;
            f[2 * e + 1] = (PLANES == 1 ? __uint_as_float(w[e] & 0xFFFF0000u) : __uint_as_float(w[2 * e + 1])) * scale;
        }
#pragma unroll
        for (int pl = 0; pl < PLANES; pl++) {
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const __half2 h = __floats2half2_rn(f[2 * e], f[2 * e + 1]);
                o[e] = *reinterpret_cast<const uint32_t*>(&h);
                if (pl + 1 < PLANES) {
                    const float2 back = __half22float2(h);
                    f[2 * e] -= back.x;
                    f[2 * e + 1] -= back.y;
                }
            }
            store(pl, make_uint4(o[0], o[1], o[2], o[3]));
        }
    }
};
// 2^s and 2^-s from the largest biased exponent; 2^126 is the largest power whose reciprocal is normal
__device__ __forceinline__ float2 row_scale(int emax) {
    const int shift = min((127 + 14) - emax, 126);
    return make_float2(__uint_as_float((uint32_t)(127 + shift) << 23), __uint_as_float((uint32_t)(127 - shift) << 23));
}

// One CTA per row.  A kernel of its own: the GEMM's CTAs set themselves up and dequantize their first stages under it.  Measured and
// not kept: converting inside the GEMM, every rank's warps their share of the rows, with tags to wait for: what a warp does for a
// row and then for the tags is a chain of trips to the L2, 4 us longer until the first MMA (77 tokens of [5003 x 2784]: 12.7 ->
// 14.4 us a call, 64 of [1000 x 1024]: 6.8 -> 9.8).
// KEEP: groups a thread keeps between the scan and the conversion; what is left of a longer row is read again.  Rows of up to 4096 elements:
// two, held to 32 registers a thread, so that eight rows and not five lie on an SM (with 46, us a call: Q4_K [1000 x 1024] 700 tokens 8.9 ->
// 10.4, [2048 x 2048] 128 tokens 8.5 -> 9.5, Q4_1 [4096 x 1024] 300 tokens 8.6 -> 9.3; 66 calls 0.996 x).  Longer rows: four, in 48 registers,
// whichever GEMM follows (155 calls of 33 - 700 tokens, K = 4608 - 11008, 0.952 x, worst 1.014: Q8_0 [1024 x 8192] 128 tokens 13.8 -> 11.4,
// Q4_0 [4096 x 11008] 96 tokens 19.9 -> 17.6).
constexpr int CONVERT_THREADS = 256;
constexpr int CONVERT_KEEP_SHORT = 2;  // rows of up to 4096 (bf16)
constexpr int CONVERT_KEEP_LONG = 4;   // up to 8192 held whole
template <int PLANES, int KEEP>
__global__ void __launch_bounds__(CONVERT_THREADS, PLANES == 1 && KEEP == CONVERT_KEEP_SHORT ? 8 : 5) convert_rows_kernel(const void* x, __half* __restrict__ x16, float* __restrict__ unscale,
                                                                       int m, int k) {
    __shared__ int s_max[CONVERT_THREADS / 32];
    // Launched with programmatic stream serialization itself: its CTAs may be placed while the previous kernel of the
    // stream drains, but nothing is read or written before that kernel has completed (it may have produced x, and a
    // previous GEMM may still be reading the fp16 copy this kernel rewrites).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the GEMM may set itself up while the rows are converted
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int groups = k >> 3, t = (int)threadIdx.x;  // k is a multiple of 32
    const int padded = (groups + 7) & ~7;             // groups of a row of x16
    const size_t plane = (size_t)m * padded;
    const int row = (int)blockIdx.x;
    const uint4* src = static_cast<const uint4*>(x) + (size_t)row * groups * (PLANES == 1 ? 1 : 2);
    RowGroup<PLANES> keep[KEEP], g;
    uint32_t mags = 0;
#pragma unroll
    for (int u = 0; u < KEEP; u++)
        if (t + u * CONVERT_THREADS < groups) keep[u].load(src, t + u * CONVERT_THREADS);
#pragma unroll
    for (int u = 0; u < KEEP; u++)
        if (t + u * CONVERT_THREADS < groups) mags = keep[u].largest(mags);
    for (int i = t + KEEP * CONVERT_THREADS; i < groups; i += CONVERT_THREADS) {
        g.load(src, i);
        mags = g.largest(mags);
    }
    int emax = PLANES == 1 ? max((int)(mags & 0xFFFFu) >> 7, (int)(mags >> 23)) : (int)(mags >> 23);
    if (PLANES == 1 && emax == 0xFF) {
        emax = 0;
#pragma unroll
        for (int u = 0; u < KEEP; u++)
            if (t + u * CONVERT_THREADS < groups) emax = max(emax, keep[u].exponent());
        for (int i = t + KEEP * CONVERT_THREADS; i < groups; i += CONVERT_THREADS) {
            g.load(src, i);
            emax = max(emax, g.exponent());
        }
    }
    emax = __reduce_max_sync(0xFFFFFFFFu, emax);
    if ((t & 31) == 0) s_max[t >> 5] = emax;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < CONVERT_THREADS / 32; w++) emax = max(emax, s_max[w]);
    const float2 scale = row_scale(emax);
    uint4* out = reinterpret_cast<uint4*>(x16) + (size_t)row * padded;
    auto store = [&](int pl, int i, const uint4& v) {  // group i of the row
        uint2* const span = reinterpret_cast<uint2*>(out + pl * plane + (i & ~7));
        const int j = (i >> 2) & 1, q = i & 3;
        span[span_piece(j, q, 0)] = make_uint2(v.x, v.y);
        span[span_piece(j, q, 1)] = make_uint2(v.z, v.w);
    };
    auto convert = [&](int i, const RowGroup<PLANES>& v) {
        v.convert(scale.x, [&](int pl, const uint4& o) { store(pl, i, o); });
    };
#pragma unroll
    for (int u = 0; u < KEEP; u++)
        if (t + u * CONVERT_THREADS < groups) convert(t + u * CONVERT_THREADS, keep[u]);
    for (int i = t + KEEP * CONVERT_THREADS; i < groups; i += CONVERT_THREADS) {
        g.load(src, i);
        convert(i, g);
    }
    if (t < padded - groups)  // the block that K lacks of its last stage
#pragma unroll
        for (int pl = 0; pl < PLANES; pl++) store(pl, groups + t, make_uint4(0u, 0u, 0u, 0u));
    if (t == 0) unscale[row] = scale.y;
}

// ---------------------------------------------------------------- epilogue pieces (one lane = one weight row)
// r[j] = accumulator of (token m0 + j, weight row n).  Rows of y are ldy floats apart; a warp writes 32
// consecutive floats of one token row per store.  m0 is a multiple of N, so the row scales load as float4.
template <int N> __device__ __forceinline__ void store_chunk(float* __restrict__ y, int64_t ldy, int64_t col0, const float* unscale,
                                            const uint32_t (&r)[N], int m0, int m, int n, int rows) {
    if (n >= rows || m0 >= m) return;
    float* yp = y + (int64_t)m0 * ldy + col0 + n;
    if (m0 + N <= m) {
        float sc[N];
#pragma unroll
        for (int i = 0; i < N / 4; i++) {
            const float4 v = reinterpret_cast<const float4*>(unscale + m0)[i];
            sc[4 * i] = v.x, sc[4 * i + 1] = v.y, sc[4 * i + 2] = v.z, sc[4 * i + 3] = v.w;
        }
#pragma unroll
        for (int j = 0; j < N; j++) yp[(int64_t)j * ldy] = __uint_as_float(r[j]) * sc[j];
    } else {
#pragma unroll
        for (int j = 0; j < N; j++)
            if (m0 + j < m) yp[(int64_t)j * ldy] = __uint_as_float(r[j]) * unscale[m0 + j];
    }
}
// A stream-K piece holds four tokens of a weight row in 16 bytes, [tokens / 4][128 rows]: a warp moves 512 contiguous
// bytes per access, eight accesses per 32 tokens (one float at a time the owner's tail read its pieces at a third of the
// speed: 8 - 11 us after the last MMA for 256 KB).
template <int N> __device__ __forceinline__ void write_piece_chunk(float* __restrict__ piece, const uint32_t (&r)[N], int tok, int row) {
    uint4* pp = reinterpret_cast<uint4*>(piece) + (size_t)(tok >> 2) * GEMM_BN + row;
#pragma unroll
    for (int j = 0; j < N / 4; j++) __stcg(pp + j * GEMM_BN, make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]));
}
template <int Q> __device__ __forceinline__ void load_piece_chunk(const float* __restrict__ piece, float4 (&v)[Q], int tok, int row) {
    const float4* pp = reinterpret_cast<const float4*>(piece) + (size_t)(tok >> 2) * GEMM_BN + row;
#pragma unroll
    for (int j = 0; j < Q; j++) v[j] = __ldcg(pp + j * GEMM_BN);
}
template <int N> __device__ __forceinline__ void add_piece_chunk(uint32_t (&r)[N], const float4 (&v)[N / 4]) {
#pragma unroll
    for (int j = 0; j < N / 4; j++) {
        r[4 * j] = __float_as_uint(__uint_as_float(r[4 * j]) + v[j].x);
        r[4 * j + 1] = __float_as_uint(__uint_as_float(r[4 * j + 1]) + v[j].y);
        r[4 * j + 2] = __float_as_uint(__uint_as_float(r[4 * j + 2]) + v[j].z);
        r[4 * j + 3] = __float_as_uint(__uint_as_float(r[4 * j + 3]) + v[j].w);
    }
}

// ---------------------------------------------------------------- dequantization to fp16
// A plane word holds the codes of 8 consecutive elements: rotated back by PLANE_ROT, nibble p of the
// low half is element 2p and nibble p of the high half element 2p + 1.  As fp16 bit patterns
//   (w & 0x000F000F) | 0x64006400  =  (1024 + e0, 1024 + e1)      codes in mantissa bits 3..0
//   (w & 0x00F000F0) | 0x54005400  =  (  64 + e2,   64 + e3)      codes in mantissa bits 7..4
// and the same two masks on the word rotated by a further 8 bits give elements 4..7.  Two rotates and
// four logic ops per 8 codes; everything after that runs on the half / float pipes.
struct Codes8 {
    uint32_t k[2];  // 1024 + code: elements (0,1), (4,5)
    uint32_t h[2];  // 64 + code:   elements (2,3), (6,7)
};
__device__ __forceinline__ Codes8 unpack8(uint32_t w) {
    const uint32_t a = __funnelshift_r(w, w, PLANE_ROT), b = __funnelshift_r(w, w, PLANE_ROT + 8);
    Codes8 c;
    c.k[0] = (a & 0x000F000Fu) | 0x64006400u;
    c.h[0] = (a & 0x00F000F0u) | 0x54005400u;
    c.k[1] = (b & 0x000F000Fu) | 0x64006400u;
    c.h[1] = (b & 0x00F000F0u) | 0x54005400u;
    return c;
}
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }

// Q4_0: s * (code - 8) with s an fp16 value.  code - 8 is exact in fp16 and the product is rounded
// once, exactly like the fp32 product rounded to fp16.
__device__ __forceinline__ uint4 word_to_half8_q4_0(uint32_t w, __half2 s2) {
    const Codes8 c = unpack8(w);
    const __half2 m1032 = __float2half2_rn(-1032.f), m72 = __float2half2_rn(-72.f);
    uint4 o;
    o.x = as_u32(__hmul2(__hadd2(as_half2(c.k[0]), m1032), s2));
    o.y = as_u32(__hmul2(__hadd2(as_half2(c.h[0]), m72), s2));
    o.z = as_u32(__hmul2(__hadd2(as_half2(c.k[1]), m1032), s2));
    o.w = as_u32(__hmul2(__hadd2(as_half2(c.h[1]), m72), s2));
    return o;
}
// What rounding left, as a second fp16: fma(code - 8, s, -rounded) is exact, a multiple of s's last place.
__device__ __forceinline__ void word_to_half8x2_q4_0(uint32_t w, __half2 s2, uint4& hi, uint4& lo) {
    const Codes8 c = unpack8(w);
    const __half2 m1032 = __float2half2_rn(-1032.f), m72 = __float2half2_rn(-72.f);
    auto two = [&](uint32_t code, __half2 off, uint32_t& h, uint32_t& l) {
        const __half2 q = __hadd2(as_half2(code), off), r = __hmul2(q, s2);
        h = as_u32(r);
        l = as_u32(__hfma2(q, s2, __hneg2(r)));
    };
    two(c.k[0], m1032, hi.x, lo.x);
    two(c.h[0], m72, hi.y, lo.y);
    two(c.k[1], m1032, hi.z, lo.z);
    two(c.h[1], m72, hi.w, lo.w);
}
// Q8_0: s * (byte - 128), byte = 16 hi + lo of the two planes' nibbles.  The halves of a byte are put side by side before anything is
// unpacked (bytes 0 and 2 of t0: elements 0, 1, bytes 1 and 3: 4, 5; t1: 2, 3 and 6, 7), and 0x64 above a byte makes it the fp16
// 1024 + byte.  byte - 128 is exact in fp16: one rounding, in the product.  18 operations per eight weights; unpacking either plane and joining
// the codes as fp16 took 24 ([11008 x 4096] 128 tokens 21.9 -> 19.1 us a call, [4096 x 4096] 512 tokens 24.2 -> 20.9, Q5_0 [5003 x 2784] 77
// tokens 11.2 -> 10.8).
struct Bytes8 {
    uint32_t t0, t1;
};
__device__ __forceinline__ Bytes8 bytes8(uint32_t wh, uint32_t wl) {
    auto join = [](uint32_t lo, uint32_t hi) { return (lo & 0x0F0F0F0Fu) | (hi & 0xF0F0F0F0u); };
    return {join(__funnelshift_r(wl, wl, PLANE_ROT), __funnelshift_r(wh, wh, PLANE_ROT + 28)),
            join(__funnelshift_r(wl, wl, PLANE_ROT + 4), __funnelshift_r(wh, wh, PLANE_ROT))};
}
template <int ODD> __device__ __forceinline__ __half2 q8_pair(uint32_t t) {
    return __hadd2(as_half2(__byte_perm(t, 0x64646464u, ODD ? 0x4341u : 0x4240u)), __float2half2_rn(-1152.f));
}
__device__ __forceinline__ uint4 words_to_half8_q8(uint32_t wh, uint32_t wl, __half2 s2) {
    const Bytes8 b = bytes8(wh, wl);
    return make_uint4(as_u32(__hmul2(q8_pair<0>(b.t0), s2)), as_u32(__hmul2(q8_pair<0>(b.t1), s2)), as_u32(__hmul2(q8_pair<1>(b.t0), s2)), as_u32(__hmul2(q8_pair<1>(b.t1), s2)));
}
__device__ __forceinline__ void words_to_half8x2_q8(uint32_t wh, uint32_t wl, __half2 s2, uint4& hi, uint4& lo) {
    const Bytes8 b = bytes8(wh, wl);
    auto two = [&](__half2 q, uint32_t& r, uint32_t& rest) {
        const __half2 v = __hmul2(q, s2);
        r = as_u32(v);
        rest = as_u32(__hfma2(q, s2, __hneg2(v)));
    };
    two(q8_pair<0>(b.t0), hi.x, lo.x);
    two(q8_pair<0>(b.t1), hi.y, lo.y);
    two(q8_pair<1>(b.t0), hi.z, lo.z);
    two(q8_pair<1>(b.t1), hi.w, lo.w);
}
// Q4_1 and Q4_K: a product of two fp16 plus an fp32 in fp32, rounded once to fp16.  The mixed-precision fma takes the codes as fp16:
// three operations a pair, where widening first took five (Q4_1 and Q4_K 26 -> 22 operations per eight weights; 33 - 2048 tokens of Q4_K
// 0.990 x the time).
__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t fma_pair(uint32_t h2, uint32_t s, float c) {  // s: an fp16 in the low half
    float x, y;
    asm("{\n\t.reg .b16 l, h, s, u;\n\t"
        "mov.b32 {l, h}, %2;\n\tmov.b32 {s, u}, %3;\n\t"
        "fma.rn.f32.f16 %0, l, s, %4;\n\tfma.rn.f32.f16 %1, h, s, %4;\n\t}"
        : "=f"(x), "=f"(y)
        : "r"(h2), "r"(s), "f"(c));
    return pack_half2(x, y);
}
// Q4_1: scale * code + min.  The 1024 or 64 that the unpacked code carries is taken off in fp16, exactly; taken off as a multiple of the
// scale inside the min, it cost up to 2^-14 of the scale, which a min of 2^-8 of the scale shows in its sixth bit, and made
// every weight of a block whose scale is Inf a NaN ([11008 x 4096], 33 tokens: 17.6 us so, 17.2 now; [8192 x 8192], 1024: 105.7, 105.5).
__device__ __forceinline__ uint4 word_to_half8_q4_1(uint32_t w, uint32_t s, float m) {
    const Codes8 c = unpack8(w);
    auto code = [](uint32_t v, float off) { return as_u32(__hadd2(as_half2(v), __float2half2_rn(off))); };
    return make_uint4(fma_pair(code(c.k[0], -1024.f), s, m), fma_pair(code(c.h[0], -64.f), s, m), fma_pair(code(c.k[1], -1024.f), s, m), fma_pair(code(c.h[1], -64.f), s, m));
}
// Q4_K: d * (sc * code) + b, b = -dmin * m: sc * code, at most 945, is exact in fp16
__device__ __forceinline__ uint4 word_to_half8_q4_k(uint32_t w, __half2 sc, uint32_t d, float b) {
    const Codes8 c = unpack8(w);
    const __half2 ok = __hmul2(sc, __float2half2_rn(-1024.f)), oh = __hmul2(sc, __float2half2_rn(-64.f));
    auto times = [&](uint32_t code, __half2 off) { return as_u32(__hfma2(as_half2(code), sc, off)); };
    return make_uint4(fma_pair(times(c.k[0], ok), d, b), fma_pair(times(c.h[0], oh), d, b), fma_pair(times(c.k[1], ok), d, b), fma_pair(times(c.h[1], oh), d, b));
}

// The same as two fp16: 22 of the fp32 value's 24 bits (it is a multiple of 2^-24, as its fp16 factors are).
__device__ __forceinline__ void word_to_half8x2(uint32_t w, float a, float b, uint4& hi, uint4& lo) {
    const Codes8 c = unpack8(w);
    auto two = [&](uint32_t code, float off, uint32_t& h, uint32_t& l) {  // code - off is exact
        const float2 f = __half22float2(__hadd2(as_half2(code), __float2half2_rn(off)));
        const float v0 = fmaf(a, f.x, b), v1 = fmaf(a, f.y, b);
        const __half2 r = __floats2half2_rn(v0, v1);
        const float2 back = __half22float2(r);
        h = as_u32(r);
        l = pack_half2(v0 - back.x, v1 - back.y);
    };
    two(c.k[0], -1024.f, hi.x, lo.x);
    two(c.h[0], -64.f, hi.y, lo.y);
    two(c.k[1], -1024.f, hi.z, lo.z);
    two(c.h[1], -64.f, hi.w, lo.w);
}

// byte `i` of w times d, exactly: (2^23 + byte) * d - 2^23 * d
__device__ __forceinline__ float byte_of(uint32_t w, uint32_t sel, float d, float neg_big_d) {
    return fmaf(__uint_as_float(__byte_perm(w, 0x4B000000u, sel)), d, neg_big_d);
}

// What a lane holds of 8 + 8 rows x 128 k of a weight tile: for row half h (rows g = lane / 4 and g + 8) the words of
// its element group (8 q .. 8 q + 7, q = lane & 3) in the four 32-k blocks, and those blocks' scales.  load() reads
// them straight from global memory (16-byte pieces, the layout is fragment-ordered); pair<SUB>() converts blocks
// 2 SUB and 2 SUB + 1 to fp16, one 16-byte chunk of the stage's row each.
template <int QT> struct DequantRegs;

template <> struct DequantRegs<WF_QTYPE_Q4_0> {
    uint4 c;
    uint2 sc;  // fp16 scales of blocks (0, 1), (2, 3)
    __device__ __forceinline__ void load(const uint8_t* tile, int, int lane, int h) {
        c = __ldg(reinterpret_cast<const uint4*>(tile + h * 512 + lane * 16));
        sc = __ldg(reinterpret_cast<const uint2*>(tile + Tile<WF_QTYPE_Q4_0>::SCALE_OFF + (lane >> 2) * 16 + h * 8));
    }
    template <int SUB> __device__ __forceinline__ void pair(uint4& o0, uint4& o1) const {
        const uint32_t w0 = SUB ? c.z : c.x, w1 = SUB ? c.w : c.y, s = SUB ? sc.y : sc.x;
        const __half2 sx = as_half2(__byte_perm(s, s, 0x1010u)), sy = as_half2(__byte_perm(s, s, 0x3232u));
        o0 = word_to_half8_q4_0(w0, sx);
        o1 = word_to_half8_q4_0(w1, sy);
    }
};

template <> struct DequantRegs<WF_QTYPE_Q4_1> {
    uint4 c;
    uint2 sc, mn;
    __device__ __forceinline__ void load(const uint8_t* tile, int, int lane, int h) {
        using T = Tile<WF_QTYPE_Q4_1>;
        c = __ldg(reinterpret_cast<const uint4*>(tile + h * 512 + lane * 16));
        sc = __ldg(reinterpret_cast<const uint2*>(tile + T::SCALE_OFF + (lane >> 2) * 16 + h * 8));
        mn = __ldg(reinterpret_cast<const uint2*>(tile + T::MIN_OFF + (lane >> 2) * 16 + h * 8));
    }
    template <int SUB> __device__ __forceinline__ void pair(uint4& o0, uint4& o1) const {  // scale * code + min in fp32, rounded once
        const uint32_t w0 = SUB ? c.z : c.x, w1 = SUB ? c.w : c.y;
        const uint32_t s = SUB ? sc.y : sc.x;
        const float2 m = __half22float2(as_half2(SUB ? mn.y : mn.x));
        o0 = word_to_half8_q4_1(w0, s, m.x);
        o1 = word_to_half8_q4_1(w1, s >> 16, m.y);
    }
};

template <> struct DequantRegs<WF_QTYPE_Q8_0> {
    uint4 ch, cl;
    uint2 sc;
    __device__ __forceinline__ void load(const uint8_t* tile, int, int lane, int h) {
        ch = __ldg(reinterpret_cast<const uint4*>(tile + h * 512 + lane * 16));
        cl = __ldg(reinterpret_cast<const uint4*>(tile + PLANE_BYTES + h * 512 + lane * 16));
        sc = __ldg(reinterpret_cast<const uint2*>(tile + Tile<WF_QTYPE_Q8_0>::SCALE_OFF + (lane >> 2) * 16 + h * 8));
    }
    template <int SUB> __device__ __forceinline__ void pair(uint4& o0, uint4& o1) const {
        const uint32_t h0 = SUB ? ch.z : ch.x, h1 = SUB ? ch.w : ch.y, l0 = SUB ? cl.z : cl.x, l1 = SUB ? cl.w : cl.y, s = SUB ? sc.y : sc.x;
        const __half2 sx = as_half2(__byte_perm(s, s, 0x1010u)), sy = as_half2(__byte_perm(s, s, 0x3232u));
        o0 = words_to_half8_q8(h0, l0, sx);
        o1 = words_to_half8_q8(h1, l1, sy);
    }
};

template <> struct DequantRegs<WF_QTYPE_Q4_K> {  // one half (plane kb & 1) of a 256-k tile
    uint4 c;
    uint32_t dd, scw, mnw;  // (d, dmin); 8-bit scales / mins of the half's four sub-blocks
    __device__ __forceinline__ void load(const uint8_t* tile, int plane, int lane, int h) {
        using T = Tile<WF_QTYPE_Q4_K>;
        const int g = lane >> 2;
        c = __ldg(reinterpret_cast<const uint4*>(tile + plane * PLANE_BYTES + h * 512 + lane * 16));
        dd = __ldg(reinterpret_cast<const uint32_t*>(tile + T::D_OFF + g * 8 + h * 4));
        scw = __ldg(reinterpret_cast<const uint32_t*>(tile + T::SC_OFF + g * 16 + h * 8 + plane * 4));
        mnw = __ldg(reinterpret_cast<const uint32_t*>(tile + T::MN_OFF + g * 16 + h * 8 + plane * 4));
    }
    template <int SUB> __device__ __forceinline__ void pair(uint4& o0, uint4& o1) const {  // (d * sc) * code - dmin * m
        const float dmin = __high2float(as_half2(dd)), nm = 8388608.f * dmin;
        const uint32_t w0 = SUB ? c.z : c.x, w1 = SUB ? c.w : c.y;
        const uint32_t first = 0x7540u + 2 * SUB, second = first + 1;
        auto scale = [&](uint32_t i) { return __hadd2(as_half2(__byte_perm(scw, 0x64646464u, 0x4040u + 0x0101u * i)), __float2half2_rn(-1024.f)); };  // byte i, twice
        o0 = word_to_half8_q4_k(w0, scale(2 * SUB), dd, byte_of(mnw, first, -dmin, nm));
        o1 = word_to_half8_q4_k(w1, scale(2 * SUB + 1), dd, byte_of(mnw, second, -dmin, nm));
    }
};

// The same of one stage alone, blocks 2 sub and 2 sub + 1, which pair2() converts to two fp16 per weight.
template <int QT> struct DequantHalf;

template <> struct DequantHalf<WF_QTYPE_Q4_0> {
    uint2 c;
    uint32_t sc;
    __device__ __forceinline__ void load(const uint8_t* tile, int, int sub, int lane, int h) {
        c = __ldg(reinterpret_cast<const uint2*>(tile + h * 512 + lane * 16 + sub * 8));
        sc = __ldg(reinterpret_cast<const uint32_t*>(tile + Tile<WF_QTYPE_Q4_0>::SCALE_OFF + (lane >> 2) * 16 + h * 8 + sub * 4));
    }
    __device__ __forceinline__ void pair2(uint4& h0, uint4& h1, uint4& l0, uint4& l1) const {
        word_to_half8x2_q4_0(c.x, as_half2(__byte_perm(sc, sc, 0x1010u)), h0, l0);
        word_to_half8x2_q4_0(c.y, as_half2(__byte_perm(sc, sc, 0x3232u)), h1, l1);
    }
};

template <> struct DequantHalf<WF_QTYPE_Q4_1> {
    uint2 c;
    uint32_t sc, mn;
    __device__ __forceinline__ void load(const uint8_t* tile, int, int sub, int lane, int h) {
        using T = Tile<WF_QTYPE_Q4_1>;
        c = __ldg(reinterpret_cast<const uint2*>(tile + h * 512 + lane * 16 + sub * 8));
        sc = __ldg(reinterpret_cast<const uint32_t*>(tile + T::SCALE_OFF + (lane >> 2) * 16 + h * 8 + sub * 4));
        mn = __ldg(reinterpret_cast<const uint32_t*>(tile + T::MIN_OFF + (lane >> 2) * 16 + h * 8 + sub * 4));
    }
    __device__ __forceinline__ void pair2(uint4& h0, uint4& h1, uint4& l0, uint4& l1) const {
        const float2 s = __half22float2(as_half2(sc)), m = __half22float2(as_half2(mn));
        word_to_half8x2(c.x, s.x, m.x, h0, l0);
        word_to_half8x2(c.y, s.y, m.y, h1, l1);
    }
};

template <> struct DequantHalf<WF_QTYPE_Q8_0> {
    uint2 ch, cl;
    uint32_t sc;
    __device__ __forceinline__ void load(const uint8_t* tile, int, int sub, int lane, int h) {
        ch = __ldg(reinterpret_cast<const uint2*>(tile + h * 512 + lane * 16 + sub * 8));
        cl = __ldg(reinterpret_cast<const uint2*>(tile + PLANE_BYTES + h * 512 + lane * 16 + sub * 8));
        sc = __ldg(reinterpret_cast<const uint32_t*>(tile + Tile<WF_QTYPE_Q8_0>::SCALE_OFF + (lane >> 2) * 16 + h * 8 + sub * 4));
    }
    __device__ __forceinline__ void pair2(uint4& h0, uint4& h1, uint4& l0, uint4& l1) const {
        words_to_half8x2_q8(ch.x, cl.x, as_half2(__byte_perm(sc, sc, 0x1010u)), h0, l0);
        words_to_half8x2_q8(ch.y, cl.y, as_half2(__byte_perm(sc, sc, 0x3232u)), h1, l1);
    }
};

template <> struct DequantHalf<WF_QTYPE_Q4_K> {
    uint2 c;
    uint32_t dd, scw, mnw;  // (d, dmin); 8-bit scales / mins of the stage's two sub-blocks
    __device__ __forceinline__ void load(const uint8_t* tile, int plane, int sub, int lane, int h) {
        using T = Tile<WF_QTYPE_Q4_K>;
        const int g = lane >> 2;
        c = __ldg(reinterpret_cast<const uint2*>(tile + plane * PLANE_BYTES + h * 512 + lane * 16 + sub * 8));
        dd = __ldg(reinterpret_cast<const uint32_t*>(tile + T::D_OFF + g * 8 + h * 4));
        scw = __ldg(reinterpret_cast<const uint16_t*>(tile + T::SC_OFF + g * 16 + h * 8 + plane * 4 + sub * 2));
        mnw = __ldg(reinterpret_cast<const uint16_t*>(tile + T::MN_OFF + g * 16 + h * 8 + plane * 4 + sub * 2));
    }
    __device__ __forceinline__ void pair2(uint4& h0, uint4& h1, uint4& l0, uint4& l1) const {
        const float2 d = __half22float2(as_half2(dd));
        const float nd = -8388608.f * d.x, nm = 8388608.f * d.y;
        word_to_half8x2(c.x, byte_of(scw, 0x7540u, d.x, nd), byte_of(mnw, 0x7540u, -d.y, nm), h0, l0);
        word_to_half8x2(c.y, byte_of(scw, 0x7541u, d.x, nd), byte_of(mnw, 0x7541u, -d.y, nm), h1, l1);
    }
};

}  // namespace wf
