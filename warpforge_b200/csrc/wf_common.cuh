// Internal declarations shared by the translation units of libwfb200.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <memory>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/wfb200.h"
#include "wf_layout.cuh"

namespace wf {

constexpr uint32_t CTX_MAGIC = 0x57464358;     // "WFCX"
constexpr uint32_t WEIGHT_MAGIC = 0x57465754;  // "WFWT"
constexpr uint32_t COMM_MAGIC = 0x5746434D;    // "WFCM"

// Device-side status bits, reported through Context::d_status by kernels that give up a wait (report_status).
constexpr int STATUS_GEMV_FIXUP_TIMEOUT = 1;
constexpr int STATUS_GEMM_PIPE_TIMEOUT = 2;
constexpr int STATUS_PEER_WAIT_TIMEOUT = 4;
constexpr int STATUS_BAD_INDEX = 8;  // an embedding index outside the table

__device__ __forceinline__ uint32_t map_to_rank(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
// 16 bytes into the shared memory of a CTA of the cluster; the bytes count on the barrier there when they have arrived
__device__ __forceinline__ void st_async_16(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t cluster_bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(cluster_addr), "r"(a), "r"(b),
                 "r"(c), "r"(d), "r"(cluster_bar)
                 : "memory");
}

// The status block: `bits` collects what kernels report (and is what running kernels look at); `host` is the device
// address of one int per bit in pinned host memory, set with it, so that the host learns the outcome of a stream it
// has waited for from its own memory.  Copying the bits back instead cost every synchronising call about 10 us.
struct StatusBlock {
    int bits;
    int pad;
    int* host;
};
constexpr int STATUS_BITS = 4;
#ifdef __CUDACC__
// Behind griddepcontrol.wait, what earlier kernels of the stream may still have been writing when this one was placed is read by
// plain loads through pointers that are not const __restrict__, or by these (of data that is read once): the non-coherent
// path, __ldg and what the compiler makes of const __restrict__, wants data that nobody writes while the kernel lives, and may be
// moved above the wait.  Volatile statements keep their order, plain loads do not pass a statement that clobbers memory.
__device__ __forceinline__ float ld_once(const float* p) {
    float v;
    asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_once(const float4* p) {
    float4 v;
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ void report_status(int* status, int bit) {
    StatusBlock* b = reinterpret_cast<StatusBlock*>(status);
    atomicOr(&b->bits, bit);
    *reinterpret_cast<volatile int*>(b->host + (31 - __clz(bit))) = 1;
    __threadfence_system();
}
// After an abort: give this CTA's asynchronous copies still in flight (its own, and those that other CTAs of its cluster have
// sent here) time to land before its shared memory is handed to another CTA (a few milliseconds at most).  Four instructions:
// what follows the last tile is fetched cold, and a loop of short pauses in its way cost small calls 1 %, a function call
// 0.3 us with fp32 tokens.
__device__ __forceinline__ void drain_after_abort() {
#pragma unroll
    for (int i = 0; i < 4; i++) __nanosleep(1000000);
}
#endif

constexpr int UPLOAD_RING = 6;  // pinned chunks

struct Context;

struct Weight {
    uint32_t magic = WEIGHT_MAGIC;
    Context* ctx = nullptr;
    WeightGeom g{};          // g.qtype is the DEVICE format (device_qtype of the file's type)
    int file_qtype = 0;      // ggml type of the blocks that were uploaded
    int64_t row0 = 0;        // first global row of this shard
    int64_t total_rows = 0;  // rows of the unsharded tensor
    uint8_t* d_tiles = nullptr;
    bool beyond_fp16 = false;  // some block may hold values outside fp16's range
    int64_t tiles_held = 0;  // bytes allocated at d_tiles (a reused buffer may be larger than g.bytes())
    int programs = 0;        // live programs whose op lists point at d_tiles
    // how the several-token decode kernel cuts this weight, per activation dtype (bf16 / fp32) and column count
    struct Split {
        short slices = -1;  // -1: not asked for yet, 0: no cut fits
        short kc = 0, batch = 0, ctas = 0;
        float ns = 0.f;  // the estimate
    } split_cache[2][33];
};

// Scratch of the kernels, one per stream that launches them (calls on different streams may overlap).  A recorded graph keeps
// a copy: its kernels hold these addresses however long it lives, whatever becomes of the stream it was recorded on and
// though a later call there may need more and put a larger buffer in the place of one.
struct GemvScratch {
    std::shared_ptr<uint2> d_slots;  // [ctas][128] {value bits, tag}
    std::shared_ptr<float> d_part;   // several-token kernel: partial sums of k-sliced launches
    std::shared_ptr<int> d_count;    // several-token kernel: arrival counters per row-tile
    int ctas = 0;
    // tensor-core GEMM
    std::shared_ptr<uint8_t> d_x16;         // fp16 copy of the activations
    int64_t x16_bytes = 0;
    std::shared_ptr<float> d_gemm_partial;  // [sm_count][256][128] pieces of tiles cut by a share boundary
    std::shared_ptr<unsigned int> d_gemm_ready;  // [sm_count][4] generation whose piece is complete, per 32-row quarter; then {generation, CTAs out}
};
// cudaMalloc for everything that a context allocates: where memory is short, its kept tile buffers go first.
cudaError_t device_alloc(Context* c, void** p, size_t bytes);
template <class T> inline cudaError_t device_alloc(Context* c, T** p, size_t bytes) { return device_alloc(c, reinterpret_cast<void**>(p), bytes); }
// Device memory that is freed with the last reference to it.
template <class T> inline cudaError_t make_shared_device(Context* c, std::shared_ptr<T>& p, size_t bytes) {
    void* q = nullptr;
    const cudaError_t e = device_alloc(c, &q, bytes);
    if (e == cudaSuccess) p.reset(static_cast<T*>(q), [](T* r) { cudaFree(r); });
    return e;
}

struct Context {
    uint32_t magic = CTX_MAGIC;
    int device = 0;
    int sm_count = 0;
    int cc_major = 0, cc_minor = 0;
    cudaStream_t stream = nullptr;  // the context's own compute stream
    int* d_status = nullptr;            // StatusBlock in device memory
    volatile int* h_status = nullptr;   // its host words, pinned; one more, set by the repack kernels (launch_repack)
    int* beyond_dev = nullptr;          // device address of that one
    int salt = 0;                            // instrumentation level, 2 = kernel timing stamps
    unsigned long long* d_timing = nullptr;  // [sm_count][8]
    std::mutex mu;  // guards against concurrent use (try_lock -> WF_ERR_BUSY)
    std::string last_error;
    std::vector<cudaStream_t> streams;
    std::vector<cudaEvent_t> events;
    std::vector<cudaGraphExec_t> graphs;
    int64_t capture_launches = 0;  // product kernels recorded by the capture in progress
    std::unordered_map<cudaGraphExec_t, int64_t> graph_launches;
    std::unordered_map<cudaGraphExec_t, GemvScratch> graph_scratch;  // of the stream it was recorded on
    std::unordered_map<int64_t, int64_t> allocs;  // device ptr -> bytes
    std::vector<void*> host_allocs;
    std::vector<Weight*> weights;
    struct SpareTiles {
        int64_t bytes;
        uint8_t* tiles;
    };
    std::vector<SpareTiles> spare_tiles;  // tile buffers of freed weights, oldest first, at most SPARE_TILES_BYTES in all
    int64_t spare_tiles_bytes = 0;
    bool foreign_streams = false;  // a stream that is not the context's own has been used: its work cannot be waited for by itself
    std::unordered_map<cudaStream_t, GemvScratch> gemv_scratch;
    // pinned staging for host-pointer calls
    void* h_stage = nullptr;
    void* h_stage_dev = nullptr;  // its address on the device
    int64_t h_stage_bytes = 0;
    void* d_stage = nullptr;
    int64_t d_stage_bytes = 0;
    void* h_upload = nullptr;  // ring of pinned chunks the weight upload streams a host tensor through
    void* d_upload = nullptr;  // their landing place on the device, read by the repack kernel
    int64_t upload_chunk_bytes = 0;
    cudaStream_t upload_stream = nullptr;
    cudaEvent_t upload_done[UPLOAD_RING] = {}, upload_repacked[UPLOAD_RING] = {};  // chunk transferred / its tiles written
    int64_t launches = 0;
    bool glue_exact = false;  // silu / softmax evaluate exp as the host does (double, one rounding) instead of expf
    int gemv_ctas_per_sm[3] = {0, 0, 0};
};

int set_error(Context* c, int status, const char* fmt, ...);
int cuda_status(Context* c, cudaError_t e, const char* what);
// Reads and clears the status after the stream has been waited for: WF_OK, or the failure a
// kernel recorded there (a bounded wait that ran out, an index outside a table).
int read_device_status(Context* c);
// WF_OK, or WF_ERR_RECORDING when `s` is being recorded into a graph: the caller is about to allocate (or
// grow) `what`, which a recording must not do -- recorded nodes would keep pointing at memory a later call
// frees.  Running the same call once before wf_graph_begin sizes everything.
int refuse_allocation_while_recording(Context* c, cudaStream_t s, const char* what);
Context* get_context(int64_t h);
Weight* get_weight(Context* c, int64_t h);
cudaStream_t resolve_stream(Context* c, int64_t stream);
cudaError_t take_tiles(Context* c, int64_t bytes, uint8_t** tiles, int64_t* held);
void release_spare_tiles(Context* c);
int ensure_stage(Context* c, int64_t host_bytes, int64_t dev_bytes);
// validated shard upload + repack shared by wf_weight_upload and wf_gguf_upload; takes the context lock
int weight_upload(Context* c, int qtype, const void* blocks, int64_t n_rows, int64_t k, int shard_rank, int shard_world,
                  int q4_0_order, int64_t* weight);

// wf_repack.cu
// *beyond (device address) is set to 1 when a block may hold values outside fp16's range
cudaError_t launch_repack(int qtype, const uint8_t* d_raw, uint8_t* d_tiles, int64_t rows, int64_t k,
                          int q4_0_order, int* beyond, cudaStream_t s);
cudaError_t launch_dequant_rows(const Weight& w, int64_t row0, int64_t nrows, float* d_out, cudaStream_t s);

// wf_gemv.cu
struct GemvCall {
    const Weight* w;
    const void* d_x;  // [m, k] bf16 or fp32
    int x_dtype;
    int64_t m;       // tokens, any value >= 1 (chunked internally)
    float* d_y;      // y[token * ldy + col0 + row]
    int64_t ldy;
    int64_t col0;
};
int gemv_launch(Context* c, const GemvCall& call, cudaStream_t s);
// what gemv_launch would refuse or allocate, without launching anything
int gemv_reserve(Context* c, const GemvCall& call, cudaStream_t s);
int gemv_max_tokens_per_pass(const Weight& w, int x_dtype);
int gemv_prepare_stream(Context* c, cudaStream_t s);
int gemv_launch_noalloc(Context* c, const GemvCall& call, cudaStream_t s);

// wf_gemm.cu
bool gemm_supported(const Weight& w, int x_dtype, int64_t m, const void* d_x);
int gemm_launch(Context* c, const GemvCall& call, cudaStream_t s);
// A projection by the kernel for its token count, wherever the result goes.  qlinear_reserve makes the scratch that
// qlinear_launch will use, or refuses the call, before anything is enqueued.
int qlinear_reserve(Context* c, const GemvCall& call, cudaStream_t s);
int qlinear_launch(Context* c, const GemvCall& call, cudaStream_t s);
// sizes the stream's scratch like the largest of the context's other streams (before a recording)
int gemm_prepare_stream(Context* c, cudaStream_t s);

struct ScopedLock {
    Context* c;
    bool ok;
    explicit ScopedLock(Context* ctx) : c(ctx), ok(ctx && ctx->mu.try_lock()) {}
    ~ScopedLock() {
        if (ok) c->mu.unlock();
    }
};

}  // namespace wf

#define WF_CUDA(c, call)                                         \
    do {                                                         \
        cudaError_t _e = (call);                                 \
        if (_e != cudaSuccess) return wf::cuda_status(c, _e, #call); \
    } while (0)
