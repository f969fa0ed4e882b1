// Which way the gather behind a row-sharded projection takes.  Plain host arithmetic over values that are the same on every
// rank -- token count and type, rows of a shard, ranks, buffer sizes the ranks have agreed on -- because the routes wait for
// one another's words and flags: ranks that chose differently would wait for stores that nobody sends.  What a rank's own
// shard holds (values that only one of the local kernels can take) decides which kernel makes its block inside a route,
// never the route.
#pragma once
#include <stdint.h>

namespace wf {

// Token counts from which on the tensor cores are used.  bf16: more than one launch of the memory-bound decode kernel takes.
constexpr int GEMM_MIN_TOKENS_BF16 = 33, GEMM_MIN_TOKENS_F32 = 11;
inline bool many_tokens(bool x_f32, int64_t m) { return m >= (x_f32 ? GEMM_MIN_TOKENS_F32 : GEMM_MIN_TOKENS_BF16); }

enum GatherRoute {
    GATHER_STORES,  // tagged stores into the peers' landing buffers
    GATHER_LOADS,   // loads out of the peers' staging areas
    GATHER_NCCL
};
struct GatherRoom {
    bool peers;  // every rank has mapped every other rank's block
    int world;
    int64_t land_bytes, stage_bytes;
};
inline GatherRoute gather_route(const GatherRoom& room, bool x_f32, int64_t m, int64_t rows) {
    if (!room.peers || room.world < 2) return GATHER_NCCL;
    // few tokens: both halves of the landing buffer hold the gathered output as 8-byte words
    const int64_t words = (int64_t)room.world * m * rows;
    if (!many_tokens(x_f32, m) && words < (1ll << 31) && 2 * words * 8 <= room.land_bytes) return GATHER_STORES;
    // every rank's block fits its own staging area
    if (m * rows * 4 <= room.stage_bytes && words < (1ll << 40)) return GATHER_LOADS;
    return GATHER_NCCL;
}

}  // namespace wf
