// compact.cu — stable active-particle compaction (compaction.wgsl:65-217,
// host src/gpu/compaction.rs:447-505).
//
// Over tiles of TILE = 2048 slots (256 threads x 8 slots):
//   1. count:   each warp ballots the active bit of 32 slots at a time and
//               sums popcounts; one count per tile;
//   2. index:   a tile's offset is the sum of the counts below it, and each
//               active slot's rank in the tile comes from ballots and a
//               prefix over the tile's warps, so the original order is kept;
//   3. move:    every field is gathered through the indices; every slot >=
//               active count receives its own old contents with the active
//               bit cleared (move_fields.cu).
// All FPG_FIELD_COUNT arrays move into a second structure-of-arrays block
// that is then swapped with the particle handle's (no copy back).
//
// HBM binds: 184 B of fields, 8 B of indices and 8 B of flags per slot.
// 5 M slots with 30 % dead: 175 us of kernels (360 us with a scatter whose
// stores followed their loads one field at a time).
#include <cuda_runtime.h>

#include <cstring>

#include "fpg_internal.h"
#include "move_fields.h"

namespace fpg {

void particles_swap_block(fpg_particles* p, void** other_block);
size_t particles_block_bytes(size_t capacity);
void particles_assign_fields(void* block, size_t capacity, void** field);

constexpr int CT_THREADS = 256;
constexpr int CT_ITEMS = 8;
constexpr int CT_TILE = CT_THREADS * CT_ITEMS;

// Per-tile active count.  Slot order inside a tile: item-major chunks of 256
// (chunk c covers slots tile*TILE + c*256 .. +255), warp w of the chunk
// covers 32 consecutive slots.
__global__ void __launch_bounds__(CT_THREADS) compact_count_kernel(const uint32_t* flags, uint32_t n,
                                                                   uint32_t* tile_counts) {
    chain_begin();
    __shared__ uint32_t s_warp[CT_THREADS / 32];
    const uint32_t tile = blockIdx.x;
    uint32_t local = 0;
#pragma unroll
    for (int c = 0; c < CT_ITEMS; ++c) {
        const uint32_t slot = tile * CT_TILE + c * CT_THREADS + threadIdx.x;
        const bool act = slot < n && (flags[slot] & 1u);
        local += __popc(__ballot_sync(0xffffffffu, act));
    }
    if ((threadIdx.x & 31u) == 0) s_warp[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < CT_THREADS / 32; ++w) t += s_warp[w];
        tile_counts[tile] = t;
    }
}

// Exclusive scan of the tile counts in one block of 1024 threads.
__global__ void __launch_bounds__(1024) compact_scan_kernel(uint32_t* tile_counts, uint32_t n_tiles) {
    chain_begin();
    __shared__ uint32_t s[1024];
    const uint32_t per = (n_tiles + 1023u) / 1024u;
    const uint32_t begin = threadIdx.x * per;
    const uint32_t end = min(begin + per, n_tiles);
    uint32_t sum = 0;
    for (uint32_t i = begin; i < end; ++i) sum += tile_counts[i];
    s[threadIdx.x] = sum;
    __syncthreads();
    for (uint32_t off = 1; off < 1024u; off <<= 1) {
        const uint32_t v = threadIdx.x >= off ? s[threadIdx.x - off] : 0u;
        __syncthreads();
        s[threadIdx.x] += v;
        __syncthreads();
    }
    uint32_t run = s[threadIdx.x] - sum;
    for (uint32_t i = begin; i < end; ++i) {
        const uint32_t v = tile_counts[i];
        tile_counts[i] = run;
        run += v;
    }
}

// The sum of one value per thread, on every thread.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* s_warp) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31u) == 0u) s_warp[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < CT_THREADS / 32; ++w) t += s_warp[w];
    return t;
}

// The original slot of each active particle, in slot order, and their number
// (to the device and to page-locked host memory).  `tiles` holds the tile
// counts, or with `scanned` their exclusive scan.  A CTA that gets the counts
// sums the ones below it itself: 20 KB from L2 per CTA at 10 M slots, about
// a microsecond beside the scan kernel's launch and its single block's
// 3.7 us; the sums grow with the square of the tiles, so above kSelfSumTiles
// (16.8 M slots, 32 KB a CTA) the scan kernel runs.
constexpr uint32_t kSelfSumTiles = 8192;

__global__ void __launch_bounds__(CT_THREADS) compact_index_kernel(const uint32_t* flags, uint32_t n,
                                                                   const uint32_t* tiles, int scanned,
                                                                   uint32_t* indices, uint32_t* active_dev,
                                                                   uint32_t* active_host) {
    chain_begin();
    constexpr int kWarps = CT_THREADS / 32;
    __shared__ uint32_t s_below[kWarps];
    __shared__ uint32_t s_pre[CT_ITEMS * kWarps];       // counts, then exclusive prefix, in slot order
    const uint32_t tile = blockIdx.x;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t below = 0;
    if (!scanned)
        for (uint32_t t = threadIdx.x; t < tile; t += CT_THREADS) below += tiles[t];
    unsigned ballots[CT_ITEMS];
#pragma unroll
    for (int c = 0; c < CT_ITEMS; ++c) {
        const uint32_t slot = tile * CT_TILE + c * CT_THREADS + threadIdx.x;
        ballots[c] = __ballot_sync(0xffffffffu, slot < n && (flags[slot] & 1u));
        if (lane == 0) s_pre[c * kWarps + warp] = __popc(ballots[c]);
    }
    const uint32_t base = scanned ? tiles[tile] : block_sum(below, s_below);
    __syncthreads();
    if (warp == 0) {
        // exclusive prefix of the 64 (chunk, warp) counts, two per lane
        static_assert(CT_ITEMS * kWarps == 64, "two counts per lane");
        const uint32_t a = s_pre[2u * lane], b = s_pre[2u * lane + 1u];
        uint32_t v = a + b;
#pragma unroll
        for (unsigned d = 1; d < 32u; d <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d) v += x;
        }
        s_pre[2u * lane] = v - a - b;
        s_pre[2u * lane + 1u] = v - b;
        if (lane == 31u && tile == gridDim.x - 1u) {
            *active_dev = base + v;
            *active_host = base + v;
        }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < CT_ITEMS; ++c)
        if (ballots[c] & (1u << lane))
            indices[base + s_pre[c * kWarps + warp] + __popc(ballots[c] & ((1u << lane) - 1u))] =
                tile * CT_TILE + c * CT_THREADS + threadIdx.x;
}

}  // namespace fpg

using namespace fpg;

extern "C" fpg_status fpg_compaction_create(fpg_ctx* ctx, size_t capacity, fpg_compaction** out) {
    if (!ctx || !out) return FPG_ERR_INVALID_ARGUMENT;
    if (capacity > (size_t)UINT32_MAX - CT_TILE) return FPG_ERR_VALUE_TOO_LARGE;
    fpg_compaction* c = new fpg_compaction();
    c->ctx = ctx;
    c->capacity = capacity;
    c->n_tiles = (capacity + CT_TILE - 1) / CT_TILE;
    cudaError_t e = cudaMalloc(&c->block, particles_block_bytes(capacity));
    if (e == cudaSuccess) e = cudaMalloc(&c->tile_counts, (c->n_tiles > 0 ? c->n_tiles : 1) * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&c->active_count_dev, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMallocHost(&c->active_count_host, sizeof(uint32_t));
    if (e != cudaSuccess) {
        cudaFree(c->block); cudaFree(c->tile_counts); cudaFree(c->active_count_dev);
        if (c->active_count_host) cudaFreeHost(c->active_count_host);
        delete c;
        return cuda_status(e);
    }
    *out = c;
    return FPG_OK;
}

extern "C" fpg_status fpg_compaction_destroy(fpg_compaction* c) {
    if (!c) return FPG_OK;
    cudaFree(c->block);
    cudaFree(c->tile_counts);
    cudaFree(c->active_count_dev);
    cudaFreeHost(c->active_count_host);
    delete c;
    return FPG_OK;
}

extern "C" fpg_status fpg_compact(fpg_ctx* ctx, fpg_particles* P, fpg_compaction* c, uint32_t* active_count,
                                  uint32_t* indices_dev, void* stream) {
    if (!ctx || !P || !c) return FPG_ERR_INVALID_ARGUMENT;
    if (c->capacity != P->capacity) return FPG_ERR_LENGTH_MISMATCH;
    const uint32_t n = (uint32_t)P->capacity;      // compaction.rs:454: all capacity slots
    if (n == 0) {
        if (active_count) *active_count = 0;
        return FPG_OK;
    }
    cudaStream_t s = ctx->pick(stream);
    void* dst[FPG_FIELD_COUNT];
    particles_assign_fields(c->block, c->capacity, dst);
    const uint32_t* flags = static_cast<const uint32_t*>(P->field[FPG_FIELD_FLAGS]);
    // without a buffer of the caller's the indices lie where the move writes last
    uint32_t* indices = indices_dev ? indices_dev : static_cast<uint32_t*>(dst[FPG_FIELD_COUNT - 1]);
    const uint32_t tiles = (uint32_t)c->n_tiles;
    const bool scan = tiles > kSelfSumTiles;
    launch_chained(compact_count_kernel, tiles, CT_THREADS, 0, s, flags, n, c->tile_counts);
    if (scan) launch_chained(compact_scan_kernel, 1, 1024, 0, s, c->tile_counts, tiles);
    launch_chained(compact_index_kernel, tiles, CT_THREADS, 0, s, flags, n, c->tile_counts, scan ? 1 : 0, indices, c->active_count_dev, c->active_count_host);
    ctx->count(scan ? 3 : 2);
    FPG_CHECK_LAUNCH();
    const fpg_status st = move_fields(ctx, P->field, dst, indices, 0, c->active_count_dev, n, true, s);
    if (st != FPG_OK) return st;
    FPG_CUDA(cudaStreamSynchronize(s));
    particles_swap_block(P, &c->block);
    const uint32_t act = *c->active_count_host;
    P->dispatch = act;                                 // timeloop.rs:1260
    if (active_count) *active_count = act;
    return FPG_OK;
}
