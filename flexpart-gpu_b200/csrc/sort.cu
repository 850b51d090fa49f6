// sort.cu — reorder particles by met cell.
//
// The reference can reorder its particle store on the host by a Morton key
// of the quantised position every few steps (ParticleStore::sort_spatially,
// src/particles/mod.rs:649-699, applied by apply_spatial_sort_if_enabled,
// src/simulation/timeloop.rs:1414-1430) so that neighbouring slots sample
// neighbouring met.  Here the key is the 3-D met cell the particle sits in,
// ((ix*ny)+iy)*nz+iz with ix, iy, iz the lower corner indices the trilinear
// sample of the fused step uses, so a warp's 32 particles mostly share their
// 8 corner nodes (broadcast gathers) and their PBL cell (one stability
// regime, no divergence).  Inactive slots get key 0xFFFFFFFF and move to the
// end, as the reference's INACTIVE_MORTON_KEY does (particles/mod.rs:27);
// on the device that key is nx*ny*nz (one past the last cell) so the radix
// sort only runs over the bits the cell count needs.
//
// Steps: the keys with the first digit's tile histograms -> a stable LSD radix
// sort of (key, slot) pairs by 8-bit digits -> gather of all FPG_FIELD_COUNT
// arrays into a second structure-of-arrays block, which is swapped in.
// A digit pass is a histogram per tile of 4096 pairs, a scan of each bin over
// the tiles, and a scatter that ranks the tile's pairs (warp match and warp
// counters, in order), sorts them in shared memory and writes each bin's run.
// No kernel waits for another CTA; the first pass reads no slots (they are
// the positions), the last writes no keys.  HBM traffic of three passes: 76 B
// a slot with the keys; the ranking's shared-memory chain binds it, half of
// the issue slots used (512 threads x 8 pairs with 64 registers; 40 of them
// spill).  Against the key kernel and a library radix sort, whose host calls
// alone took 60 us: a step and its reorder 716 -> 677 us at 6 M slots, 97 ->
// 70 us at 300 k, 64 -> 42 us at 10 k.
// Philox streams follow the slot, as in the reference after its sort.
#include <cuda_runtime.h>

#include <algorithm>

#include "fpg_internal.h"
#include "move_fields.h"
#include "physics.cuh"
#include "step_core.cuh"

struct fpg_sorter {
    fpg_ctx* ctx = nullptr;
    size_t capacity = 0;
    uint32_t* keys[2] = {};
    uint32_t* vals[2] = {};
    uint32_t* hist = nullptr;               // kBins x tiles: tile histograms, then their offsets in the bin
    uint32_t* bin_total = nullptr;          // kBins
    void* block = nullptr;
};

namespace fpg {

void particles_swap_block(fpg_particles* p, void** other_block);
size_t particles_block_bytes(size_t capacity);
void particles_assign_fields(void* block, size_t capacity, void** field);

struct KeyArgs {
    const int32_t* cell_x; const int32_t* cell_y; const float* pos_x; const float* pos_y; const float* pos_z;
    const uint32_t* flags;
    Levels lv;
    uint32_t n, nx, ny, nz;
};

// Same lower-corner arithmetic as the fused step (axis_bracket and
// meters_to_level, advection_dual_wind.wgsl:94-138).
__device__ __forceinline__ uint32_t lower_index(float coord, uint32_t n) {
    return (uint32_t)floorf(clampf(coord, 0.0f, (float)(n - 1u)));
}

// lower_index(meters_to_level(z)): the level (k - 1) + (z - h[k-1]) / (h[k] -
// h[k-1]) has lower corner k - 1 unless the quotient rounds up to 1, so the
// IEEE division runs only for the last hundredth of a layer (k <= 256: a
// float sum below k - 0.0099 cannot round to k).
__device__ __forceinline__ uint32_t lower_level(const Levels& lv, float z) {
    if (!lv.has) return lower_index(z, lv.nz);
    const float h0 = lv.h[0];
    if (z <= h0) return lower_index(h0 > 0.0f ? z / h0 : 0.0f, lv.nz);
    const uint32_t k = level_index(lv, z);
    if (k >= lv.nz) return lv.nz - 1u;
    const float hprev = lv.h[k - 1u];
    const float denom = lv.h[k] - hprev, above = z - hprev;
    if (!(denom > 0.0f) || above < 0.99f * denom) return k - 1u;
    return lower_index((float)(k - 1u) + above / denom, lv.nz);
}

__device__ __forceinline__ uint32_t cell_key(const KeyArgs& a, uint32_t flags, int32_t cx, int32_t cy, float px,
                                             float py, float z) {
    if (!(flags & FLAG_ACTIVE)) return a.nx * a.ny * a.nz;
    const uint32_t ix = lower_index((float)cx + px, a.nx), iy = lower_index((float)cy + py, a.ny);
    return (ix * a.ny + iy) * a.nz + lower_level(a.lv, z);
}

constexpr uint32_t kDigitBits = 8, kBins = 1u << kDigitBits;
constexpr uint32_t kSortThreads = 512, kSortWarps = kSortThreads / 32;
constexpr uint32_t kSortItems = 8;                                    // pairs per thread
constexpr uint32_t kScanThreads = 256;
constexpr uint32_t kSortTile = kSortThreads * kSortItems;             // 4096

__device__ __forceinline__ uint32_t digit_of(uint32_t key, uint32_t shift) { return (key >> shift) & (kBins - 1u); }

// Adds a warp's digits to the CTA's histogram: one shared atomic per distinct
// digit of the warp (neighbouring slots share most of their digits).
__device__ __forceinline__ void histogram_add(uint32_t* s_hist, uint32_t digit, bool valid) {
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? digit : kBins);
    if (valid && (threadIdx.x & 31u) == (unsigned)(__ffs(peers) - 1)) atomicAdd(s_hist + digit, (uint32_t)__popc(peers));
}

// The keys of a tile, two adjacent slots per thread and pass with 8-byte
// accesses, every load issued before the flags are looked at, the level found
// by the met's bucket table through L1; and the tile's histogram of the first
// digit.  28 B a slot, HBM-bound.
__global__ void __launch_bounds__(kSortThreads) cell_key_kernel(KeyArgs a, uint32_t* keys, uint32_t* hist, uint32_t tiles) {
    chain_begin();
    __shared__ uint32_t s_hist[kBins];
    if (threadIdx.x < kBins) s_hist[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t base = blockIdx.x * kSortTile;
#pragma unroll 2
    for (uint32_t k = 0; k < kSortItems / 2u; ++k) {
        const uint32_t p = base + 2u * (k * kSortThreads + threadIdx.x);
        uint32_t k0 = 0u, k1 = 0u;
        if (p + 1u < a.n) {
            const uint2 f = *reinterpret_cast<const uint2*>(a.flags + p);
            const int2 cx = *reinterpret_cast<const int2*>(a.cell_x + p);
            const int2 cy = *reinterpret_cast<const int2*>(a.cell_y + p);
            const float2 px = *reinterpret_cast<const float2*>(a.pos_x + p);
            const float2 py = *reinterpret_cast<const float2*>(a.pos_y + p);
            const float2 z = *reinterpret_cast<const float2*>(a.pos_z + p);
            k0 = cell_key(a, f.x, cx.x, cy.x, px.x, py.x, z.x);
            k1 = cell_key(a, f.y, cx.y, cy.y, px.y, py.y, z.y);
            *reinterpret_cast<uint2*>(keys + p) = make_uint2(k0, k1);
        } else if (p < a.n) {
            k0 = cell_key(a, a.flags[p], a.cell_x[p], a.cell_y[p], a.pos_x[p], a.pos_y[p], a.pos_z[p]);
            keys[p] = k0;
        }
        histogram_add(s_hist, digit_of(k0, 0u), p < a.n);
        histogram_add(s_hist, digit_of(k1, 0u), p + 1u < a.n);
    }
    __syncthreads();
    if (threadIdx.x < kBins) hist[(size_t)threadIdx.x * tiles + blockIdx.x] = s_hist[threadIdx.x];
}

__global__ void __launch_bounds__(kSortThreads) digit_histogram_kernel(const uint32_t* keys, uint32_t n, uint32_t shift,
                                                                       uint32_t* hist, uint32_t tiles) {
    chain_begin();
    __shared__ uint32_t s_hist[kBins];
    if (threadIdx.x < kBins) s_hist[threadIdx.x] = 0u;
    __syncthreads();
    const uint32_t base = blockIdx.x * kSortTile;
    uint32_t key[kSortItems];
#pragma unroll
    for (uint32_t k = 0; k < kSortItems; ++k) {
        const uint32_t p = base + k * kSortThreads + threadIdx.x;
        if (p < n) key[k] = keys[p];
    }
#pragma unroll
    for (uint32_t k = 0; k < kSortItems; ++k)
        histogram_add(s_hist, digit_of(key[k], shift), base + k * kSortThreads + threadIdx.x < n);
    __syncthreads();
    if (threadIdx.x < kBins) hist[(size_t)threadIdx.x * tiles + blockIdx.x] = s_hist[threadIdx.x];
}

// Exclusive scan of each bin's counts over the tiles, one CTA per bin, and
// the bin's total.
__global__ void __launch_bounds__(kScanThreads) bin_scan_kernel(uint32_t* hist, uint32_t tiles, uint32_t* bin_total) {
    chain_begin();
    __shared__ uint32_t s_warp[(kScanThreads / 32)];
    uint32_t* row = hist + (size_t)blockIdx.x * tiles;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t carry = 0u;
    for (uint32_t base = 0; base < tiles; base += kScanThreads) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t v = i < tiles ? row[i] : 0u;
        uint32_t x = v;
#pragma unroll
        for (unsigned d = 1; d < 32u; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31u) s_warp[warp] = x;
        __syncthreads();
        uint32_t before = carry, total = 0u;
#pragma unroll
        for (unsigned w = 0; w < (kScanThreads / 32); ++w) {
            if (w < warp) before += s_warp[w];
            total += s_warp[w];
        }
        if (i < tiles) row[i] = before + x - v;
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) bin_total[blockIdx.x] = carry;
}

// Exclusive scan of one value per thread over the CTA.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* s_warp) {
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (unsigned d = 1; d < 32u; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31u) s_warp[warp] = x;
    __syncthreads();
    uint32_t before = 0u;
#pragma unroll
    for (unsigned w = 0; w < kSortWarps; ++w)
        if (w < warp) before += s_warp[w];
    __syncthreads();
    return before + x - v;
}

// One digit's stable scatter.  vals_in NULL: the slots are the positions;
// keys_out NULL: the keys are not needed any more.
__global__ void __launch_bounds__(kSortThreads, 2) digit_scatter_kernel(const uint32_t* keys_in, const uint32_t* vals_in,
                                                                     uint32_t n, uint32_t shift, const uint32_t* hist,
                                                                     const uint32_t* bin_total, uint32_t tiles,
                                                                     uint32_t* keys_out, uint32_t* vals_out) {
    chain_begin();
    __shared__ uint32_t s_key[kSortTile], s_val[kSortTile];
    __shared__ __align__(4) uint16_t s_rank[kSortWarps][kBins];          // counts per warp, then the warp's first position
    __shared__ uint32_t s_global[kBins];                    // a bin's output position minus its position in the tile
    __shared__ uint32_t s_warp[kSortWarps];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t base = blockIdx.x * kSortTile, count = min(kSortTile, n - base);
    // a warp's pairs are contiguous, so that its counters run in slot order
    const uint32_t mine = base + warp * (32u * kSortItems) + lane;
    uint32_t key[kSortItems], val[kSortItems], rank[kSortItems];
#pragma unroll
    for (uint32_t k = 0; k < kSortItems; ++k) {
        const uint32_t p = mine + 32u * k;
        key[k] = p < n ? keys_in[p] : 0u;
        val[k] = p < n && vals_in ? vals_in[p] : p;
    }
    for (uint32_t i = threadIdx.x; i < kSortWarps * kBins / 2u; i += kSortThreads) reinterpret_cast<uint32_t*>(s_rank)[i] = 0u;
    __syncthreads();
    uint16_t* counter = s_rank[warp];
#pragma unroll
    for (uint32_t k = 0; k < kSortItems; ++k) {
        const bool valid = mine + 32u * k < n;
        const uint32_t d = valid ? digit_of(key[k], shift) : kBins;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int leader = __ffs(peers) - 1;
        uint32_t before = 0u;
        if (valid && lane == (unsigned)leader) {
            before = counter[d];
            counter[d] = (uint16_t)(before + (uint32_t)__popc(peers));
        }
        __syncwarp();
        rank[k] = __shfl_sync(0xffffffffu, before, leader) + (uint32_t)__popc(peers & ((1u << lane) - 1u));
    }
    __syncthreads();
    // thread t < 256: bin t.  The bin's warps in order, the bins in order, and
    // where the bin's run of this tile goes.
    const bool bin = threadIdx.x < kBins;
    uint32_t in_tile = 0u;
    if (bin)
#pragma unroll
        for (unsigned w = 0; w < kSortWarps; ++w) {
            const uint32_t c = s_rank[w][threadIdx.x];
            s_rank[w][threadIdx.x] = (uint16_t)in_tile;
            in_tile += c;
        }
    const uint32_t first = block_exclusive(in_tile, s_warp);
    const uint32_t bin_first = block_exclusive(bin ? bin_total[threadIdx.x] : 0u, s_warp);
    if (bin) {
        s_global[threadIdx.x] = bin_first + hist[(size_t)threadIdx.x * tiles + blockIdx.x] - first;
#pragma unroll
        for (unsigned w = 0; w < kSortWarps; ++w) s_rank[w][threadIdx.x] = (uint16_t)(s_rank[w][threadIdx.x] + first);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kSortItems; ++k)
        if (mine + 32u * k < n) {
            const uint32_t at = counter[digit_of(key[k], shift)] + rank[k];
            s_key[at] = key[k];
            s_val[at] = val[k];
        }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kSortItems; ++k) {
        const uint32_t i = k * kSortThreads + threadIdx.x;
        if (i < count) {
            const uint32_t q = s_key[i];
            const uint32_t to = s_global[digit_of(q, shift)] + i;
            if (keys_out) keys_out[to] = q;
            vals_out[to] = s_val[i];
        }
    }
}

// Bits needed for keys 0..cells (cells itself is the inactive key).
static int key_bits(size_t cells) {
    int b = 1;
    while (b < 32 && ((size_t)1 << b) <= cells) ++b;
    return b;
}

}  // namespace fpg

using namespace fpg;

extern "C" fpg_status fpg_sorter_create(fpg_ctx* ctx, size_t capacity, fpg_sorter** out) {
    if (!ctx || !out) return FPG_ERR_INVALID_ARGUMENT;
    if (capacity > (size_t)INT32_MAX) return FPG_ERR_VALUE_TOO_LARGE;
    fpg_sorter* s = new fpg_sorter();
    s->ctx = ctx;
    s->capacity = capacity;
    const size_t n = capacity > 0 ? capacity : 1;
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 2 && e == cudaSuccess; ++k) {
        e = cudaMalloc(&s->keys[k], n * sizeof(uint32_t));
        if (e == cudaSuccess) e = cudaMalloc(&s->vals[k], n * sizeof(uint32_t));
    }
    const size_t tiles = (n + kSortTile - 1) / kSortTile;
    if (e == cudaSuccess) e = cudaMalloc(&s->hist, tiles * kBins * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&s->bin_total, kBins * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&s->block, particles_block_bytes(capacity));
    if (e != cudaSuccess) {
        for (int k = 0; k < 2; ++k) { cudaFree(s->keys[k]); cudaFree(s->vals[k]); }
        cudaFree(s->hist); cudaFree(s->bin_total); cudaFree(s->block);
        delete s;
        return cuda_status(e);
    }
    *out = s;
    return FPG_OK;
}

extern "C" fpg_status fpg_sorter_destroy(fpg_sorter* s) {
    if (!s) return FPG_OK;
    for (int k = 0; k < 2; ++k) { cudaFree(s->keys[k]); cudaFree(s->vals[k]); }
    cudaFree(s->hist);
    cudaFree(s->bin_total);
    cudaFree(s->block);
    delete s;
    return FPG_OK;
}

extern "C" fpg_status fpg_sort_by_cell(fpg_ctx* ctx, fpg_particles* P, const fpg_met* met, fpg_sorter* s,
                                       uint32_t* perm_dev, void* stream) {
    if (!ctx || !P || !met || !s) return FPG_ERR_INVALID_ARGUMENT;
    if (s->capacity != P->capacity) return FPG_ERR_LENGTH_MISMATCH;
    if (met->nx * met->ny * met->nz >= (size_t)UINT32_MAX) return FPG_ERR_VALUE_TOO_LARGE;
    const uint32_t n = (uint32_t)P->dispatch;
    if (n == 0) return FPG_OK;
    cudaStream_t st = ctx->pick(stream);
    KeyArgs a;
    a.cell_x = (const int32_t*)P->field[FPG_FIELD_CELL_X];
    a.cell_y = (const int32_t*)P->field[FPG_FIELD_CELL_Y];
    a.pos_x = (const float*)P->field[FPG_FIELD_POS_X];
    a.pos_y = (const float*)P->field[FPG_FIELD_POS_Y];
    a.pos_z = (const float*)P->field[FPG_FIELD_POS_Z];
    a.flags = (const uint32_t*)P->field[FPG_FIELD_FLAGS];
    a.n = n;
    a.nx = (uint32_t)met->nx; a.ny = (uint32_t)met->ny; a.nz = (uint32_t)met->nz;
    a.lv = Levels{met->heights_dev, met->level_table_dev, met->level_inv_w, a.nz,
                  met->heights_set && met->heights[met->nz - 1] > 0.0f, level_mode(met)};
    const uint32_t tiles = (n + kSortTile - 1u) / kSortTile;
    launch_chained(cell_key_kernel, tiles, kSortThreads, 0, st, a, s->keys[0], s->hist, tiles);
    const uint32_t passes = ((uint32_t)key_bits(met->nx * met->ny * met->nz) + kDigitBits - 1u) / kDigitBits;
    const uint32_t* vals = nullptr;                      // the first pass sorts the positions themselves
    for (uint32_t k = 0; k < passes; ++k) {
        const uint32_t *keys_in = s->keys[k & 1u], shift = k * kDigitBits;
        if (k > 0) launch_chained(digit_histogram_kernel, tiles, kSortThreads, 0, st, keys_in, n, shift, s->hist, tiles);
        launch_chained(bin_scan_kernel, kBins, kScanThreads, 0, st, s->hist, tiles, s->bin_total);
        uint32_t* vals_out = s->vals[(k + 1u) & 1u];
        launch_chained(digit_scatter_kernel, tiles, kSortThreads, 0, st, keys_in, vals, n, shift, s->hist, s->bin_total, tiles,
                       k + 1u < passes ? s->keys[(k + 1u) & 1u] : nullptr, vals_out);
        vals = vals_out;
    }
    ctx->count(3u * passes);
    FPG_CHECK_LAUNCH();
    const uint32_t* perm = vals;
    void* dst[FPG_FIELD_COUNT];
    particles_assign_fields(s->block, s->capacity, dst);
    const fpg_status moved = move_fields(ctx, P->field, dst, perm, n, nullptr, (uint32_t)P->capacity, false, st);
    if (moved != FPG_OK) return moved;
    if (perm_dev) FPG_CUDA(cudaMemcpyAsync(perm_dev, perm, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    particles_swap_block(P, &s->block);
    return FPG_OK;
}
