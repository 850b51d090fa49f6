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
// Steps: key kernel -> stable LSD radix sort of (key, slot) pairs (CUB,
// header-only, compiled into this library) -> gather of all FPG_FIELD_COUNT
// arrays into a second structure-of-arrays block, which is swapped in.
// Philox streams follow the slot, as in the reference after its sort.
#include <cuda_runtime.h>
#include <cub/cub.cuh>

#include "fpg_internal.h"
#include "move_fields.h"
#include "physics.cuh"
#include "step_core.cuh"

struct fpg_sorter {
    fpg_ctx* ctx = nullptr;
    size_t capacity = 0;
    uint32_t* keys[2] = {};
    uint32_t* vals[2] = {};
    void* temp = nullptr;
    size_t temp_bytes = 0;
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

// Two adjacent slots per thread with 8-byte accesses, every load issued
// before the flags are looked at, the level found by the met's bucket table
// through L1.  32 B a slot, HBM-bound.
__global__ void __launch_bounds__(256) cell_key_kernel(KeyArgs a, uint32_t* __restrict__ keys,
                                                       uint32_t* __restrict__ vals) {
    chain_begin();
    const uint32_t p = 2u * (blockIdx.x * blockDim.x + threadIdx.x);
    if (p + 1u < a.n) {
        const uint2 f = *reinterpret_cast<const uint2*>(a.flags + p);
        const int2 cx = *reinterpret_cast<const int2*>(a.cell_x + p);
        const int2 cy = *reinterpret_cast<const int2*>(a.cell_y + p);
        const float2 px = *reinterpret_cast<const float2*>(a.pos_x + p);
        const float2 py = *reinterpret_cast<const float2*>(a.pos_y + p);
        const float2 z = *reinterpret_cast<const float2*>(a.pos_z + p);
        *reinterpret_cast<uint2*>(keys + p) = make_uint2(cell_key(a, f.x, cx.x, cy.x, px.x, py.x, z.x),
                                                         cell_key(a, f.y, cx.y, cy.y, px.y, py.y, z.y));
        *reinterpret_cast<uint2*>(vals + p) = make_uint2(p, p + 1u);
    } else if (p < a.n) {
        keys[p] = cell_key(a, a.flags[p], a.cell_x[p], a.cell_y[p], a.pos_x[p], a.pos_y[p], a.pos_z[p]);
        vals[p] = p;
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
    if (e == cudaSuccess) {
        cub::DoubleBuffer<uint32_t> kb(s->keys[0], s->keys[1]), vb(s->vals[0], s->vals[1]);
        e = cub::DeviceRadixSort::SortPairs(nullptr, s->temp_bytes, kb, vb, (int)n, 0, 32, ctx->stream);
    }
    if (e == cudaSuccess) e = cudaMalloc(&s->temp, s->temp_bytes > 0 ? s->temp_bytes : 1);
    if (e == cudaSuccess) e = cudaMalloc(&s->block, particles_block_bytes(capacity));
    if (e != cudaSuccess) {
        for (int k = 0; k < 2; ++k) { cudaFree(s->keys[k]); cudaFree(s->vals[k]); }
        cudaFree(s->temp); cudaFree(s->block);
        delete s;
        return cuda_status(e);
    }
    *out = s;
    return FPG_OK;
}

extern "C" fpg_status fpg_sorter_destroy(fpg_sorter* s) {
    if (!s) return FPG_OK;
    for (int k = 0; k < 2; ++k) { cudaFree(s->keys[k]); cudaFree(s->vals[k]); }
    cudaFree(s->temp);
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
    launch_chained(cell_key_kernel, (unsigned)(((uint64_t)n + 511u) / 512u), 256, 0, st, a, s->keys[0], s->vals[0]);
    ctx->count();
    FPG_CHECK_LAUNCH();
    cub::DoubleBuffer<uint32_t> kb(s->keys[0], s->keys[1]), vb(s->vals[0], s->vals[1]);
    size_t tb = s->temp_bytes;
    const int bits = key_bits(met->nx * met->ny * met->nz);
    FPG_CUDA(cub::DeviceRadixSort::SortPairs(s->temp, tb, kb, vb, (int)n, 0, bits, st));
    ctx->count(1 + (bits + 7) / 8);  // histogram + one pass per 8-bit digit
    const uint32_t* perm = vb.Current();
    void* dst[FPG_FIELD_COUNT];
    particles_assign_fields(s->block, s->capacity, dst);
    const fpg_status moved = move_fields(ctx, P->field, dst, perm, n, nullptr, (uint32_t)P->capacity, false, st);
    if (moved != FPG_OK) return moved;
    if (perm_dev) FPG_CUDA(cudaMemcpyAsync(perm_dev, perm, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    particles_swap_block(P, &s->block);
    return FPG_OK;
}
