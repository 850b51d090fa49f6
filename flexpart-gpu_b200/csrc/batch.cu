// batch.cu — many independent release scenarios stepped as one population.
//
// Each scenario reproduces one plain forward run (ForwardTimeLoopDriver with
// a single release, capacity = its particle count, its own Philox key and
// counter chain; src/simulation/timeloop.rs:915-1316): release lattice and
// slots (release/mod.rs:156-275), Philox block index = slot within the
// scenario, counter advanced by capacity * blocks per step
// (gpu/langevin_fused.rs:229-233).  All scenarios share one met frame ring
// and one clock.  Scenario s owns the 256-aligned slot segment
// [offset_s, offset_s + capacity_s) of one structure-of-arrays population;
// tile t (256 slots) belongs to exactly one scenario.
//
// One step is a short kernel sequence that reads its per-step values
// (clock, alpha, bracket, release ranges, counters) from device memory, so
// it is captured into CUDA graphs and replayed:
//   batch_pre       bracket from the ring when it changed, PBL (and wet
//                   forcing) per cell, new particles of every scenario
//                   (lattice in f64), grids cleared before an output step,
//                   and the next step's state: counters += capacity * blocks,
//                   clock += dt, its bracket, alpha and release ranges
//   batch_step      the fused per-particle step (step_core.cuh): one CTA per
//                   work item, or persistent CTAs that pull items
//   batch_grid      per-scenario grids at output steps
// The state of a step and the next lie in two buffers that swap every step.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <algorithm>
#include <vector>

#include "../../include/fpg_driver.h"
#include "batch_core.cuh"
#include "fpg_internal.h"
#include "grid_core.cuh"

namespace fpg {

size_t particles_block_bytes(size_t capacity);

namespace {


// The state of the coming step from the clock: bracket and alpha, and per
// scenario the release range and the Philox head.
__device__ __forceinline__ void advance_clock(BatchState* st, const BatchConst& c) {
    const int64_t t = st->t;
    // bracket holding t; at a frame time stay in the bracket ending there
    int64_t k = (t - c.start) / c.frame_seconds;
    if (t - c.start == k * c.frame_seconds && k > 0) k -= 1;
    const int32_t fa = (int32_t)(k % c.n_frames), fb = (int32_t)((k + 1) % c.n_frames);
    const int64_t ta = c.start + k * c.frame_seconds;
    st->changed = !st->have_bracket || fa != st->fa || fb != st->fb || ta != st->ta;
    st->fa = fa;
    st->fb = fb;
    st->ta = ta;
    st->have_bracket = 1;
    // interpolation_alpha (timeloop.rs:2117-2119)
    st->alpha = (float)((double)(t - ta) / (double)c.frame_seconds);
    st->work = 0;
}

// The release range and Philox head of scenario d at time t; `lo` particles
// are out already.
__device__ __forceinline__ void advance_scenario(ScenDev& d, int64_t t, uint32_t lo) {
    uint32_t hi = target_emitted(d.start, d.end, d.count, t, lo);
    if (hi < lo) hi = lo;
    d.rel_lo = lo;
    d.rel_hi = hi;
    d.released = hi;
    d.head = philox_head(d.counter, d.key0, d.key1);
    d.head_ok = (uint64_t)d.counter.x + 2u * (uint64_t)d.capacity <= (1ull << 32);
}

// The first step's state, when the batch is created or reset.
__global__ void __launch_bounds__(256) batch_begin_kernel(BatchState* st, ScenDev* sc, BatchConst c) {
    chain_begin();
    for (uint32_t s = threadIdx.x; s < c.n_scen; s += blockDim.x) advance_scenario(sc[s], st->t, sc[s].released);
    if (threadIdx.x == 0) advance_clock(st, c);
}

// The next step's state from this one's (counters and clock moved on), by one
// CTA.  The two steps' states lie in two buffers, so that this runs beside
// the step that reads the first.
__device__ __forceinline__ void turn(const BatchState* st, const ScenDev* sc, const BatchConst& c, BatchState* next_st,
                                     ScenDev* next_sc) {
    const int64_t t = st->t + c.dt;
    for (uint32_t s = threadIdx.x; s < c.n_scen; s += blockDim.x) {
        ScenDev d = sc[s];
        d.counter = counter_add64(d.counter, (uint64_t)d.capacity * c.bpp);
        advance_scenario(d, t, d.released);
        next_sc[s] = d;
    }
    if (threadIdx.x == 0) {
        BatchState n = *st;
        n.t = t;
        n.step += 1u;
        advance_clock(&n, c);
        *next_st = n;
    }
}

// ReleaseManager::inject_for_time + geo_to_grid + to_relative
// (release/mod.rs:103-146, coords/mod.rs:92-114,169-178) on the device, in
// the same f64 arithmetic as the host release manager.  CTA `part` of `parts`
// of one scenario.
__device__ __forceinline__ void release_particles(const BatchState* st, const ScenDev& d, const BatchConst& c,
                                                  const PopFields& F, uint32_t part, uint32_t parts, int32_t* error) {
    const int32_t now = (int32_t)st->t;
    for (uint32_t k = d.rel_lo + part * blockDim.x + threadIdx.x; k < d.rel_hi; k += parts * blockDim.x) {
        const uint64_t idx = k;
        const uint64_t ix = idx % d.lat_nx, iy = (idx / d.lat_nx) % d.lat_nx, iz = (idx / d.lat_nxy) % d.lat_nz;
        const double fx = ((double)ix + 0.5) / (double)d.lat_nx;
        const double fy = ((double)iy + 0.5) / (double)d.lat_nx;
        const double fz = ((double)iz + 0.5) / (double)d.lat_nz;
        const double lon = d.lon_min + fx * (d.lon_max - d.lon_min);
        const double lat = d.lat_min + fy * (d.lat_max - d.lat_min);
        const double z = d.z_min + fz * (d.z_max - d.z_min);
        const double x = (lon - c.xlon0) / c.dx;
        const double y = (lat - c.ylat0) / c.dy;
        if (!(x >= 0.0 && x < (double)(c.gnx - 1) && y >= 0.0 && y < (double)(c.gny - 1))) {
            atomicOr(error, 1);
            continue;
        }
        const double fxf = floor(x), fyf = floor(y);
        const uint32_t p = d.offset + k;
        F.f[FPG_FIELD_CELL_X][p] = (uint32_t)(int32_t)fxf;
        F.f[FPG_FIELD_CELL_Y][p] = (uint32_t)(int32_t)fyf;
        F.f[FPG_FIELD_POS_X][p] = __float_as_uint((float)(x - fxf));
        F.f[FPG_FIELD_POS_Y][p] = __float_as_uint((float)(y - fyf));
        F.f[FPG_FIELD_POS_Z][p] = __float_as_uint((float)z);
        F.f[FPG_FIELD_FLAGS][p] = FPG_FLAG_ACTIVE;
        F.f[FPG_FIELD_MASS0][p] = __float_as_uint(d.mass_per_particle);
        F.f[FPG_FIELD_TIME][p] = (uint32_t)now;
        F.f[FPG_FIELD_TIME_MEM][p] = (uint32_t)now;
        // every other field of a fresh slot is zero (the population starts zeroed)
    }
}

// Everything a step does beside its particle pass, one launch before it: the
// CTAs are shared out over independent parts that read the step's state, and
// one CTA writes the next step's.
// A step of a small ensemble is bound by its launches (separate advance,
// pack, PBL, release and end kernels took 11 us of device time and five
// launches a step beside an 11 us pass at 160 k particles).
struct PreArgs {
    const float4* ring;                  // pack the bracket when it changed
    float4* bracket;
    uint32_t nodes, pack_ctas;
    const fpg_surface_cell* sring;       // PBL cells, and the wet cells when the bracket changed
    const float* precip;
    fpg_pbl_options pbl;
    uint32_t ncell, pbl_ctas;
    float* field[7];
    float4* packed;
    CellHanna* hanna;
    int wet_on;
    float wet_a, wet_b;
    float2* wet;
    uint32_t parts;                      // release CTAs per scenario
    PopFields F;
    BatchState* st_out;                  // inversion: the step's state kept per tape slice (NULL: not kept)
    ScenDev* sc_out;
    uint32_t slices;
    BatchState* st_next;                 // the next step's state
    ScenDev* sc_next;
    int32_t* error;
    uint32_t* clear[2];                  // the output grids, cleared on output steps
    size_t clear_n;
    uint32_t clear_ctas;
};
constexpr uint32_t kPreThreads = 128;

__global__ void __launch_bounds__(kPreThreads) batch_pre_kernel(const BatchState* st, const ScenDev* sc, BatchConst c,
                                                                PreArgs a) {
    chain_begin();
    if (blockIdx.x == 0) {
        turn(st, sc, c, a.st_next, a.sc_next);
        return;
    }
    uint32_t b = blockIdx.x - 1u;
    if (b < a.pbl_ctas) {
        const uint32_t i = b * kPreThreads + threadIdx.x;
        if (i >= a.ncell) return;
        pbl_cell(a.sring + (size_t)st->fa * a.ncell, a.sring + (size_t)st->fb * a.ncell, st->alpha, a.pbl, i, a.field[0],
                 a.field[1], a.field[2], a.field[3], a.field[4], a.field[5], a.field[6], a.packed, a.hanna);
        if (a.wet_on && st->changed)
            a.wet[i] = wet_cell_forcing(a.precip[(size_t)st->fa * a.ncell + i], 0.0f, 1.0f, a.wet_a, a.wet_b);
        return;
    }
    b -= a.pbl_ctas;
    if (b < c.n_scen * a.parts) {
        release_particles(st, sc[b / a.parts], c, a.F, b % a.parts, a.parts, a.error);
        return;
    }
    b -= c.n_scen * a.parts;
    if (b < a.pack_ctas) {
        if (!st->changed) return;
        const float4* f0 = a.ring + (size_t)st->fa * a.nodes;
        const float4* f1 = a.ring + (size_t)st->fb * a.nodes;
        for (uint32_t n = b * kPreThreads + threadIdx.x; n < a.nodes; n += a.pack_ctas * kPreThreads)
            st_node(a.bracket, n, f0[n], f1[n]);
        return;
    }
    b -= a.pack_ctas;
    if (b < a.clear_ctas) {
        for (size_t i = (size_t)b * kPreThreads + threadIdx.x; i < a.clear_n; i += (size_t)a.clear_ctas * kPreThreads) {
            a.clear[0][i] = 0u;
            a.clear[1][i] = 0u;
        }
        return;
    }
    // the last CTA: the clock and scenario state of the step's tape slice
    const uint32_t j = st->step % a.slices;
    if (threadIdx.x == 0) a.st_out[j] = *st;
    for (uint32_t s = threadIdx.x; s < c.n_scen; s += kPreThreads) a.sc_out[(size_t)j * c.n_scen + s] = sc[s];
}

// One work item is a chunk of BLOCK * PPT consecutive slots of one scenario
// (x: scenario, y: first slot within the scenario).  CTAs stay resident and
// pull items from a device counter until none is left, so small and large
// scenarios share the machine without a per-scenario launch.
template <int BLOCK, int MINB, int PPT>
__global__ void __launch_bounds__(BLOCK, MINB) batch_step_kernel(StepArgs a, BatchState* st,
                                                                 const ScenDev* sc,
                                                                 const uint2* items, uint32_t n_items) {
    chain_begin();
    extern __shared__ float s_levels[];
    __shared__ uint32_t s_item;
    const Levels lv = stage_levels(a, s_levels);
    const float alpha = st->alpha;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(&st->work, 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= n_items) break;
        const uint2 w = items[it];
        const ScenDev& d = sc[w.x];
        const uint32_t released = d.released;
#pragma unroll 1
        for (int j = 0; j < PPT; ++j) {
            const uint32_t local = w.y + (uint32_t)(j * BLOCK) + threadIdx.x;
            if (local < released)
                particle_step(a, lv, d.offset + local, local, alpha, d.counter, d.key0, d.key1);
        }
    }
}

// The same pass with one CTA per work item of BLOCK slots, launched over all
// items (particles_per_thread 0 in the tuning records): no work counter and
// no barrier, the level arrays read from global memory, and the hardware's
// block scheduler spreading the items of small and large scenarios.
template <int BLOCK, int MINB>
__global__ void __launch_bounds__(BLOCK, MINB) batch_step_flat_kernel(StepArgs a, BatchState* st,
                                                                      const ScenDev* sc,
                                                                      const uint2* items,
                                                                      uint32_t n_items) {
    chain_begin();
    if (blockIdx.x >= n_items) return;
    const uint2 w = items[blockIdx.x];
    const ScenDev& d = sc[w.x];
    const uint32_t local = w.y + threadIdx.x;
    if (local < d.released)
        particle_step(a, global_levels(a), d.offset + local, local, st->alpha, d.counter, d.key0, d.key1);
}

// The flat pass when the configuration is in the production form
// (production_form in step_core.cuh), compiled for 40 warps per SM (48
// registers) whatever the shape: 24 scenarios (2.1 M particles) 119 us a
// pass, against 146 us of the general body and 128, 123 and 121 us with 8, 9
// and 12 CTAs of 128 threads; 150 scenarios 697 us, against 757, 724, 699.
template <bool kWet, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1280 / BLOCK) batch_production_kernel(StepArgs a, BatchState* st,
                                                                       const ScenDev* sc,
                                                                       const uint2* items,
                                                                       uint32_t n_items) {
    chain_begin();
    if (blockIdx.x >= n_items) return;
    const uint2 w = items[blockIdx.x];
    const ScenDev& d = sc[w.x];
    const uint32_t local = w.y + threadIdx.x;
    if (local < d.released)
        production_step<kWet>(a, d.offset + local, local, st->alpha, d.counter, d.key0, d.key1, d.head,
                              HeadKeys{d.head.k0, d.head.k1}, d.head_ok != 0u);
}

// The launch shapes the particle pass is compiled for; the tuner picks one,
// and the first is the default.  ppt 0: batch_step_flat_kernel, one CTA per
// item of `block` slots, with its production form (dry, wet).
using StepKernel = void (*)(StepArgs, BatchState*, const ScenDev*, const uint2*, uint32_t);
struct StepVariant {
    uint32_t block, minb, ppt;
    StepKernel kernel;
    StepKernel production[2];
};

template <int BLOCK, int MINB>
constexpr StepVariant flat_variant() {
    return StepVariant{BLOCK, MINB, 0, batch_step_flat_kernel<BLOCK, MINB>,
                       {batch_production_kernel<false, BLOCK>, batch_production_kernel<true, BLOCK>}};
}

const StepVariant kVariants[] = {
    flat_variant<128, 12>(),
    {256, 4, 1, batch_step_kernel<256, 4, 1>}, {256, 4, 2, batch_step_kernel<256, 4, 2>},
    {256, 3, 1, batch_step_kernel<256, 3, 1>}, {256, 2, 1, batch_step_kernel<256, 2, 1>},
    {128, 8, 1, batch_step_kernel<128, 8, 1>}, {128, 8, 2, batch_step_kernel<128, 8, 2>},
    {512, 2, 1, batch_step_kernel<512, 2, 1>}, {256, 5, 1, batch_step_kernel<256, 5, 1>},
    flat_variant<256, 5>(), flat_variant<128, 10>(),
};
static_assert(sizeof(kVariants) / sizeof(kVariants[0]) == kNumVariants, "launch shape table");

// What shape v runs for these arguments.  In the production form the two flat
// shapes of 128 threads are one kernel.
StepKernel pass_kernel(const StepVariant& v, const StepArgs& a) {
    return v.ppt == 0 && production_form(a) ? v.production[a.wet_mode == FPG_FORCING_PER_CELL] : v.kernel;
}

struct GridConst {
    uint32_t nx, ny, nz, cells;
    int meters, sorted;
    float scale;
    uint32_t every;
    float h[FPG_MAX_LEVELS];
    float lower[kSortedLevels - 1];     // level_sorted's table when `sorted`
};

// concentration_gridding.wgsl:323-345 per scenario.  Each CTA bins a
// contiguous range of tiles (a tile is 256 slots of one scenario); the key of
// a particle is its index in the scenario-major grid, so one CTA table holds
// the cells of every scenario its tiles touch.  Runs of equal keys in a warp
// are summed by the segmented scan, the run ends add to the table, and the
// table goes to the grids once per cell per CTA (grid_core.cuh).
__global__ void __launch_bounds__(256) batch_grid_kernel(const BatchState* st, const ScenDev* sc,
                                                         const uint32_t* tile_scen, PopFields F,
                                                         GridConst g, uint32_t n_tiles, uint32_t tiles_per_cta,
                                                         uint32_t* counts, uint32_t* mass) {
    chain_begin();
    if (g.every == 0 || (st->step + 1u) % g.every != 0u) return;
    __shared__ float s_h[FPG_MAX_LEVELS];
    __shared__ uint32_t t_key[kTable], t_cnt[kTable], t_mass[kTable];
    if (!g.sorted)
        for (uint32_t i = threadIdx.x; i < g.nz; i += blockDim.x) s_h[i] = g.h[i];
    for (uint32_t i = threadIdx.x; i < kTable; i += blockDim.x) {
        t_key[i] = kEmpty;
        t_cnt[i] = 0u;
        t_mass[i] = 0u;
    }
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t t0 = blockIdx.x * tiles_per_cta;
    const uint32_t t1 = min(t0 + tiles_per_cta, n_tiles);
    for (uint32_t tile = t0; tile < t1; ++tile) {                       // uniform across the CTA
        const uint32_t s = tile_scen[tile];
        const ScenDev& d = sc[s];
        const uint32_t local = (tile - d.first_tile) * TILE + threadIdx.x;
        const uint32_t p = d.offset + local;
        uint32_t key = kEmpty, q = 0u;
        if (local < d.released && (F.f[FPG_FIELD_FLAGS][p] & 1u)) {
            const int32_t cx = (int32_t)F.f[FPG_FIELD_CELL_X][p], cy = (int32_t)F.f[FPG_FIELD_CELL_Y][p];
            const uint32_t ix = (uint32_t)min(max(cx, 0), (int)g.nx - 1);
            const uint32_t iy = (uint32_t)min(max(cy, 0), (int)g.ny - 1);
            const float z = __uint_as_float(F.f[FPG_FIELD_POS_Z][p]);
            const uint32_t iz = g.sorted ? level_sorted(z, g.lower, g.nz) : level_of(z, s_h, g.nz, g.meters);
            key = s * g.cells + (ix * g.ny + iy) * g.nz + iz;
            q = quantize(fmaxf(__uint_as_float(F.f[FPG_FIELD_MASS0][p]), 0.0f), g.scale);
        }
        warp_runs_add(key, q, lane, t_key, t_cnt, t_mass, counts, mass);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kTable; i += blockDim.x) {
        const uint32_t k = t_key[i];
        if (k != kEmpty) {
            atomicAdd(counts + k, t_cnt[i]);
            atomicAdd(mass + k, t_mass[i]);
        }
    }
}

}  // namespace

StepArgs make_step_args(fpg_batch* b) {
    fpg_particles* P = b->pop;
    StepArgs a;
    std::memset(&a, 0, sizeof(a));
    a.cell_x = (int32_t*)P->field[FPG_FIELD_CELL_X];
    a.cell_y = (int32_t*)P->field[FPG_FIELD_CELL_Y];
    a.pos_x = (float*)P->field[FPG_FIELD_POS_X];
    a.pos_y = (float*)P->field[FPG_FIELD_POS_Y];
    a.pos_z = (float*)P->field[FPG_FIELD_POS_Z];
    a.flags = (const uint32_t*)P->field[FPG_FIELD_FLAGS];
    for (int k = 0; k < 4; ++k) a.mass[k] = (float*)P->field[FPG_FIELD_MASS0 + k];
    a.vel_u = (float*)P->field[FPG_FIELD_VEL_U];
    a.vel_v = (float*)P->field[FPG_FIELD_VEL_V];
    a.vel_w = (float*)P->field[FPG_FIELD_VEL_W];
    a.turb_u = (float*)P->field[FPG_FIELD_TURB_U];
    a.turb_v = (float*)P->field[FPG_FIELD_TURB_V];
    a.turb_w = (float*)P->field[FPG_FIELD_TURB_W];
    a.cbt = (int32_t*)P->field[FPG_FIELD_CBT];
    a.n = (uint32_t)P->capacity;
    a.n_species = 1;                                  // each release fills species 0 only
    const fpg_batch_config& c = b->cfg;
    a.stages = FPG_STAGE_ADVECT | FPG_STAGE_TURBULENCE;
    a.bracket = b->met->bracket;
    a.heights = b->met->heights_dev;
    a.nx = (uint32_t)b->met->nx; a.ny = (uint32_t)b->met->ny; a.nz = (uint32_t)b->met->nz;
    a.has_heights = b->met->heights_set && b->met->heights[b->met->nz - 1] > 0.0f;
    a.level_mode = level_mode(b->met);
    a.level_table = b->met->level_table_dev;
    a.level_inv_w = b->met->level_inv_w;
    a.dt = (float)c.timestep_seconds;
    a.xs = c.x_grid_per_meter; a.ys = c.y_grid_per_meter; a.zs = c.z_grid_per_meter;
    a.hcell = b->pbl->hanna;
    a.pnx = (uint32_t)b->pbl->nx; a.pny = (uint32_t)b->pbl->ny;
    a.tdt = (float)c.timestep_seconds;
    a.rho = c.rho_grad_over_rho;
    a.zmin = c.min_height_m;
    a.n_sub = c.n_substeps;
    a.href = fmaxf(c.dry_reference_height_m, 0.1f);
    a.dry_mode = c.dry_velocity_m_s != 0.0f ? FPG_FORCING_UNIFORM : FPG_FORCING_NONE;
    if (a.dry_mode) a.stages |= FPG_STAGE_DRY;
    a.dry_v = c.dry_velocity_m_s;
    a.wet_mode = c.wet_from_precipitation ? FPG_FORCING_PER_CELL : FPG_FORCING_NONE;
    if (a.wet_mode) {
        a.stages |= FPG_STAGE_WET;
        a.wet_cells = b->wet->lf;
        a.wnx = (uint32_t)b->wet->nx; a.wny = (uint32_t)b->wet->ny;
    }
    return a;
}

BatchConst make_const(const fpg_batch* b) {
    BatchConst c;
    c.start = b->cfg.start_seconds;
    c.frame_seconds = b->cfg.frame_seconds;
    c.dt = b->cfg.timestep_seconds;
    c.n_frames = b->cfg.n_frames;
    c.n_scen = (uint32_t)b->scen.size();
    c.n_tiles = b->n_tiles;
    c.bpp = b->cfg.n_substeps <= 2u ? 1u : 2u;
    c.xlon0 = b->cfg.release_grid.xlon0; c.ylat0 = b->cfg.release_grid.ylat0;
    c.dx = b->cfg.release_grid.dx; c.dy = b->cfg.release_grid.dy;
    c.gnx = b->cfg.release_grid.nx; c.gny = b->cfg.release_grid.ny;
    return c;
}

GridConst make_grid_const(const fpg_batch* b) {
    GridConst g;
    std::memset(&g, 0, sizeof(g));
    g.nx = b->cfg.out_nx; g.ny = b->cfg.out_ny; g.nz = b->cfg.out_nz;
    g.cells = g.nx * g.ny * g.nz;
    for (uint32_t k = 0; k < g.nz; ++k) g.h[k] = b->outheights[k];
    g.meters = g.nz > 0 && g.h[g.nz - 1] > 0.0f;
    g.sorted = sorted_levels(g.h, g.nz, g.lower);
    g.scale = 1.0e6f;
    g.every = b->cfg.output_every_steps;
    return g;
}

PopFields pop_fields(fpg_batch* b) {
    PopFields F;
    for (int f = 0; f < FPG_FIELD_COUNT; ++f) F.f[f] = static_cast<uint32_t*>(b->pop->field[f]);
    return F;
}

static bool grid_step(const fpg_batch* b, uint64_t step) {
    const fpg_batch_config& c = b->cfg;
    return c.output_every_steps && c.out_nx && c.out_ny && c.out_nz && b->n_tiles &&
           (step + 1) % c.output_every_steps == 0;
}

bool output_step(const fpg_batch* b, uint64_t step) { return grid_step(b, step) || inverse_sample_step(b, step); }

// Everything before the particle pass; `output`: the step ends with grids.
// st_out, sc_out: where an inversion keeps the step's state.
void enqueue_pre(fpg_batch* b, cudaStream_t s, uint32_t side, bool output, BatchState* st_out, ScenDev* sc_out,
                 uint32_t slices) {
    const BatchConst c = make_const(b);
    PreArgs a;
    std::memset(&a, 0, sizeof(a));
    a.ring = b->ring;
    a.bracket = b->met->bracket;
    a.nodes = (uint32_t)(b->met->nx * b->met->ny * b->met->nz);
    a.pack_ctas = std::min<uint32_t>((a.nodes + kPreThreads - 1u) / kPreThreads, (uint32_t)b->ctx->sm_count * 8u);
    a.sring = b->sring;
    a.precip = b->pring;
    a.pbl = b->cfg.pbl_options;
    a.ncell = (uint32_t)(b->pbl->nx * b->pbl->ny);
    a.pbl_ctas = (a.ncell + kPreThreads - 1u) / kPreThreads;
    for (int k = 0; k < 7; ++k) a.field[k] = b->pbl->field[k];
    a.packed = b->pbl->packed;
    a.hanna = b->pbl->hanna;
    a.wet_on = b->cfg.wet_from_precipitation;
    a.wet_a = b->cfg.wet_gas_a;
    a.wet_b = b->cfg.wet_gas_b;
    a.wet = b->wet ? b->wet->lf : nullptr;
    a.parts = std::max<uint32_t>(1u, std::min<uint32_t>(32u, 1024u / c.n_scen));
    a.F = pop_fields(b);
    a.st_out = st_out;
    a.sc_out = sc_out;
    a.slices = std::max(slices, 1u);
    a.st_next = b->st + (side ^ 1u);
    a.sc_next = b->scen_state(side ^ 1u);
    a.error = b->error;
    if (output && b->cfg.output_every_steps) {
        a.clear[0] = b->grid_counts;
        a.clear[1] = b->grid_mass;
        a.clear_n = (size_t)b->cfg.out_nx * b->cfg.out_ny * b->cfg.out_nz * b->scen.size();
        a.clear_ctas = (uint32_t)b->ctx->sm_count * 8u;
    }
    const uint32_t ctas = a.pbl_ctas + c.n_scen * a.parts + a.pack_ctas + a.clear_ctas + (st_out ? 2u : 1u);
    launch_chained(batch_pre_kernel, ctas, kPreThreads, 0, s, b->st + side, b->scen_state(side), c, a);
    b->ctx->count(1);
}

// The grids or receptor samples of an output step.
void enqueue_post(fpg_batch* b, cudaStream_t s, uint32_t side, bool output) {
    if (output && b->cfg.output_every_steps) {
        const GridConst g = make_grid_const(b);
        // 8 resident CTAs per SM, each over a contiguous range of tiles
        const uint32_t ctas = std::max<uint32_t>(1u, std::min<uint32_t>(b->n_tiles, (uint32_t)b->ctx->sm_count * 8u));
        const uint32_t per = (b->n_tiles + ctas - 1u) / ctas;
        const uint32_t blocks = std::max<uint32_t>(1u, (b->n_tiles + per - 1u) / per);
        launch_chained(batch_grid_kernel, blocks, 256, 0, s, b->st + side, b->scen_state(side), b->tile_scen, pop_fields(b),
                       g, b->n_tiles, per, b->grid_counts, b->grid_mass);
        b->ctx->count(1);
    }
    if (output && b->inv) enqueue_inverse_sample(b, s, side);
}

static void enqueue_begin(fpg_batch* b, cudaStream_t s) {
    launch_chained(batch_begin_kernel, 1, 256, 0, s, b->st, b->sc, make_const(b));
    b->ctx->count(1);
}

void enqueue_step_kernel(fpg_batch* b, cudaStream_t s, uint32_t side) {
    const StepVariant& v = kVariants[b->variant];
    const StepArgs a = make_step_args(b);
    if (v.ppt == 0) {
        launch_chained(pass_kernel(v, a), std::max(b->n_items, 1u), v.block, 0, s, a, b->st + side,
                       b->scen_state(side), b->items, b->n_items);
    } else {
        const uint32_t grid = (uint32_t)b->ctx->sm_count * std::max(b->resident[b->variant], 1u);
        launch_chained(v.kernel, grid, v.block, level_smem_bytes(b->met), s, a, b->st + side, b->scen_state(side), b->items,
                       b->n_items);
    }
    b->ctx->count(1);
}

void enqueue_batched_step(fpg_batch* b, cudaStream_t s, uint64_t step, bool output) {
    const uint32_t side = (uint32_t)(step & 1u);
    enqueue_pre(b, s, side, output, nullptr, nullptr, 0);
    enqueue_step_kernel(b, s, side);
    enqueue_post(b, s, side, output);
}

static void drop_graphs(fpg_batch* b) {
    for (int o = 0; o < 4; ++o) {
        if (b->exec[o]) cudaGraphExecDestroy(b->exec[o]);
        if (b->graph[o]) cudaGraphDestroy(b->graph[o]);
        b->exec[o] = nullptr;
        b->graph[o] = nullptr;
    }
}

// Work items of shape `v`: every scenario cut into chunks of block * ppt slots.
fpg_status build_items(fpg_batch* b, uint32_t v) {
    const uint32_t chunk = kVariants[v].block * std::max(kVariants[v].ppt, 1u);
    std::vector<uint2> items;
    for (size_t s = 0; s < b->scen.size(); ++s)
        for (uint32_t l = 0; l < b->scen[s].capacity; l += chunk) items.push_back(make_uint2((uint32_t)s, l));
    if (items.size() > b->items_cap) {
        cudaFree(b->items);
        b->items = nullptr;
        b->items_cap = 0;
        FPG_CUDA(cudaMalloc(&b->items, items.size() * sizeof(uint2)));
        b->items_cap = items.size();
    }
    FPG_CUDA(cudaMemcpyAsync(b->items, items.data(), items.size() * sizeof(uint2), cudaMemcpyHostToDevice,
                             b->ctx->stream));
    FPG_CUDA(cudaStreamSynchronize(b->ctx->stream));
    b->n_items = (uint32_t)items.size();
    b->variant = v;
    drop_graphs(b);                                      // the captured graphs hold the old shape
    return FPG_OK;
}

__global__ void __launch_bounds__(256) batch_pack_forced_kernel(const BatchState* st, const float4* __restrict__ ring,
                                                                uint32_t nodes, float4* __restrict__ bracket) {
    const float4* f0 = ring + (size_t)st->fa * nodes;
    const float4* f1 = ring + (size_t)st->fb * nodes;
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n < nodes; n += gridDim.x * blockDim.x) {
        st_node(bracket, n, f0[n], f1[n]);
    }
}

void enqueue_pack_forced(fpg_batch* b, const BatchState* st, cudaStream_t s) {
    const uint32_t nodes = (uint32_t)(b->met->nx * b->met->ny * b->met->nz);
    batch_pack_forced_kernel<<<b->ctx->sm_count * 4, 256, 0, s>>>(st, b->ring, nodes, b->met->bracket);
    b->ctx->count(1);
}

fpg_status batch_reset(fpg_batch* b) {
    cudaStream_t s = b->ctx->stream;
    FPG_CUDA(cudaMemsetAsync(b->pop->block, 0, particles_block_bytes(b->capacity), s));
    BatchState s0;
    std::memset(&s0, 0, sizeof(s0));
    s0.t = b->cfg.start_seconds;
    FPG_CUDA(cudaMemcpyAsync(b->st, &s0, sizeof(s0), cudaMemcpyHostToDevice, s));
    FPG_CUDA(cudaMemcpyAsync(b->sc, b->scen.data(), b->scen.size() * sizeof(ScenDev), cudaMemcpyHostToDevice, s));
    FPG_CUDA(cudaMemsetAsync(b->error, 0, sizeof(int32_t), s));
    enqueue_begin(b, s);
    FPG_CHECK_LAUNCH();
    FPG_CUDA(cudaStreamSynchronize(s));
    b->steps_done = 0;
    b->t_h = b->cfg.start_seconds;
    for (size_t k = 0; k < b->scen.size(); ++k) {
        b->released_h[k] = 0;
        b->counter_h[k] = b->scen[k].counter;
    }
    return FPG_OK;
}

// The graph of a step, by its side of the state (1) and whether it ends with
// grids (2).
static int graph_of(const fpg_batch* b, uint64_t step) { return (int)(step & 1u) + (output_step(b, step) ? 2 : 0); }

// Captures the graph of `step` if it is not held yet.
static fpg_status ensure_graph(fpg_batch* b, uint64_t step, cudaStream_t s) {
    const int which = graph_of(b, step);
    if (b->exec[which]) return FPG_OK;
    FPG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    const uint64_t before = b->ctx->launches.load();
    enqueue_batched_step(b, s, step, output_step(b, step));
    // capture launches nothing: take the count back, keep it per replay
    b->graph_launches[which] = b->ctx->launches.load() - before;
    b->ctx->launches.fetch_sub(b->graph_launches[which]);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(s, &g);
    if (e != cudaSuccess) return cuda_status(e);
    e = cudaGraphInstantiate(&b->exec[which], g, 0);
    if (e != cudaSuccess) {
        b->exec[which] = nullptr;
        cudaGraphDestroy(g);
        return cuda_status(e);
    }
    b->graph[which] = g;
    return FPG_OK;
}

static fpg_status launch_step_graph(fpg_batch* b, uint64_t step, cudaStream_t s) {
    const int which = graph_of(b, step);
    FPG_CUDA(cudaGraphLaunch(b->exec[which], s));
    b->ctx->count(b->graph_launches[which]);
    return FPG_OK;
}

// ReleaseError::OutOfGridDomain (release/mod.rs:41) of scenario d, checked at
// the lattice's extreme points (lon, lat grow monotonically with the lattice
// index, so every other point lies between them).
fpg_status check_release_grid(const ScenDev& d, const fpg_grid_domain& g) {
    const uint64_t ix_hi = std::min<uint64_t>(d.lat_nx - 1, d.count - 1);
    const uint64_t iy_hi = std::min<uint64_t>(d.lat_nx - 1, (d.count - 1) / d.lat_nx);
    for (int e = 0; e < 4; ++e) {
        const uint64_t ix = (e & 1) ? ix_hi : 0, iy = (e & 2) ? iy_hi : 0;
        const double lon = d.lon_min + (((double)ix + 0.5) / (double)d.lat_nx) * (d.lon_max - d.lon_min);
        const double lat = d.lat_min + (((double)iy + 0.5) / (double)d.lat_nx) * (d.lat_max - d.lat_min);
        const double x = (lon - g.xlon0) / g.dx;
        const double y = (lat - g.ylat0) / g.dy;
        if (!(x >= 0.0 && x < (double)(g.nx - 1) && y >= 0.0 && y < (double)(g.ny - 1))) return FPG_ERR_OUT_OF_GRID;
    }
    return FPG_OK;
}

}  // namespace fpg

using namespace fpg;

extern "C" fpg_status fpg_batch_destroy(fpg_batch* b) {
    if (!b) return FPG_OK;
    cudaStreamSynchronize(b->ctx->stream);
    drop_graphs(b);
    fpg_particles_destroy(b->pop);
    fpg_met_destroy(b->met);
    fpg_pbl_destroy(b->pbl);
    fpg_cellfield_destroy(b->wet);
    cudaFree(b->ring); cudaFree(b->sring); cudaFree(b->pring); cudaFree(b->staging);
    cudaFree(b->st); cudaFree(b->sc); cudaFree(b->error); cudaFree(b->tile_scen); cudaFree(b->items); cudaFree(b->grid_counts); cudaFree(b->grid_mass);
    delete b;
    return FPG_OK;
}

extern "C" fpg_status fpg_batch_create(fpg_ctx* ctx, const fpg_batch_config* cfg, const fpg_batch_scenario* scen,
                                       size_t n_scen, size_t nx, size_t ny, size_t nz, const float* heights,
                                       fpg_batch** out) {
    if (!ctx || !cfg || !out || !scen || n_scen == 0 || n_scen > 65535) return FPG_ERR_INVALID_ARGUMENT;
    if (cfg->start_seconds > cfg->end_seconds) return FPG_ERR_INVALID_TIME_RANGE;
    if (cfg->timestep_seconds <= 0 || cfg->frame_seconds <= 0 || cfg->n_frames == 0) return FPG_ERR_INVALID_TIME_STEP;
    if (cfg->output_every_steps && (cfg->out_nx == 0 || cfg->out_ny == 0 || cfg->out_nz == 0)) return FPG_ERR_ZERO_SHAPE;
    if (cfg->out_nz > FPG_MAX_LEVELS) return FPG_ERR_TOO_MANY_LEVELS;
    fpg_batch* b = new fpg_batch();
    b->ctx = ctx;
    b->cfg = *cfg;
    if (cfg->outheights && cfg->out_nz) b->outheights.assign(cfg->outheights, cfg->outheights + cfg->out_nz);
    else b->outheights.assign(cfg->out_nz, 0.0f);
    b->cfg.outheights = nullptr;
    size_t offset = 0;
    for (size_t s = 0; s < n_scen; ++s) {
        const fpg_release& r = scen[s].release;
        if (r.lon_min > r.lon_max || r.lat_min > r.lat_max || r.z_min > r.z_max) { delete b; return FPG_ERR_INVALID_BOUNDS; }
        if (r.particle_count == 0 || r.particle_count >= (1ull << 32) || r.end_seconds - r.start_seconds >= (1ll << 32)) {
            delete b;
            return FPG_ERR_VALUE_TOO_LARGE;
        }
        ScenDev d;
        std::memset(&d, 0, sizeof(d));
        d.offset = (uint32_t)offset;
        d.capacity = (uint32_t)r.particle_count;
        d.first_tile = (uint32_t)(offset / TILE);
        d.n_tiles = (uint32_t)((r.particle_count + TILE - 1) / TILE);
        d.key0 = scen[s].key[0]; d.key1 = scen[s].key[1];
        d.counter = u32x4{scen[s].counter[0], scen[s].counter[1], scen[s].counter[2], scen[s].counter[3]};
        d.mass_per_particle = (float)(r.mass_kg / (double)r.particle_count);
        d.start = r.start_seconds; d.end = r.end_seconds;
        d.lon_min = r.lon_min; d.lon_max = r.lon_max; d.lat_min = r.lat_min; d.lat_max = r.lat_max;
        d.z_min = r.z_min; d.z_max = r.z_max;
        d.count = r.particle_count;
        // the lattice size of ReleaseBounds::sample_stratified (release/mod.rs:257-260), computed on the host
        double c = std::ceil(std::cbrt((double)r.particle_count));
        if (c < 1.0) c = 1.0;
        d.lat_nx = (uint64_t)c;
        d.lat_nxy = d.lat_nx * d.lat_nx > 0 ? d.lat_nx * d.lat_nx : 1;
        d.lat_nz = (r.particle_count + d.lat_nxy - 1) / d.lat_nxy;
        if (d.lat_nz < 1) d.lat_nz = 1;
        if (check_release_grid(d, cfg->release_grid) != FPG_OK) {
            delete b;
            return FPG_ERR_OUT_OF_GRID;
        }
        b->scen.push_back(d);
        for (uint32_t t = 0; t < d.n_tiles; ++t) b->tile_scen_h.push_back((uint32_t)s);
        offset += (size_t)d.n_tiles * TILE;
    }
    if (offset >= (size_t)UINT32_MAX) { delete b; return FPG_ERR_VALUE_TOO_LARGE; }
    b->capacity = offset;
    b->n_tiles = (uint32_t)b->tile_scen_h.size();
    b->total_steps = (uint64_t)((cfg->end_seconds - cfg->start_seconds) / cfg->timestep_seconds) + 1;
    b->released_h.assign(n_scen, 0);
    for (const ScenDev& d : b->scen) b->counter_h.push_back(d.counter);
    b->t_h = cfg->start_seconds;

    fpg_status st = fpg_particles_create(ctx, b->capacity, &b->pop);
    if (st == FPG_OK) st = fpg_met_create(ctx, nx, ny, nz, &b->met);
    if (st == FPG_OK && heights) st = fpg_met_set_level_heights(b->met, heights, nz);
    if (st == FPG_OK) st = fpg_pbl_create(ctx, nx, ny, &b->pbl);
    if (st == FPG_OK && cfg->wet_from_precipitation) st = fpg_cellfield_create(ctx, nx, ny, &b->wet);
    if (st != FPG_OK) { fpg_batch_destroy(b); return st; }
    b->met->uploaded[0] = b->met->uploaded[1] = true;   // the graph packs the bracket on the device
    b->pbl->ready = true;
    if (b->wet) b->wet->ready = true;
    const size_t nodes = nx * ny * nz, cells = nx * ny;
    const size_t grid_total = (size_t)cfg->out_nx * cfg->out_ny * cfg->out_nz * n_scen;
    cudaError_t e = cudaMalloc(&b->ring, nodes * cfg->n_frames * sizeof(float4));
    if (e == cudaSuccess) e = cudaMalloc(&b->sring, cells * cfg->n_frames * sizeof(fpg_surface_cell));
    if (e == cudaSuccess) e = cudaMalloc(&b->pring, cells * cfg->n_frames * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&b->staging, nodes * 3 * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&b->st, 2 * sizeof(BatchState));
    if (e == cudaSuccess) e = cudaMalloc(&b->error, sizeof(int32_t));
    if (e == cudaSuccess) e = cudaMemsetAsync(b->error, 0, sizeof(int32_t), ctx->stream);
    if (e == cudaSuccess) e = cudaMalloc(&b->sc, 2 * n_scen * sizeof(ScenDev));
    if (e == cudaSuccess) e = cudaMalloc(&b->tile_scen, b->n_tiles * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&b->grid_counts, (grid_total ? grid_total : 1) * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&b->grid_mass, (grid_total ? grid_total : 1) * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemsetAsync(b->pring, 0, cells * cfg->n_frames * sizeof(float), ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(b->grid_counts, 0, (grid_total ? grid_total : 1) * 4, ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(b->grid_mass, 0, (grid_total ? grid_total : 1) * 4, ctx->stream);
    BatchState s0;
    std::memset(&s0, 0, sizeof(s0));
    s0.t = cfg->start_seconds;
    if (e == cudaSuccess) e = cudaMemcpyAsync(b->st, &s0, sizeof(s0), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->sc, b->scen.data(), n_scen * sizeof(ScenDev), cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->tile_scen, b->tile_scen_h.data(), b->n_tiles * sizeof(uint32_t), cudaMemcpyHostToDevice,
                            ctx->stream);
    if (e == cudaSuccess) {
        enqueue_begin(b, ctx->stream);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) { fpg_batch_destroy(b); return cuda_status(e); }
    for (uint32_t v = 0; v < kNumVariants; ++v) {
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kVariants[v].kernel, (int)kVariants[v].block,
                                                          nz * sizeof(float) + FPG_LEVEL_BUCKETS);
        if (e != cudaSuccess) { fpg_batch_destroy(b); return cuda_status(e); }
        b->resident[v] = (uint32_t)std::max(per_sm, 1);
    }
    st = build_items(b, 0);
    if (st != FPG_OK) { fpg_batch_destroy(b); return st; }
    *out = b;
    return FPG_OK;
}

namespace fpg {
__global__ void __launch_bounds__(256) batch_pack_ring_kernel(const float* __restrict__ u, const float* __restrict__ v,
                                                              const float* __restrict__ w, uint32_t nodes, float4* out) {
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < nodes) out[n] = make_float4(u[n], v[n], w[n], 0.0f);
}
}  // namespace fpg

extern "C" fpg_status fpg_batch_upload_frame(fpg_batch* b, uint32_t k, const float* u, const float* v, const float* w,
                                             const fpg_surface_cell* surface, const float* precip) {
    if (!b || !u || !v || !w || !surface || k >= b->cfg.n_frames) return FPG_ERR_INVALID_ARGUMENT;
    cudaStream_t s = b->ctx->stream;
    const size_t nodes = b->met->nx * b->met->ny * b->met->nz, cells = b->met->nx * b->met->ny;
    FPG_CUDA(cudaMemcpyAsync(b->staging, u, nodes * 4, cudaMemcpyHostToDevice, s));
    FPG_CUDA(cudaMemcpyAsync(b->staging + nodes, v, nodes * 4, cudaMemcpyHostToDevice, s));
    FPG_CUDA(cudaMemcpyAsync(b->staging + 2 * nodes, w, nodes * 4, cudaMemcpyHostToDevice, s));
    batch_pack_ring_kernel<<<(unsigned)((nodes + 255) / 256), 256, 0, s>>>(b->staging, b->staging + nodes,
                                                                          b->staging + 2 * nodes, (uint32_t)nodes,
                                                                          b->ring + k * nodes);
    b->ctx->count();
    FPG_CHECK_LAUNCH();
    FPG_CUDA(cudaMemcpyAsync(b->sring + k * cells, surface, cells * sizeof(fpg_surface_cell), cudaMemcpyHostToDevice, s));
    if (precip) FPG_CUDA(cudaMemcpyAsync(b->pring + k * cells, precip, cells * 4, cudaMemcpyHostToDevice, s));
    FPG_CUDA(cudaStreamSynchronize(s));
    return FPG_OK;
}

extern "C" fpg_status fpg_batch_run(fpg_batch* b, uint32_t n_steps, int32_t use_graph) {
    if (!b) return FPG_ERR_INVALID_ARGUMENT;
    if (b->steps_done >= b->total_steps) return FPG_ERR_SIMULATION_COMPLETE;
    const uint64_t n = std::min<uint64_t>(n_steps, b->total_steps - b->steps_done);
    cudaStream_t s = b->ctx->stream;
    const bool form = pass_kernel(kVariants[b->variant], make_step_args(b)) != kVariants[b->variant].kernel;
    // every graph of the run before its first step: a capture that fails
    // leaves the batch as it was
    for (uint64_t i = 0; use_graph && i < n; ++i) {
        const fpg_status st = ensure_graph(b, b->steps_done + i, s);
        if (st != FPG_OK) return st;
    }
    fpg_status st = FPG_OK;
    uint64_t done = 0;
    for (; done < n; ++done) {
        const uint64_t step = b->steps_done + done;
        if (use_graph) {
            st = launch_step_graph(b, step, s);
        } else {
            enqueue_batched_step(b, s, step, output_step(b, step));
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) st = cuda_status(e);
        }
        if (st != FPG_OK) break;
        if (form) b->ctx->count_form(FPG_FORM_STEP);
    }
    // keep the host mirror (used by the sequential path) and the state's side
    // with the steps launched
    const uint32_t bpp = b->cfg.n_substeps <= 2u ? 1u : 2u;
    for (uint64_t i = 0; i < done; ++i) {
        for (size_t k = 0; k < b->scen.size(); ++k) {
            const ScenDev& d = b->scen[k];
            uint32_t hi = target_emitted(d.start, d.end, d.count, b->t_h, b->released_h[k]);
            if (hi > b->released_h[k]) b->released_h[k] = hi;
            b->counter_h[k] = counter_add64(b->counter_h[k], (uint64_t)d.capacity * bpp);
        }
        b->t_h += b->cfg.timestep_seconds;
    }
    b->steps_done += done;
    return st;
}

extern "C" fpg_status fpg_batch_run_sequential(fpg_batch* b, uint32_t n_steps) {
    if (!b) return FPG_ERR_INVALID_ARGUMENT;
    if (b->steps_done >= b->total_steps) return FPG_ERR_SIMULATION_COMPLETE;
    const uint64_t n = std::min<uint64_t>(n_steps, b->total_steps - b->steps_done);
    cudaStream_t s = b->ctx->stream;
    const uint32_t bpp = b->cfg.n_substeps <= 2u ? 1u : 2u;
    StepArgs base = make_step_args(b);
    // alpha of the step comes from the host clock (same formula as the device)
    for (uint64_t i = 0; i < n; ++i) {
        const bool output = output_step(b, b->steps_done + i);
        const uint32_t side = (uint32_t)((b->steps_done + i) & 1u);
        enqueue_pre(b, s, side, output, nullptr, nullptr, 0);
        int64_t k = (b->t_h - b->cfg.start_seconds) / b->cfg.frame_seconds;
        if (b->t_h - b->cfg.start_seconds == k * b->cfg.frame_seconds && k > 0) k -= 1;
        const int64_t ta = b->cfg.start_seconds + k * b->cfg.frame_seconds;
        const float alpha = (float)((double)(b->t_h - ta) / (double)b->cfg.frame_seconds);
        for (size_t sidx = 0; sidx < b->scen.size(); ++sidx) {
            const ScenDev& d = b->scen[sidx];
            uint32_t hi = target_emitted(d.start, d.end, d.count, b->t_h, b->released_h[sidx]);
            if (hi > b->released_h[sidx]) b->released_h[sidx] = hi;
            const uint32_t released = b->released_h[sidx];
            const u32x4 counter = b->counter_h[sidx];
            // the counter advances every step, released particles or not (as the driver's)
            b->counter_h[sidx] = counter_add64(counter, (uint64_t)d.capacity * bpp);
            if (released == 0) continue;
            // one launch of the step over this scenario's segment, as fpg_step makes it
            StepArgs a = base;
            const uint32_t o = d.offset;
            a.cell_x += o; a.cell_y += o; a.pos_x += o; a.pos_y += o; a.pos_z += o; a.flags += o;
            for (int m = 0; m < 4; ++m) a.mass[m] += o;
            a.vel_u += o; a.vel_v += o; a.vel_w += o; a.turb_u += o; a.turb_v += o; a.turb_w += o; a.cbt += o;
            a.n = released;
            a.alpha = alpha;
            a.key0 = d.key0; a.key1 = d.key1;
            a.counter = counter;
            const fpg_status st = launch_step(b->ctx, a, s);
            if (st != FPG_OK) return st;
        }
        enqueue_post(b, s, side, output);
        FPG_CHECK_LAUNCH();
        b->t_h += b->cfg.timestep_seconds;
    }
    b->steps_done += n;
    return FPG_OK;
}

extern "C" uint64_t fpg_batch_steps_done(const fpg_batch* b) { return b ? b->steps_done : 0; }

extern "C" fpg_status fpg_batch_scenario_slots(const fpg_batch* b, size_t s, size_t* first, size_t* count) {
    if (!b || s >= b->scen.size() || !first || !count) return FPG_ERR_INVALID_ARGUMENT;
    *first = b->scen[s].offset;
    *count = b->scen[s].capacity;
    return FPG_OK;
}

extern "C" fpg_particles* fpg_batch_particles(fpg_batch* b) { return b ? b->pop : nullptr; }

extern "C" fpg_status fpg_batch_download_grids(fpg_batch* b, uint32_t* counts, uint32_t* mass) {
    if (!b) return FPG_ERR_INVALID_ARGUMENT;
    const size_t total = (size_t)b->cfg.out_nx * b->cfg.out_ny * b->cfg.out_nz * b->scen.size();
    cudaStream_t s = b->ctx->stream;
    if (counts) FPG_CUDA(cudaMemcpyAsync(counts, b->grid_counts, total * 4, cudaMemcpyDeviceToHost, s));
    if (mass) FPG_CUDA(cudaMemcpyAsync(mass, b->grid_mass, total * 4, cudaMemcpyDeviceToHost, s));
    FPG_CUDA(cudaStreamSynchronize(s));
    return FPG_OK;
}

extern "C" fpg_status fpg_batch_errors(fpg_batch* b, int32_t* flags) {
    if (!b || !flags) return FPG_ERR_INVALID_ARGUMENT;
    FPG_CUDA(cudaMemcpyAsync(flags, b->error, sizeof(int32_t), cudaMemcpyDeviceToHost, b->ctx->stream));
    FPG_CUDA(cudaStreamSynchronize(b->ctx->stream));
    return FPG_OK;
}

// ---- launch-shape tuner ------------------------------------------------------

extern "C" uint32_t fpg_batch_tuning_candidates(fpg_batch_tuning* out, uint32_t max) {
    for (uint32_t v = 0; out && v < kNumVariants && v < max; ++v)
        out[v] = fpg_batch_tuning{kVariants[v].block, kVariants[v].minb, kVariants[v].ppt, 0.0f};
    return kNumVariants;
}

static int find_variant(const fpg_batch_tuning* t) {
    for (uint32_t v = 0; v < kNumVariants; ++v)
        if (kVariants[v].block == t->block_threads && kVariants[v].minb == t->min_blocks_per_sm &&
            kVariants[v].ppt == t->particles_per_thread)
            return (int)v;
    return -1;
}

extern "C" fpg_status fpg_batch_set_tuning(fpg_batch* b, const fpg_batch_tuning* t) {
    if (!b || !t) return FPG_ERR_INVALID_ARGUMENT;
    const int v = find_variant(t);
    if (v < 0) return FPG_ERR_INVALID_ARGUMENT;
    b->tuned_ms = t->step_ms;
    return build_items(b, (uint32_t)v);
}

extern "C" fpg_status fpg_batch_get_tuning(const fpg_batch* b, fpg_batch_tuning* t) {
    if (!b || !t) return FPG_ERR_INVALID_ARGUMENT;
    const StepVariant& v = kVariants[b->variant];
    *t = fpg_batch_tuning{v.block, v.minb, v.ppt, b->tuned_ms};
    return FPG_OK;
}

// Times the particle pass of the next step under every compiled launch
// shape, each from the same snapshot of the live state (population, clock,
// release and counter state), restores the snapshot and keeps the fastest
// shape; two shapes that run one kernel are timed once.  Each particle's
// arithmetic does not depend on the launch shape, so the choice changes speed
// only, never results.
extern "C" fpg_status fpg_batch_autotune(fpg_batch* b, uint32_t reps, fpg_batch_tuning* results, uint32_t max_results,
                                         fpg_batch_tuning* best) {
    if (!b) return FPG_ERR_INVALID_ARGUMENT;
    if (b->steps_done >= b->total_steps) return FPG_ERR_SIMULATION_COMPLETE;
    if (reps == 0) reps = 1;
    cudaStream_t s = b->ctx->stream;
    const size_t pop_bytes = particles_block_bytes(b->capacity);
    const size_t sc_bytes = 2 * b->scen.size() * sizeof(ScenDev), st_bytes = 2 * sizeof(BatchState);
    const uint32_t side = (uint32_t)(b->steps_done & 1u);
    void* snap = nullptr;
    BatchState* st_snap = nullptr;
    ScenDev* sc_snap = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    fpg_status status = FPG_OK;
    uint32_t best_v = b->variant;
    float best_ms = 0.0f;
    cudaError_t e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaMalloc(&snap, pop_bytes);
    if (e == cudaSuccess) e = cudaMalloc(&st_snap, st_bytes);
    if (e == cudaSuccess) e = cudaMalloc(&sc_snap, sc_bytes);
    if (e == cudaSuccess) e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    if (e == cudaSuccess) e = cudaMemcpyAsync(snap, b->pop->block, pop_bytes, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(st_snap, b->st, st_bytes, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(sc_snap, b->sc, sc_bytes, cudaMemcpyDeviceToDevice, s);
    auto restore = [&]() {
        cudaError_t r = cudaMemcpyAsync(b->pop->block, snap, pop_bytes, cudaMemcpyDeviceToDevice, s);
        if (r == cudaSuccess) r = cudaMemcpyAsync(b->st, st_snap, st_bytes, cudaMemcpyDeviceToDevice, s);
        if (r == cudaSuccess) r = cudaMemcpyAsync(b->sc, sc_snap, sc_bytes, cudaMemcpyDeviceToDevice, s);
        return r;
    };
    const StepArgs args = make_step_args(b);
    float time_of[kNumVariants] = {};
    for (uint32_t v = 0; e == cudaSuccess && status == FPG_OK && v < kNumVariants; ++v) {
        uint32_t same = 0;                               // the first shape that runs this kernel
        while (pass_kernel(kVariants[same], args) != pass_kernel(kVariants[v], args)) ++same;
        float& tmin = time_of[v];
        if (same < v) tmin = time_of[same]; else status = build_items(b, v);
        for (uint32_t r = 0; same == v && status == FPG_OK && e == cudaSuccess && r < reps; ++r) {
            e = restore();
            if (e != cudaSuccess) break;
            enqueue_pre(b, s, side, false, nullptr, nullptr, 0);
            e = cudaEventRecord(e0, s);
            if (e != cudaSuccess) break;
            enqueue_step_kernel(b, s, side);
            e = cudaGetLastError();
            if (e == cudaSuccess) e = cudaEventRecord(e1, s);
            if (e == cudaSuccess) e = cudaEventSynchronize(e1);
            float ms = 0.0f;
            if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
            if (e == cudaSuccess && (r == 0 || ms < tmin)) tmin = ms;
        }
        if (e != cudaSuccess || status != FPG_OK) break;
        if (results && v < max_results)
            results[v] = fpg_batch_tuning{kVariants[v].block, kVariants[v].minb, kVariants[v].ppt, tmin};
        if (v == 0 || tmin < best_ms) { best_ms = tmin; best_v = v; }
    }
    if (e == cudaSuccess) e = restore();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(snap); cudaFree(st_snap); cudaFree(sc_snap);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (e != cudaSuccess) return cuda_status(e);
    if (status != FPG_OK) return status;
    status = build_items(b, best_v);
    b->tuned_ms = best_ms;
    if (best) fpg_batch_get_tuning(b, best);
    return status;
}
