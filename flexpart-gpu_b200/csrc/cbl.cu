// cbl.cu — convective-boundary-layer sampling and convective mixing
// (the per-slot Hanna records they read come from fpg_dispatch_hanna_params,
// built with the step in step.cu):
//
// * fpg_cbl_sample: the bi-Gaussian vertical-velocity PDF of the CBL and one
//   sampled w' per slot from caller uniforms (cbl.wgsl, src/gpu/cbl.rs);
// * fpg_cbl_sample_philox: the same sample fused with the Hanna sigma_w at
//   the particle's cell and Philox uniforms, so the per-slot 64-byte Hanna
//   record and the 16-byte uniform record never go through HBM;
// * fpg_convection_*: the column redistribution matrix applied to particle
//   heights (convective_mixing.wgsl, src/gpu/convection.rs).  The expected
//   destination height depends only on the source level, so it is computed
//   once per level when the matrix is set (one thread per level, the same
//   sequential f32 sum the reference runs per particle); the per-particle
//   kernel is a level search plus one table read: 8 bytes read and 8 bytes
//   written per active slot, four slots per thread, HBM-bound.
//
// The PDF follows the CPU routine (physics/cbl.rs:126-226): cbrt for the
// signed cube root and repeated multiplication for powi(3) / powi(2); the
// shader's pow() forms agree within the 5e-5 relative tolerance its own GPU
// test allows (src/gpu/cbl.rs:446-515).
#include <cmath>
#include <cstring>
#include <vector>

#include "fpg_internal.h"
#include "physics.cuh"
#include "slots.cuh"

namespace fpg {
namespace {

constexpr float kMinH = 1.0f;
constexpr float kMinSigmaW = 1.0e-5f;
constexpr float kSkewEps = 1.0e-6f;
constexpr float kW3Eps = 1.0e-6f;
constexpr float kFluarw = 2.0f / 3.0f;
constexpr float kPi = 3.14159265358979323846f;   // std::f32::consts::PI

// cbl_transition_factor (physics/cbl.rs:109-124, cbl.wgsl:133-146).
__device__ __forceinline__ float cbl_transition(float h, float ol) {
    if (!finitef(h) || h <= 0.0f || !finitef(ol) || ol == 0.0f) return 1.0f;
    const float ratio = -h / ol;
    const float t = ratio < 15.0f ? sinf(((ratio + 10.0f) / 10.0f) * kPi) * 0.5f + 0.5f : 1.0f;
    return clampf(t, 0.0f, 1.0f);
}

// CblSamplingOutput field order (src/gpu/cbl.rs:66-92) minus the sample.
struct CblPdf {
    float aw, am, as, bw, bm, bs, w2, w3, skew, trans, zoh;
};

// compute_cbl_moments + compute_cbl_bigaussian_pdf (physics/cbl.rs:126-226).
__device__ __forceinline__ CblPdf cbl_pdf(float z_in, float h_in, float wst_in, float sigw_in, float ol) {
    const float h = fmaxf(h_in, kMinH);
    const float z = clampf(z_in, 0.0f, h);
    const float zoh = z / h;
    const float wst = fmaxf(wst_in, 0.0f);
    const float sw = fmaxf(sigw_in, kMinSigmaW);
    const float trans = cbl_transition(h, ol);
    const float w2 = sw * sw;
    const float shape = 1.2f * zoh * powf(1.0f - zoh, 1.5f) + kW3Eps;
    const float w3 = shape * (wst * wst * wst) * trans;
    const float skew = w3 / powf(w2, 1.5f);
    CblPdf p{0.5f, 0.0f, sw, 0.5f, 0.0f, sw, w2, w3, skew, trans, zoh};
    if (!finitef(skew) || fabsf(skew) <= kSkewEps) return p;
    const float fl = kFluarw * cbrtf(skew);
    const float fl2 = fl * fl;
    if (!finitef(fl) || fabsf(fl) <= kSkewEps) return p;
    const float skew2 = skew * skew;
    const float a1 = 1.0f + fl2, a3 = 3.0f + fl2;
    const float num = (a1 * a1 * a1) * skew2;
    const float den = (a3 * a3) * fl2;
    const float r = fmaxf(num / fmaxf(den, kSkewEps), 0.0f);
    const float x = sqrtf(r);
    const float aw = clampf(0.5f * (1.0f - x / sqrtf(4.0f + r)), 1.0e-4f, 1.0f - 1.0e-4f);
    const float bw = 1.0f - aw;
    const float sa = sw * sqrtf(bw / (aw * (1.0f + fl2)));
    const float sb = sw * sqrtf(aw / (bw * (1.0f + fl2)));
    p.aw = aw; p.am = fl * sa; p.as = fmaxf(sa, kMinSigmaW);
    p.bw = bw; p.bm = -(fl * sb); p.bs = fmaxf(sb, kMinSigmaW);
    return p;
}

// sample_cbl_vertical_velocity (physics/cbl.rs:274-288, cbl.wgsl:270-277).
__device__ __forceinline__ float cbl_draw(const CblPdf& p, float ub, float eta) {
    return ub < p.aw ? p.am + p.as * eta : p.bm + p.bs * eta;
}

// Three 16-byte stores per slot (moving them through shared memory into
// whole lines measured 8 % slower: the kernel issues more than it stores).
__device__ __forceinline__ void store_output(fpg_cbl_sampling_output* out, size_t p, const float4 (&row)[3]) {
    float4* o = reinterpret_cast<float4*>(out + p);
    o[0] = row[0];
    o[1] = row[1];
    o[2] = row[2];
}

__device__ __forceinline__ void output_row(float w, const CblPdf& p, float4 (&row)[3]) {
    row[0] = make_float4(w, p.aw, p.am, p.as);
    row[1] = make_float4(p.bw, p.bm, p.bs, p.w2);
    row[2] = make_float4(p.w3, p.skew, p.trans, p.zoh);
}

// cbl.wgsl:251-298: PDF from the slot's Hanna record, sample from its uniforms.
__global__ void __launch_bounds__(256) cbl_sample_kernel(SlotView v, const fpg_hanna_params* hanna,
                                                         const fpg_cbl_sampling_input* in,
                                                         fpg_cbl_sampling_output* out) {
    chain_begin();
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= v.n) return;
    float4 row[3] = {};
    if (v.flags[p] & FLAG_ACTIVE) {
        const float4 h0 = *reinterpret_cast<const float4*>(hanna + p);       // ust, wst, ol, h
        const float sigw = hanna[p].sigw;
        const float4 u = *reinterpret_cast<const float4*>(in + p);
        const CblPdf pdf = cbl_pdf(v.pos_z[p], h0.w, h0.y, sigw, h0.z);
        output_row(cbl_draw(pdf, u.x, box_muller(u.y, u.z).x), pdf, row);
    }
    store_output(out, p, row);
}

// The fused form: sigma_w of compute_hanna at the slot's cell (the vertical
// branch of hanna_short_w gives the same sigma_w bits as compute_hanna) from
// the cell's Hanna constants (the floored u*, w*, h, the Obukhov length, the
// regime and the constant products the PBL pass stores per cell, so the
// per-cell part is not redone per slot), and the uniforms of one Philox
// block at counter + slot: u0, u1, u2 of PhiloxRng::next_uniform4 on a
// stream that starts at that counter (physics/cbl.rs:291-295,
// physics/rng.rs:130-164).
// `head_ok`: no block's counter carries, and Philox starts after its uniform
// rounds.
__global__ void __launch_bounds__(256) cbl_sample_philox_kernel(SlotView v, const CellHanna* hcell, uint32_t pnx,
                                                                uint32_t pny, uint32_t k0, uint32_t k1, u32x4 counter,
                                                                PhiloxHead head, PhiloxKeys keys, int head_ok,
                                                                fpg_cbl_sampling_output* out) {
    chain_begin();
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= v.n) return;
    float4 row[3] = {};
    if (v.flags[p] & FLAG_ACTIVE) {
        const CellHanna cell = ld_cell_hanna(hcell + pbl_cell_index(v, p, pnx, pny));
        const float z = v.pos_z[p];
        float sigw, dsigwdz, tlw;
        hanna_short_cell_t<float>(cell, z, sigw, dsigwdz, tlw);
        const u32x4 b = head_ok ? philox_from_head(head, keys, counter.x + (uint32_t)p)
                                : philox4x32_10(counter_add(counter, (uint32_t)p), k0, k1);
        const CblPdf pdf = cbl_pdf(z, cell.h, cell.wst, sigw, cell.ol);
        output_row(cbl_draw(pdf, u32_to_uniform01(b.x), box_muller_plain(b.y, b.z).x), pdf, row);
    }
    store_output(out, p, row);
}

// expected_destination_height_m (physics/convection.rs:398-427): one thread
// per source level sums its matrix column in destination order, as the
// shader's per-particle loop does (convective_mixing.wgsl:98-104), then
// clamps to the column (the shader's clamp of the quotient).
__global__ void conv_heights_kernel(uint32_t L, const float* __restrict__ m, const float* __restrict__ centers,
                                    float z_min, float z_max, float* __restrict__ heights) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= L) return;
    float wh = 0.0f, ws = 0.0f;
    const float* col = m + (size_t)s * L;
    for (uint32_t d = 0; d < L; ++d) {
        const float w = fmaxf(col[d], 0.0f);
        wh = wh + w * centers[d];
        ws = ws + w;
    }
    heights[s] = ws > 0.0f ? clampf(wh / ws, z_min, z_max) : 0.0f;
}

// convective_mixing.wgsl:87-113 per active slot.  With strictly increasing
// finite interfaces the shader's linear scan (first level with
// lower <= z < upper, else the top level) is the last level whose lower
// interface is <= z: a bucket table gives a level at most a few below it
// (entry b is the last level whose lower interface lies at or below the lower
// edge of bucket b - 1, so rounding of the bucket index cannot pass it) and
// the search scans up, one comparison or two where a bisection of 60 levels
// takes six dependent loads.  A column whose bucket width is not a normal
// float, or with more than kMixScan levels in three adjacent buckets (the
// longest scan: about as many loads as a bisection of those columns, which
// have 1000s of levels or crowd them), is bisected; without sorted interfaces
// the scan over all levels runs.
enum { MIX_SCAN = 0, MIX_BISECT = 1, MIX_TABLE = 2 };
constexpr uint32_t kMixBuckets = 1024, kMixScan = 8;

struct MixColumn {
    const float* iface;                  // L + 1
    const float* heights;                // L: the mixed height of every source level
    const uint16_t* table;               // kMixBuckets
    float inv_w;
    uint32_t L;
};

template <int kSearch>
__device__ __forceinline__ uint32_t source_level(float z, float z_min, const MixColumn& c) {
    if constexpr (kSearch == MIX_TABLE) {
        const uint32_t b = min(__float2uint_rz((z - z_min) * c.inv_w), kMixBuckets - 1u);
        uint32_t lo = c.table[b];
        while (lo + 1u < c.L && c.iface[lo + 1u] <= z) ++lo;
        return lo;
    } else if constexpr (kSearch == MIX_BISECT) {
        uint32_t lo = 0u, hi = c.L;               // count of iface[0..L) <= z lies in [1, L]
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (c.iface[mid] <= z) lo = mid; else hi = mid;
        }
        return lo;
    } else {
        for (uint32_t l = 0; l < c.L; ++l)
            if (z >= c.iface[l] && z < c.iface[l + 1u]) return l;
        return c.L - 1u;
    }
}

// The mixed height and the source level of one active slot (a column that
// passed fpg_convection_set_matrix always has a positive weight).
template <int kSearch>
__device__ __forceinline__ float mix_height(float z_in, float z_min, float z_max, const MixColumn& c, int32_t& level_out) {
    const uint32_t level = source_level<kSearch>(clampf(z_in, z_min, z_max), z_min, c);
    level_out = (int32_t)level;
    return c.heights[level];
}

// Four slots per thread: the flags and heights of a quad arrive in one
// 16-byte load each (the fields are 256-byte aligned); a quad of active
// slots is written with one 16-byte store per field, otherwise only the
// active slots are written.  The last n % 4 slots take scalar loads.
template <int kSearch>
__global__ void __launch_bounds__(256) conv_apply_kernel(size_t n, const uint32_t* flags, float* pos_z, int32_t* cbt,
                                                         MixColumn c) {
    chain_begin();
    const size_t p0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4u;
    if (p0 >= n) return;
    const float z_min = c.iface[0], z_max = c.iface[c.L];
    if (p0 + 4u <= n) {
        const uint4 f = *reinterpret_cast<const uint4*>(flags + p0);
        const float4 z = *reinterpret_cast<const float4*>(pos_z + p0);
        int4 lv;
        float4 zo;
        zo.x = mix_height<kSearch>(z.x, z_min, z_max, c, lv.x);
        zo.y = mix_height<kSearch>(z.y, z_min, z_max, c, lv.y);
        zo.z = mix_height<kSearch>(z.z, z_min, z_max, c, lv.z);
        zo.w = mix_height<kSearch>(z.w, z_min, z_max, c, lv.w);
        if (f.x & f.y & f.z & f.w & FLAG_ACTIVE) {
            *reinterpret_cast<float4*>(pos_z + p0) = zo;
            *reinterpret_cast<int4*>(cbt + p0) = lv;
            return;
        }
        if (f.x & FLAG_ACTIVE) { pos_z[p0] = zo.x; cbt[p0] = lv.x; }
        if (f.y & FLAG_ACTIVE) { pos_z[p0 + 1] = zo.y; cbt[p0 + 1] = lv.y; }
        if (f.z & FLAG_ACTIVE) { pos_z[p0 + 2] = zo.z; cbt[p0 + 2] = lv.z; }
        if (f.w & FLAG_ACTIVE) { pos_z[p0 + 3] = zo.w; cbt[p0 + 3] = lv.w; }
    } else {
        for (size_t p = p0; p < n; ++p)
            if (flags[p] & FLAG_ACTIVE) {
                int32_t level;
                pos_z[p] = mix_height<kSearch>(pos_z[p], z_min, z_max, c, level);
                cbt[p] = level;
            }
    }
}

}  // namespace
}  // namespace fpg

using namespace fpg;

struct fpg_convection {
    fpg_ctx* ctx = nullptr;
    size_t levels = 0;
    float* matrix = nullptr;        // levels^2, column-major (source * levels + destination)
    float* iface = nullptr;         // levels + 1, and in the same block:
    float* centers = nullptr;       // levels
    uint16_t* table = nullptr;      // kMixBuckets: the level search (MIX_TABLE)
    float* heights = nullptr;       // levels: expected destination height per source level
    float inv_w = 0.0f;
    int search = MIX_SCAN;
    bool ready = false;
};

// Bytes of a column of L levels: interfaces, centres, bucket table.
static size_t column_bytes(size_t L) { return (2 * L + 1) * sizeof(float) + kMixBuckets * sizeof(uint16_t); }

extern "C" fpg_status fpg_cbl_sample(fpg_ctx* ctx, const fpg_particles* P, const fpg_hanna_params* hanna_dev,
                                     size_t n_hanna, const fpg_cbl_sampling_input* inputs_dev, size_t n_inputs,
                                     fpg_cbl_sampling_output* out_dev, void* stream) {
    if (!ctx || !P) return FPG_ERR_INVALID_ARGUMENT;
    const SlotView v = slot_view(P);
    // GpuCblError::MismatchedInputLengths (src/gpu/cbl.rs:210-216)
    if (n_hanna != v.n || n_inputs != v.n) return FPG_ERR_LENGTH_MISMATCH;
    if (v.n == 0) return FPG_OK;
    if (!hanna_dev || !inputs_dev || !out_dev) return FPG_ERR_INVALID_ARGUMENT;
    if (!aligned16(hanna_dev) || !aligned16(inputs_dev) || !aligned16(out_dev)) return FPG_ERR_INVALID_ARGUMENT;
    if (v.n > UINT32_MAX) return FPG_ERR_VALUE_TOO_LARGE;
    launch_chained(cbl_sample_kernel, (unsigned)((v.n + 255) / 256), 256, 0, ctx->pick(stream), v, hanna_dev, inputs_dev, out_dev);
    ctx->count();
    FPG_CHECK_LAUNCH();
    return FPG_OK;
}

extern "C" fpg_status fpg_cbl_sample_philox(fpg_ctx* ctx, const fpg_particles* P, const fpg_pbl* pbl,
                                            const uint32_t key[2], const uint32_t counter[4],
                                            fpg_cbl_sampling_output* out_dev, void* stream) {
    if (!ctx || !P || !pbl || !key || !counter) return FPG_ERR_INVALID_ARGUMENT;
    if (pbl->nx == 0 || pbl->ny == 0) return FPG_ERR_ZERO_SHAPE;
    if (pbl->nx > UINT32_MAX || pbl->ny > UINT32_MAX || P->dispatch > UINT32_MAX) return FPG_ERR_VALUE_TOO_LARGE;
    if (!pbl->ready) return FPG_ERR_NOT_READY;
    const SlotView v = slot_view(P);
    if (v.n == 0) return FPG_OK;
    if (!out_dev || !aligned16(out_dev)) return FPG_ERR_INVALID_ARGUMENT;
    const u32x4 c{counter[0], counter[1], counter[2], counter[3]};
    const PhiloxHead head = philox_head(c, key[0], key[1]);
    const int head_ok = (uint64_t)c.x + v.n <= (1ull << 32);
    launch_chained(cbl_sample_philox_kernel, (unsigned)((v.n + 255) / 256), 256, 0, ctx->pick(stream), v, pbl->hanna,
                   (uint32_t)pbl->nx, (uint32_t)pbl->ny, key[0], key[1], c, head, philox_keys(head), head_ok, out_dev);
    ctx->count();
    FPG_CHECK_LAUNCH();
    return FPG_OK;
}

extern "C" fpg_status fpg_convection_create(fpg_ctx* ctx, size_t level_count, fpg_convection** out) {
    if (!ctx || !out) return FPG_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    // GpuConvectionError::InvalidLevelCount (src/gpu/convection.rs:74-79)
    if (level_count == 0) return FPG_ERR_ZERO_SHAPE;
    if (level_count > (size_t)INT32_MAX || level_count > (size_t)65535) return FPG_ERR_VALUE_TOO_LARGE;
    auto* c = new fpg_convection;
    c->ctx = ctx;
    c->levels = level_count;
    const size_t L = level_count;
    cudaError_t e = cudaMalloc(&c->matrix, L * L * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&c->iface, column_bytes(L));
    if (e == cudaSuccess) e = cudaMalloc(&c->heights, L * sizeof(float));
    if (e != cudaSuccess) {
        fpg_convection_destroy(c);
        return cuda_status(e);
    }
    c->centers = c->iface + L + 1;
    c->table = reinterpret_cast<uint16_t*>(c->centers + L);
    *out = c;
    return FPG_OK;
}

extern "C" fpg_status fpg_convection_destroy(fpg_convection* c) {
    if (!c) return FPG_ERR_INVALID_ARGUMENT;
    cudaFree(c->matrix);
    cudaFree(c->iface);
    cudaFree(c->heights);
    delete c;
    return FPG_OK;
}

extern "C" fpg_status fpg_convection_set_matrix(fpg_convection* c, const float* matrix_column_major,
                                                size_t n_matrix, const float* level_interfaces_m,
                                                size_t n_interfaces, void* stream) {
    if (!c || !matrix_column_major || !level_interfaces_m) return FPG_ERR_INVALID_ARGUMENT;
    const size_t L = c->levels;
    // ConvectionError::MatrixLengthMismatch (physics/convection.rs:163-170) and
    // GpuConvectionError::InvalidLevelInterfaces (src/gpu/convection.rs:81-86)
    if (n_matrix != L * L || n_interfaces != L + 1) return FPG_ERR_LENGTH_MISMATCH;
    // validate_column_stochasticity (physics/convection.rs:196-218): the
    // reference's matrix type holds this invariant from construction.
    for (size_t s = 0; s < L; ++s) {
        float sum = 0.0f;
        for (size_t d = 0; d < L; ++d) {
            const float w = matrix_column_major[s * L + d];
            if (w < -1.0e-4f || !std::isfinite(w)) return FPG_ERR_NON_STOCHASTIC_COLUMN;
            sum += w;
        }
        if (std::fabs(sum - 1.0f) > 1.0e-4f) return FPG_ERR_NON_STOCHASTIC_COLUMN;
    }
    bool sorted = true;
    for (size_t l = 0; l <= L; ++l) {
        if (!std::isfinite(level_interfaces_m[l]) || (l > 0 && !(level_interfaces_m[l] > level_interfaces_m[l - 1])))
            sorted = false;
    }
    // interfaces, centres (level_centers_from_interfaces, src/gpu/convection.rs:63-69)
    // and the bucket table (in double), one copy
    std::vector<float> column(column_bytes(L) / sizeof(float));
    float* centers = column.data() + L + 1;
    uint16_t* table = reinterpret_cast<uint16_t*>(centers + L);
    std::memcpy(column.data(), level_interfaces_m, (L + 1) * sizeof(float));
    for (size_t l = 0; l < L; ++l) centers[l] = 0.5f * (level_interfaces_m[l] + level_interfaces_m[l + 1]);
    int search = sorted ? MIX_BISECT : MIX_SCAN;
    const double span = (double)level_interfaces_m[L] - (double)level_interfaces_m[0];
    const float inv_w = sorted ? (float)(kMixBuckets / span) : 0.0f;
    if (sorted && std::isnormal(inv_w) && std::isfinite((float)span)) {
        search = MIX_TABLE;
        uint32_t last[3] = {}, l = 0;                   // the levels at the three buckets' edges below
        for (uint32_t b = 0; b < kMixBuckets + 3u; ++b) {
            const double edge = (double)level_interfaces_m[0] + ((double)b - 1.0) * (span / kMixBuckets);
            while (l + 1u < L && (double)level_interfaces_m[l + 1u] <= edge) ++l;
            if (b < kMixBuckets) table[b] = (uint16_t)l;
            if (l - last[b % 3u] > kMixScan) search = MIX_BISECT;
            last[b % 3u] = l;
        }
    }
    cudaStream_t s = c->ctx->pick(stream);
    FPG_CUDA(cudaMemcpyAsync(c->matrix, matrix_column_major, L * L * sizeof(float), cudaMemcpyHostToDevice, s));
    FPG_CUDA(cudaMemcpyAsync(c->iface, column.data(), column_bytes(L), cudaMemcpyHostToDevice, s));
    conv_heights_kernel<<<(unsigned)((L + 127) / 128), 128, 0, s>>>((uint32_t)L, c->matrix, c->centers,
                                                                   level_interfaces_m[0], level_interfaces_m[L],
                                                                   c->heights);
    c->ctx->count();
    FPG_CHECK_LAUNCH();
    // the host vectors are released on return: wait for their copies
    FPG_CUDA(cudaStreamSynchronize(s));
    c->search = search;
    c->inv_w = inv_w;
    c->ready = true;
    return FPG_OK;
}

extern "C" fpg_status fpg_convection_heights(const fpg_convection* c, float* heights_host) {
    if (!c || !heights_host) return FPG_ERR_INVALID_ARGUMENT;
    if (!c->ready) return FPG_ERR_NOT_READY;
    FPG_CUDA(cudaMemcpy(heights_host, c->heights, c->levels * sizeof(float), cudaMemcpyDeviceToHost));
    return FPG_OK;
}

extern "C" fpg_status fpg_convective_mixing(fpg_ctx* ctx, fpg_particles* P, const fpg_convection* c, void* stream) {
    if (!ctx || !P || !c) return FPG_ERR_INVALID_ARGUMENT;
    if (!c->ready) return FPG_ERR_NOT_READY;
    const size_t n = P->dispatch;
    if (n == 0) return FPG_OK;
    if (n > UINT32_MAX) return FPG_ERR_VALUE_TOO_LARGE;
    const auto* flags = static_cast<const uint32_t*>(P->field[FPG_FIELD_FLAGS]);
    auto* pos_z = static_cast<float*>(P->field[FPG_FIELD_POS_Z]);
    auto* cbt = static_cast<int32_t*>(P->field[FPG_FIELD_CBT]);
    const unsigned grid = (unsigned)(((n + 3) / 4 + 255) / 256);
    const MixColumn column{c->iface, c->heights, c->table, c->inv_w, (uint32_t)c->levels};
    const auto kernel = c->search == MIX_TABLE    ? conv_apply_kernel<MIX_TABLE>
                        : c->search == MIX_BISECT ? conv_apply_kernel<MIX_BISECT>
                                                  : conv_apply_kernel<MIX_SCAN>;
    launch_chained(kernel, grid, 256, 0, ctx->pick(stream), n, flags, pos_z, cbt, column);
    ctx->count();
    FPG_CHECK_LAUNCH();
    return FPG_OK;
}
