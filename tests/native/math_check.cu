// math_check.cu — the step's own square root, reciprocal product and
// Box-Muller forms over their whole input ranges, against sqrtf, the step's
// division and the general Box-Muller (which the CPU tests hold to the exact
// values).  Built twice, with the flags of the step's units and with those of
// the others (MATH_CHECK names the two).
#include <cstdint>
#include <cuda_runtime.h>

#include "physics.cuh"

using namespace fpg;

namespace {

constexpr unsigned kThreads = 256, kBlocks = 2048;
constexpr uint32_t kWords = 1u << 24;                  // the distinct words of a 24-bit uniform, v = k << 8

struct Result {
    unsigned long long differ;                         // inputs with another bit pattern
    unsigned long long first;                          // the smallest of them
};

__device__ void report(Result* r, unsigned long long input) {
    atomicAdd(&r->differ, 1ull);
    atomicMin(&r->first, input);
}

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ bool same(float2 a, float2 b) { return same(a.x, b.x) && same(a.y, b.y); }

// Every float of [2^-100, 2^100].
__global__ void root_kernel(Result* r) {
    const uint32_t lo = __float_as_uint(0x1p-100f), hi = __float_as_uint(0x1p100f);
    for (uint64_t b = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b <= hi; b += (uint64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((uint32_t)b);
        if (!same(plain_sqrt(x), sqrtf(x))) report(r, b);
    }
}

#ifdef FPG_RECIPROCAL_DIVISION
// a * rcp_of(b) against the step's division: every significand of a, each
// with 64 divisors spread over the floats of [1e-4, 1e6] by a multiplicative
// hash.
__global__ void quotient_kernel(Result* r) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 1u << 29; i += gridDim.x * blockDim.x) {
        const uint32_t h = i * 2654435761u;
        const float a = __uint_as_float(0x3f800000u | (i & 0x7fffffu));
        const uint32_t lo = __float_as_uint(1.0e-4f), hi = __float_as_uint(1.0e6f);
        const float b = __uint_as_float(lo + __umulhi(h ^ (i >> 23), hi - lo + 1u));
        if (!same(a * rcp_of(b), sdiv(a, b))) report(r, i);
    }
}
#endif

// The radius: every radius word at the angle 0, whose cosine is 1.
__global__ void radius_kernel(Result* plain, Result* first, Result* second) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < kWords; k += gridDim.x * blockDim.x) {
        const float2 want = box_muller(u32_to_uniform01(k << 8), 0.0f);
        const uint2 word = make_uint2(k << 8, 0u), other = make_uint2(~(k << 8), k << 8);
        float2 a, b, c, d;
        box_muller2(word, other, a, b);
        box_muller2(other, word, c, d);
        if (!same(box_muller_plain(word.x, word.y), want)) report(plain, k);
        if (!same(a, want) || !same(d, box_muller(u32_to_uniform01(word.x), 0.0f))) report(first, k);
        if (!same(b, box_muller(u32_to_uniform01(other.x), u32_to_uniform01(other.y))) || !same(c, b)) report(second, k);
    }
}

// A radius word whose radius is exactly 1, so that a product is the cosine or
// the sine itself; 0 if there is none.
__global__ void unit_radius_kernel(uint32_t* word) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < kWords; k += gridDim.x * blockDim.x)
        if (box_muller(u32_to_uniform01(k << 8), 0.0f).x == 1.0f) atomicMax(word, k << 8);
}

// The cosine and sine: every angle word, at radius 1 and at `radius`.
__global__ void angle_kernel(const uint32_t* unit, uint32_t radius, Result* plain, Result* first, Result* second) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < kWords; k += gridDim.x * blockDim.x) {
        const uint2 p = make_uint2(*unit, k << 8), q = make_uint2(radius, k << 8);
        const float2 wp = box_muller(u32_to_uniform01(p.x), u32_to_uniform01(p.y));
        const float2 wq = box_muller(u32_to_uniform01(q.x), u32_to_uniform01(q.y));
        float2 a, b, c, d;
        box_muller2(p, q, a, b);
        box_muller2(q, p, c, d);
        if (!same(box_muller_plain(p.x, p.y), wp) || !same(box_muller_plain(q.x, q.y), wq)) report(plain, k);
        if (!same(a, wp) || !same(c, wq)) report(first, k);
        if (!same(b, wq) || !same(d, wp)) report(second, k);
    }
}

}  // namespace

// Fills out[2 i], out[2 i + 1] with the differing inputs and the first of
// them for: the square root, the quotient, the radius (scalar, lane 0, lane 1
// of the packed form), the angle (the same three); out[16] with the unit
// radius word.  Returns the CUDA status.
extern "C" int MATH_CHECK(uint64_t* out) {
    constexpr int kResults = 8;
    Result host[kResults], *r = nullptr;
    uint32_t* unit = nullptr;
    for (Result& x : host) x = Result{0ull, ~0ull};
    cudaError_t e = cudaMalloc(&r, sizeof(host));
    if (e == cudaSuccess) e = cudaMalloc(&unit, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemcpy(r, host, sizeof(host), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(unit, 0, sizeof(uint32_t));
    uint32_t word = 0;
    if (e == cudaSuccess) {
        root_kernel<<<kBlocks, kThreads>>>(r);
#ifdef FPG_RECIPROCAL_DIVISION
        quotient_kernel<<<kBlocks, kThreads>>>(r + 1);     // only the step's units divide this way
#endif
        radius_kernel<<<kBlocks, kThreads>>>(r + 2, r + 3, r + 4);
        unit_radius_kernel<<<kBlocks, kThreads>>>(unit);
        angle_kernel<<<kBlocks, kThreads>>>(unit, 0x12345600u, r + 5, r + 6, r + 7);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(host, r, sizeof(host), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&word, unit, sizeof(word), cudaMemcpyDeviceToHost);
    cudaFree(r);
    cudaFree(unit);
    for (int k = 0; k < kResults; ++k) {
        out[2 * k] = host[k].differ;
        out[2 * k + 1] = host[k].first;
    }
    out[2 * kResults] = word;
    return (int)e;
}
