// move_fields.cu — the data movement of the compaction and of the reorder:
// every field array gathered through an index array into a second block.
#include "move_fields.h"

namespace fpg {
namespace {

struct MoveFields {
    const uint32_t* src[FPG_FIELD_COUNT];
    uint32_t* dst[FPG_FIELD_COUNT];
};

constexpr int kMoveThreads = 256;
constexpr int kMoveBatch = 8;

// One slot per thread; the loads of eight fields are issued before the first
// of their stores.  The field arrays come through pointers the compiler must
// assume to overlap, so a plain load-store sequence over the 23 fields keeps
// one load in flight per thread (22 registers: 351 us for the compaction of
// 5 M slots, 312 us for the reorder of 6 M); with the loads of a batch held
// in registers the same moves take 162 us (5.7 TB/s of the 184 B a slot and
// the index need) and 229 us.  A compaction's index is increasing, so a
// warp's 32 loads touch 4 to 8 sectors and HBM binds.  A reorder gathers from
// all over the column a warp's cell lies in, about one 128-byte line per two
// lanes: the L1 lookups of those lines bind it, not HBM (a field-outer form
// that keeps a CTA in one column window, 8 slots a thread, 256 to 1024
// threads: 240-295 us; batches of 4 to 23 fields, one or two slots a thread:
// 229-240 us; 32 registers, eight CTAs per SM, kept).
__global__ void __launch_bounds__(kMoveThreads, 8) move_fields_kernel(MoveFields m, const uint32_t* index,
                                                                      uint32_t n_host,
                                                                      const uint32_t* n_dev,
                                                                      uint32_t capacity, int clear_tail) {
    chain_begin();
    const uint32_t i = blockIdx.x * kMoveThreads + threadIdx.x;
    if (i >= capacity) return;
    const uint32_t n = n_dev ? *n_dev : n_host;
    const uint32_t from = i < n ? index[i] : i;
#pragma unroll
    for (int f0 = 0; f0 < FPG_FIELD_COUNT; f0 += kMoveBatch) {
        uint32_t v[kMoveBatch];
#pragma unroll
        for (int j = 0; j < kMoveBatch; ++j)
            if (f0 + j < FPG_FIELD_COUNT) v[j] = m.src[f0 + j][from];
        if (FPG_FIELD_FLAGS >= f0 && FPG_FIELD_FLAGS < f0 + kMoveBatch && clear_tail && i >= n)
            v[FPG_FIELD_FLAGS % kMoveBatch] &= ~FPG_FLAG_ACTIVE;
#pragma unroll
        for (int j = 0; j < kMoveBatch; ++j)
            if (f0 + j < FPG_FIELD_COUNT) m.dst[f0 + j][i] = v[j];
    }
}

}  // namespace

fpg_status move_fields(fpg_ctx* ctx, void* const* src, void* const* dst, const uint32_t* index, uint32_t n,
                       const uint32_t* n_dev, uint32_t capacity, bool clear_tail, cudaStream_t s) {
    MoveFields m;
    for (int f = 0; f < FPG_FIELD_COUNT; ++f) {
        m.src[f] = static_cast<const uint32_t*>(src[f]);
        m.dst[f] = static_cast<uint32_t*>(dst[f]);
    }
    const uint32_t blocks = (uint32_t)(((uint64_t)capacity + kMoveThreads - 1u) / kMoveThreads);
    launch_chained(move_fields_kernel, blocks, kMoveThreads, 0, s, m, index, n, n_dev, capacity, clear_tail ? 1 : 0);
    ctx->count();
    FPG_CHECK_LAUNCH();
    return FPG_OK;
}

}  // namespace fpg
