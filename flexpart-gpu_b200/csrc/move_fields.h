// move_fields.h — moving every field of a particle block by an index array
// (compaction and reorder).
#pragma once

#include "fpg_internal.h"

namespace fpg {

// dst[f][i] = src[f][index[i]] for i < n and src[f][i] for n <= i < capacity,
// for every field f; with `clear_tail` the slots from n on lose their active
// bit.  n is *n_dev when n_dev is given.  src and dst are the field arrays
// of two blocks that do not overlap; index may be the last field of dst
// (each thread reads its entry before it writes that slot).
fpg_status move_fields(fpg_ctx* ctx, void* const* src, void* const* dst, const uint32_t* index, uint32_t n,
                       const uint32_t* n_dev, uint32_t capacity, bool clear_tail, cudaStream_t s);

}  // namespace fpg
