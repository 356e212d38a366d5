// edge_batches.h -- the batches of a range of edges [x, e) of fewer than 2^31
// edges, where e may be close to 2^32: places past e may wrap around, so they are
// told by how many edges are left, which may be negative.  Plain code without
// CUDA types.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define GRUS_EDGE_HD __host__ __device__ __forceinline__
#else
#define GRUS_EDGE_HD inline
#endif

namespace grus {

GRUS_EDGE_HD int edges_left(uint32_t x, uint32_t e) { return (int)(e - x); }

// The end of the batch of `size` edges that begins at x, `left` before the end.
GRUS_EDGE_HD uint32_t batch_end(uint32_t x, int left, int size) {
  return x + (uint32_t)(left < size ? left : size);
}

}  // namespace grus
