// Rows of a container by warps: 32 consecutive rows are one run of edges.
#pragma once

#include "vg_internal.h"

namespace vg {
namespace {

__device__ __forceinline__ void copy_elem(int size, const void *in, uint64_t i, void *out,
                                          uint64_t o) {
  switch (size) {
    case 1: ((uint8_t *)out)[o] = ((const uint8_t *)in)[i]; break;
    case 2: ((uint16_t *)out)[o] = ((const uint16_t *)in)[i]; break;
    case 4: ((uint32_t *)out)[o] = ((const uint32_t *)in)[i]; break;
    case 8: ((uint64_t *)out)[o] = ((const uint64_t *)in)[i]; break;
  }
}

// The in-edges of a warp's 32 rows as one run, 32 consecutive edges at a
// time: f(e, owner, has) with the edge's number and the lane whose row it is.
// A lane per row would read and write its own short run, and the longest
// row of the 32 would set the pace.
template <class F>
__device__ __forceinline__ void warp_edges(uint32_t b, uint32_t deg, F f) {
  const unsigned lane = threadIdx.x & 31;
  // (rows are consecutive: lane l's run starts where lane l - 1's ends; rows
  // beyond the container are empty and start at the end)
  const uint32_t begin = __shfl_sync(0xffffffffu, b, 0);
  const uint32_t end = __shfl_sync(0xffffffffu, b + deg, 31);
  for (uint32_t e0 = begin; e0 < end; e0 += 32) {
    const uint32_t e = e0 + lane;
    unsigned owner = 0;  // the last lane whose run starts at or before e
#pragma unroll
    for (unsigned o = 16; o; o >>= 1) {
      const uint32_t bo = __shfl_sync(0xffffffffu, b, owner + o);
      if (bo <= e) owner += o;
    }
    f(e, owner, e < end);
  }
}

// start and length of row i, for warp_edges
__device__ __forceinline__ uint32_t row_run(const DevCSRView &c, uint64_t i, uint32_t &deg) {
  if (i >= c.nrows) {
    deg = 0;
    return (uint32_t)c.nedges;
  }
  const uint32_t b = c.row_ptr[i];
  deg = c.row_ptr[i + 1] - b;
  return b;
}

}  // namespace
}  // namespace vg
