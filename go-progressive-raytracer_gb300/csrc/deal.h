// deal.h - how a batch of n rays is dealt out to the warps or blocks of a
// launch.  Plain arithmetic on counts up to 2^32 - 1 (a batch of device rays
// may be that long), shared by the kernels and the host.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define GPRT_HD __host__ __device__ __forceinline__
#else
#define GPRT_HD inline
#endif

namespace gprt {

// Rays per chunk: `most`, or a warp's share of a batch that is smaller.
GPRT_HD uint32_t deal_chunk(uint32_t n, uint32_t warps, uint32_t most) {
  const uint32_t share = n / warps + (n % warps != 0);
  return share < most ? share : most;
}

// The first ray of a chunk that starts at `at`, or n past the end of the batch.
GPRT_HD uint32_t deal_at(uint32_t n, uint64_t at) { return at < n ? (uint32_t)at : n; }

// body(first ray) for a block's ranges of the batch: `first`, first + stride, ...
template <class Body>
GPRT_HD void deal_blocks(uint32_t n, uint32_t first, uint32_t stride, Body body) {
  for (uint64_t base = first; base < n; base += stride) body(base);
}

}  // namespace gprt
