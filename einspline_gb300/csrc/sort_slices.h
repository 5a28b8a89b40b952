// The slices into which the counting sort's blocks divide a batch; plain C++,
// so that the arithmetic can be checked on the host up to the largest batch.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define EG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define EG_HOST_DEVICE inline
#endif

namespace eg {

// Points lo .. hi - 1 of n, for block b of `blocks`.  64-bit: near INT_MAX
// points a slice's end, and a thread's step beyond it, leave 32 bits.
struct SortSlice {
  int64_t lo, hi;
};
EG_HOST_DEVICE SortSlice sort_slice(int64_t n, int b, int blocks) {
  const int64_t chunk = (n + blocks - 1) / blocks, lo = b * chunk < n ? b * chunk : n;
  return {lo, lo + chunk < n ? lo + chunk : n};
}

}  // namespace eg
