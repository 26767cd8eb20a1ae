// Hash tables and sorting of the kernels that build tiles (set-up work).
#pragma once

#include "fv_tile.cuh"

namespace mb {

__device__ __forceinline__ unsigned tile_hash(int key, int mask) { return ((unsigned)key * 2654435761u >> 15) & mask; }

// key's slot, inserting it if absent (was_new); -1 when the table is full
__device__ inline int hash_put(int *keys, int cap, int key, bool &was_new) {
  unsigned h = tile_hash(key, cap - 1);
  was_new = false;
  for (int probe = 0; probe < cap; ++probe, h = (h + 1) & (cap - 1)) {
    const int old = atomicCAS(keys + h, -1, key);
    if (old == -1) { was_new = true; return (int)h; }
    if (old == key) return (int)h;
  }
  return -1;
}
__device__ inline int hash_get(const int *keys, const uint16_t *vals, int cap, int key) {
  unsigned h = tile_hash(key, cap - 1);
  for (int probe = 0; probe < cap; ++probe, h = (h + 1) & (cap - 1)) {
    if (keys[h] == key) return vals[h];
    if (keys[h] == -1) break;
  }
  return 0;
}

// ascending sort of a[0, n) by the block (bitonic, padded to a power of two with INT_MAX; the
// array has room for it)
__device__ inline void block_sort(int *a, int n) {
  int p = 1;
  while (p < n) p <<= 1;
  for (int i = n + threadIdx.x; i < p; i += blockDim.x) a[i] = 0x7fffffff;
  __syncthreads();
  for (int k = 2; k <= p; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < p; i += blockDim.x) {
        const int q = i ^ j;
        if (q > i) {
          const int x = a[i], y = a[q];
          if ((x > y) == ((i & k) == 0)) { a[i] = y; a[q] = x; }
        }
      }
      __syncthreads();
    }
}

// last launch of a fill (fv_tile_plan.cu)
void tile_filled(cudaStream_t st);

}  // namespace mb
