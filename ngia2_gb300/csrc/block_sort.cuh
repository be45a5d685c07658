// block_sort.cuh -- a block sorts distinct 64-bit keys in shared memory
// (internal header).
#pragma once

#include <cstdint>

namespace ngia {

// keys[0, n) into increasing order by a bitonic network over the next power of
// two (at most the array's size), whose missing keys are all ones.  Every
// thread of the block calls it; the keys are in place and in order after it.
__device__ __forceinline__ void block_sort(uint64_t *keys, uint32_t n) {
  uint32_t size = 1;
  while (size < n) size <<= 1;
  for (uint32_t k = n + threadIdx.x; k < size; k += blockDim.x) keys[k] = ~0ull;
  __syncthreads();
  for (uint32_t run = 2; run <= size; run <<= 1)
    for (uint32_t d = run >> 1; d > 0; d >>= 1) {
      for (uint32_t e = threadIdx.x; e < size / 2; e += blockDim.x) {
        const uint32_t i = 2 * e - (e & (d - 1)), j = i + d;  // i: bit d clear
        const uint64_t a = keys[i], b = keys[j];
        if ((a > b) == ((i & run) == 0)) {
          keys[i] = b;
          keys[j] = a;
        }
      }
      __syncthreads();
    }
}

}  // namespace ngia
