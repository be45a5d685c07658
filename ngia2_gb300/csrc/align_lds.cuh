// align_lds.cuh -- match-mask tables in shared memory (internal header).
//
// When a row block of the representative enters the band its match masks (one
// per nonzero residue code: bit r set when row r has that code) are written
// once into the lane's table; every column step then reads the mask of each
// live row word with one shared-memory load, so the integer ALU only does the
// three operations of the LCS update per word
//     t = V & M;   s = V + t + carry;   V = s | (V ^ t)
// Targets are read as 4-bit codes packed eight per word (nibble layout, first
// residue in the high nibble).
//
// Shared memory per warp: [K codes][W slots][32 lanes] words, so the 32 lanes
// of a load hit 32 different banks.
#pragma once

#include "align.cuh"

namespace ngia {

// K = entries per row block: 16 (all residue codes), or 8 / 5 when the
// database uses at most 7 / 4 nonzero codes and the records were recoded
// densely (the table, and so the shared memory per thread, shrinks to a half /
// under a third; nucleotides take 5).
template <int W, int K = 16>
struct LdsTable {
  uint32_t *base;  // this thread's column of the warp's table
  __device__ __forceinline__ uint32_t *slot(uint32_t s) const { return base + s * 32; }
  static constexpr uint32_t kCodeStride = W * 32;  // words between codes
  __device__ __forceinline__ void clear(uint32_t s) const {
    uint32_t *p = slot(s);
#pragma unroll
    for (int c = 1; c < K; ++c) p[c * kCodeStride] = 0u;
  }
  __device__ __forceinline__ void move(uint32_t to, uint32_t from) const {
    uint32_t *d = slot(to);
    const uint32_t *p = slot(from);
#pragma unroll
    for (int c = 1; c < K; ++c) d[c * kCodeStride] = p[c * kCodeStride];
  }
  // masks of one row block from its four bit planes
  __device__ __forceinline__ void fill(uint32_t s, const uint4 &pl) const {
    uint32_t *p = slot(s);
    if constexpr (K == 16) {
      const uint32_t lo[4] = {~pl.x & ~pl.y, pl.x & ~pl.y, ~pl.x & pl.y, pl.x & pl.y};
      const uint32_t hi[4] = {~pl.z & ~pl.w, pl.z & ~pl.w, ~pl.z & pl.w, pl.z & pl.w};
#pragma unroll
      for (int c = 1; c < 16; ++c) p[c * kCodeStride] = lo[c & 3] & hi[c >> 2];
    } else {  // K = 5 or 8: the code planes (aligner code bits in planes 0-2)
#pragma unroll
      for (int d = 1; d < K; ++d)
        p[d * kCodeStride] = ((d & 1) ? pl.x : ~pl.x) & ((d & 2) ? pl.y : ~pl.y) &
                             ((d & 4) ? pl.z : ~pl.z);
    }
  }
};

__device__ __forceinline__ uint4 load4(const uint32_t *p) {
  return make_uint4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// bits 0..7 of b to bits 0, 4, ..., 28
__device__ __forceinline__ uint32_t spread8(uint32_t b) {
  b = (b | (b << 12)) & 0x000F000Fu;
  b = (b | (b << 6)) & 0x03030303u;
  return (b | (b << 3)) & 0x11111111u;
}

// Four plane words of a block (bit r of plane e = bit e of the code of
// residue r) -> its four nibble words (word q: residues 8q..8q+7, the first in
// the high nibble).
__device__ __forceinline__ void planes_to_nibbles(const uint32_t (&pl)[4], int np,
                                                  uint32_t (&out)[4]) {
  uint32_t rv[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) rv[e] = e < np ? __brev(pl[e]) : 0u;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t w = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < np) w |= spread8((rv[e] >> (24 - 8 * q)) & 0xFFu) << e;
    out[q] = w;
  }
}

__device__ __forceinline__ uint4 planes_to_nibbles(const uint4 &pl) {
  const uint32_t in[4] = {pl.x, pl.y, pl.z, pl.w};
  uint32_t out[4];
  planes_to_nibbles(in, 4, out);
  return make_uint4(out[0], out[1], out[2], out[3]);
}

// Adds the warp's computed 32x32 blocks (row words x column blocks) to *work.
__device__ __forceinline__ void count_work(uint32_t blocks, unsigned long long *work) {
  // two 16-bit halves, so that a warp's sum cannot overflow
  const uint32_t lo = __reduce_add_sync(kFull, blocks & 0xFFFFu);
  const uint32_t hi = __reduce_add_sync(kFull, blocks >> 16);
  const unsigned long long sum = ((unsigned long long)hi << 16) + lo;
  if ((threadIdx.x & 31u) == 0 && sum) atomicAdd(work, sum);
}

}  // namespace ngia
