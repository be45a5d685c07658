// align.cu -- the load-time layouts of the aligner's records, and the batched
// round's launches.
#include <mutex>
#include <vector>

#include "align.cuh"
#include "align_lds.cuh"
#include "kernels.cuh"

namespace ngia {

// Load-time layout kernels: one warp per record, lane k taking the record's
// 32-residue blocks k, k + 32, ... (four words each, coalesced across the
// warp); bit work by shifts and masks, no per-residue loops.

// mask of the residues of a block whose code is c, from its four planes
__device__ __forceinline__ uint32_t code_mask(const uint32_t (&pl)[4], uint32_t c) {
  return ((c & 1u) ? pl[0] : ~pl[0]) & ((c & 2u) ? pl[1] : ~pl[1]) &
         ((c & 4u) ? pl[2] : ~pl[2]) & ((c & 8u) ? pl[3] : ~pl[3]);
}

// Planes -> nibbles: the same record layout, with each block's four plane
// words replaced by four words of eight 4-bit codes.  The length word is
// copied.  presence |= bit c for every code c of a real residue.  A record
// whose offset lies outside the `words` of the region, whose length word is
// not lens[i], or whose blocks run past the region is left alone and sets
// kBadRecord in presence.
__global__ void __launch_bounds__(256)
nibble_kernel(const uint32_t *__restrict__ packed, const uint64_t *__restrict__ offs,
              const uint32_t *__restrict__ lens, uint32_t n, uint64_t words,
              uint32_t *__restrict__ nib, uint32_t *__restrict__ presence) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  uint32_t mine = 0;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const uint64_t o = offs[i];
    if (o >= words) {
      mine |= kBadRecord;
      continue;
    }
    const uint32_t len = __ldg(packed + o);
    if (len != lens[i] || o + 1 + 4ull * ((len + 31) >> 5) > words) {
      // flagged; an empty record in its place, so that a kernel reading the
      // layout before the flag is seen stays inside the region
      if (lane == 0) nib[o] = 0;
      mine |= kBadRecord;
      continue;
    }
    if (lane == 0) nib[o] = len;
    const uint32_t blocks = (len + 31) >> 5;
    for (uint32_t k = lane; k < blocks; k += 32) {
      const uint32_t *src = packed + o + 1 + 4 * k;
      const uint32_t pl[4] = {__ldg(src), __ldg(src + 1), __ldg(src + 2), __ldg(src + 3)};
      uint32_t w[4];
      planes_to_nibbles(pl, 4, w);
      uint32_t *dst = nib + o + 1 + 4 * k;
#pragma unroll
      for (int q = 0; q < 4; ++q) dst[q] = w[q];
      const uint32_t left = len - 32 * k;
      const uint32_t real = left >= 32 ? kFull : (1u << left) - 1u;
#pragma unroll
      for (uint32_t c = 0; c < 16; ++c)
        if (code_mask(pl, c) & real) mine |= 1u << c;
    }
  }
  mine = __reduce_or_sync(kFull, mine);
  if (lane == 0 && mine) atomicOr(presence, mine);
}

// Recoded databases from their packed planes, in one pass: the aligner-code
// nibbles (each residue code c replaced by map nibble c) and the planes of the aligner codes
// (planes 0-2, plane 3 zero).  bits[b] = the residue codes whose aligner code
// has bit b set.
__global__ void __launch_bounds__(256)
dense_layouts_kernel(const uint32_t *__restrict__ packed, const uint64_t *__restrict__ offs,
                     uint32_t n, uint32_t bit0, uint32_t bit1, uint32_t bit2,
                     uint32_t *__restrict__ dense_nib, uint32_t *__restrict__ dplanes) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const uint64_t o = offs[i];
    const uint32_t len = __ldg(packed + o);
    if (lane == 0) {
      dense_nib[o] = len;
      dplanes[o] = len;
    }
    const uint32_t blocks = (len + 31) >> 5;
    for (uint32_t k = lane; k < blocks; k += 32) {
      const uint32_t *src = packed + o + 1 + 4 * k;
      const uint32_t pl[4] = {__ldg(src), __ldg(src + 1), __ldg(src + 2), __ldg(src + 3)};
      uint32_t d[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (uint32_t c = 1; c < 16; ++c) {
        const uint32_t m = code_mask(pl, c);
        d[0] |= (bit0 >> c) & 1u ? m : 0u;
        d[1] |= (bit1 >> c) & 1u ? m : 0u;
        d[2] |= (bit2 >> c) & 1u ? m : 0u;
      }
      uint32_t w[4];
      planes_to_nibbles(d, 3, w);
      uint32_t *dn = dense_nib + o + 1 + 4 * k, *dp = dplanes + o + 1 + 4 * k;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        dn[q] = w[q];
        dp[q] = d[q];
      }
    }
  }
}

int launch_nibbles(const uint32_t *packed, const uint64_t *offs, const uint32_t *lens,
                   uint32_t n, uint64_t words, uint32_t *nib, uint32_t *presence, cudaStream_t s,
                   bool accumulate) {
  if (n == 0) return NGIA_OK;
  int dev = 0, sms = 0;
  NGIA_CUDA(cudaGetDevice(&dev));
  NGIA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint32_t want = ceil_div(n, 8u), cap = (uint32_t)sms * 16u;
  if (!accumulate) NGIA_CUDA(cudaMemsetAsync(presence, 0, sizeof(uint32_t), s));
  nibble_kernel<<<want < cap ? want : cap, 256, 0, s>>>(packed, offs, lens, n, words, nib,
                                                        presence);
  NGIA_LAUNCHED();
  return NGIA_OK;
}

// The layouts a recoded database needs, for a run of records in one pass over
// their planes, for loads whose code map is assumed ahead (the pipelined
// load): recoded nibbles and code planes (the sketch reads residue codes from
// the planes themselves).  Only the map's own codes are looked at: a residue
// of another code (or a record outside words [w0, w1), which is then left
// empty) sets *bad, and the load falls back.  Any subset of the map's codes
// is served by the same map (it stays one-to-one on the codes present).
// codes[k], k < ncodes: the residue codes of the map, aligner code k + 1.
// kDense / kPlanes: which of the two layouts a launch writes (a null output
// pointer leaves its layout out).
template <bool kDense, bool kPlanes>
__global__ void __launch_bounds__(256)
load_layouts_kernel(const uint32_t *__restrict__ packed, const uint64_t *__restrict__ offs,
                    const uint32_t *__restrict__ lens, uint32_t n, uint64_t w0, uint64_t w1,
                    uint64_t words, uint32_t codes, uint32_t ncodes,
                    uint32_t *__restrict__ dense_nib, uint32_t *__restrict__ dplanes,
                    uint32_t *__restrict__ bad) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  bool wrong = false;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const uint64_t o = offs[i];
    // a record outside its piece or with the wrong length word is flagged and,
    // when its offset lies in the region, left empty in every layout (the
    // sketch also bounds every record it reads by the region)
    if (o < w0 || o >= w1) {
      if (lane == 0 && o < words) {
        if (kDense) dense_nib[o] = 0;
        if (kPlanes) dplanes[o] = 0;
      }
      wrong = true;
      continue;
    }
    const uint32_t len = __ldg(packed + o);
    const uint32_t blocks = (len + 31) >> 5;
    if (len != lens[i] || o + 1 + 4ull * blocks > w1) {
      if (lane == 0) {
        if (kDense) dense_nib[o] = 0;
        if (kPlanes) dplanes[o] = 0;
      }
      wrong = true;
      continue;
    }
    if (lane == 0) {
      if (kDense) dense_nib[o] = len;
      if (kPlanes) dplanes[o] = len;
    }
    for (uint32_t k = lane; k < blocks; k += 32) {
      const uint64_t b = o + 1 + 4ull * k;
      const uint32_t pl[4] = {__ldg(packed + b), __ldg(packed + b + 1), __ldg(packed + b + 2),
                              __ldg(packed + b + 3)};
      const uint32_t left = len - 32 * k;
      const uint32_t real = left >= 32 ? kFull : (1u << left) - 1u;
      uint32_t d[4] = {0u, 0u, 0u, 0u}, known = 0u;
      for (uint32_t j = 0; j < ncodes; ++j) {
        const uint32_t m = code_mask(pl, (codes >> (4 * j)) & 15u);
        const uint32_t a = j + 1;  // aligner code
        known |= m;
        d[0] |= a & 1u ? m : 0u;
        d[1] |= a & 2u ? m : 0u;
        d[2] |= a & 4u ? m : 0u;
      }
      if (real & ~known) wrong = true;
      if (kDense) {
        uint32_t dn[4];
        planes_to_nibbles(d, 3, dn);
#pragma unroll
        for (int q = 0; q < 4; ++q) dense_nib[b + q] = dn[q];
      }
      if (kPlanes) {
#pragma unroll
        for (int q = 0; q < 4; ++q) dplanes[b + q] = d[q];
      }
    }
  }
  if (__ballot_sync(kFull, wrong) && lane == 0) atomicOr(bad, 1u);
}

static int map_bits(uint64_t map, uint32_t (&bits)[3]) {
  bits[0] = bits[1] = bits[2] = 0u;
  for (uint32_t c = 1; c < 16; ++c) {
    const uint32_t d = (uint32_t)(map >> (4 * c)) & 15u;
    if (d > 7) return NGIA_ERR_ARG;  // three planes hold aligner codes 0..7
    for (int b = 0; b < 3; ++b)
      if ((d >> b) & 1u) bits[b] |= 1u << c;
  }
  return NGIA_OK;
}

int launch_load_layouts(const uint32_t *packed, const uint64_t *offs, const uint32_t *lens,
                        uint32_t n, uint64_t w0, uint64_t w1, uint64_t words, uint64_t inv,
                        uint32_t *dense_nib, uint32_t *dplanes, uint32_t *bad,
                        cudaStream_t s) {
  if (w0 > w1 || w1 > words) return NGIA_ERR_ARG;
  if (n == 0) return NGIA_OK;
  uint32_t codes = 0, ncodes = 0;  // inv nibble d = residue code of aligner code d
  for (uint32_t d = 1; d < 8; ++d) {
    const uint32_t c = (uint32_t)(inv >> (4 * d)) & 15u;
    if (c == 0) break;
    codes |= c << (4 * ncodes++);
  }
  int dev = 0, sms = 0;
  NGIA_CUDA(cudaGetDevice(&dev));
  NGIA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint32_t want = ceil_div(n, 8u), cap = (uint32_t)sms * 16u;
  if (!dense_nib && !dplanes) return NGIA_OK;
  if (dense_nib && dplanes)
    load_layouts_kernel<true, true><<<want < cap ? want : cap, 256, 0, s>>>(
        packed, offs, lens, n, w0, w1, words, codes, ncodes, dense_nib, dplanes, bad);
  else if (dense_nib)
    load_layouts_kernel<true, false><<<want < cap ? want : cap, 256, 0, s>>>(
        packed, offs, lens, n, w0, w1, words, codes, ncodes, dense_nib, dplanes, bad);
  else
    load_layouts_kernel<false, true><<<want < cap ? want : cap, 256, 0, s>>>(
        packed, offs, lens, n, w0, w1, words, codes, ncodes, dense_nib, dplanes, bad);
  NGIA_LAUNCHED();
  return NGIA_OK;
}

int launch_dense_layouts(const uint32_t *packed, const uint64_t *offs, uint32_t n,
                         uint64_t map, uint32_t *dense_nib, uint32_t *dplanes,
                         cudaStream_t s) {
  if (n == 0) return NGIA_OK;
  uint32_t bits[3];
  NGIA_TRY(map_bits(map, bits));
  int dev = 0, sms = 0;
  NGIA_CUDA(cudaGetDevice(&dev));
  NGIA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint32_t want = ceil_div(n, 8u), cap = (uint32_t)sms * 16u;
  dense_layouts_kernel<<<want < cap ? want : cap, 256, 0, s>>>(packed, offs, n, bits[0], bits[1],
                                                               bits[2], dense_nib, dplanes);
  NGIA_LAUNCHED();
  return NGIA_OK;
}

struct OccEntry {
  const void *func;
  int dev, per_sm, sms;
};
static std::mutex g_occ_mu;
static std::vector<OccEntry> g_occ;

int persistent_grid(const void *func, int threads, size_t smem, uint32_t want, uint32_t *grid) {
  int dev = 0;
  NGIA_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(g_occ_mu);
  const OccEntry *hit = nullptr;
  for (const OccEntry &e : g_occ)
    if (e.func == func && e.dev == dev) hit = &e;
  if (!hit) {
    OccEntry e{func, dev, 0, 0};
    NGIA_CUDA(cudaDeviceGetAttribute(&e.sms, cudaDevAttrMultiProcessorCount, dev));
    NGIA_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // the most shared memory per SM the L1 split allows: more resident blocks
    NGIA_CUDA(cudaFuncSetAttribute(func, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   (int)cudaSharedmemCarveoutMaxShared));
    NGIA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&e.per_sm, func, threads, smem));
    if (e.per_sm < 1) e.per_sm = 1;
    g_occ.push_back(e);
    hit = &g_occ.back();
  }
  const uint32_t cap = (uint32_t)(hit->per_sm * hit->sms);
  *grid = want < cap ? want : cap;
  return NGIA_OK;
}

// The general class: one pair per thread, grid-stride over the class's range.
// A launch of its own, without tables: some 20 warps per multiprocessor where
// the kernel of the 32-lane classes leaves room for seven.  One-warp blocks
// spread few pairs over the multiprocessors, whose row words (up to 8 KB a
// thread in local memory) are what binds it.  Rounds of related proteins, ms in
// that kernel, here in blocks of 128, here: 60,000 pairs of 20,000 residues at
// identity 50 571, 670, 515; 2,000 116, 129, 113; 1,000
// of 60,000 at 40 1,175, 1,391, 1,175.
__global__ void __launch_bounds__(32)
align_general_kernel(const __grid_constant__ RoundArgs a) {
  const uint32_t begin = a.bounds[kGeneralClass], end = a.bounds[kGeneralClass + 1];
  uint32_t done = 0;
  for (uint32_t k = begin + blockIdx.x * 32u + threadIdx.x; k < end; k += gridDim.x * 32u) {
    const uint32_t p = a.order[k];
    const uint2 pr = a.pairs[p];
    const uint32_t *rep = a.packed + a.offs[pr.x];
    const uint32_t *tar = a.packed + a.offs[pr.y];
    const uint32_t lr = __ldg(rep), lt = __ldg(tar);
    const Band b = make_band(lr, lt, a.t, a.fm);
    uint32_t lines[kMaxRowBlocks];
    uint32_t blocks;
    const uint32_t lcs = lcs_general(rep, tar, b, lines, blocks);
    done += blocks * ((b.width + 7u) & ~7u);
    a.scores[p] = identity_score(lcs, lr, lt, a.t);
  }
  count_work(done, a.work);
}

int launch_align_general(const RoundArgs &a, uint32_t m, cudaStream_t s) {
  uint32_t grid = 0;
  NGIA_TRY(persistent_grid(reinterpret_cast<const void *>(align_general_kernel), 32, 0,
                           ceil_div(m, 32u), &grid));
  align_general_kernel<<<grid, 32, 0, s>>>(a);
  NGIA_LAUNCHED();
  return NGIA_OK;
}

template <int K>
int launch_align_k(int kernel, const RoundArgs &a, uint32_t m, cudaStream_t s);

int launch_align(int kernel, const RoundArgs &a, int K, uint32_t m, cudaStream_t s) {
  return K == 5   ? launch_align_k<5>(kernel, a, m, s)
         : K == 8 ? launch_align_k<8>(kernel, a, m, s)
                  : launch_align_k<16>(kernel, a, m, s);
}

}  // namespace ngia
