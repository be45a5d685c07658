// sketch.cu -- stage (a): 64 minhash signatures per packed record.
//
// Restates the signing loop of MakeDB::packData (src/makedb.hpp:224-248):
//   k-mer  = the last 8 residue codes as one 32-bit word, newest code in the
//            low nibble (codes before position 0 are 0);
//   signed positions: 7..L-1, or only L-1 when L < 8; none when L = 0;
//   band k = min over signed positions of H(kmer ^ (k*0x9e3779b1 + 0x85ebca6b))
//   with H Wang's 32-bit integer hash followed by two extra xor-shift-multiply
//   rounds (the steps below), minimum 0xFFFFFFFF when nothing is signed.
//
// Mapping: one warp per record, two bands per lane (sketch_kernel); few records
// or few bands take runs of bands, each lane a run of the positions
// (sketch_bands_kernel).  Records are in length-descending index order, so the
// longest are scheduled first.
//
// The work is integer-bound: 64 hashes of 13 integer instructions per
// position against half a byte read.  On this GPU the logic/shift pipe and
// the integer multiply-add pipe draw on the same integer issue budget, and a
// multiply-high costs two of its slots, so the shifts stay shifts.
#include <algorithm>

#include "align_lds.cuh"
#include "kernels.cuh"

namespace ngia {

// First xor-shift of the hash with the band seed folded in:
//   x = kmer ^ seed;  x = (x ^ 61) ^ (x >> 16)
//     = (kmer ^ (kmer >> 16)) ^ (seed ^ 61 ^ (seed >> 16))
__host__ __device__ constexpr uint32_t band_seed_fold(uint32_t band) {
  return (band * 0x9e3779b1u + 0x85ebca6bu) ^ 61u ^
         ((band * 0x9e3779b1u + 0x85ebca6bu) >> 16);
}

__device__ __forceinline__ uint32_t band_hash_tail(uint32_t x) {
  x = x * 9u;  // x + (x << 3)
  x ^= x >> 4;
  x *= 0x27d4eb2du;
  x ^= x >> 15;
  x = (x ^ (x >> 8)) * 0x9e3779b1u;
  x ^= x >> 14;
  return x;
}

// k-mers from the bit planes of a packed record (ABI entry point).
struct PlaneKmers {
  const uint32_t *rec;
  __device__ static PlaneKmers make(const uint32_t *r) {
    PlaneKmers k;
    k.rec = r;
    return k;
  }
  // code word w of a record: residues 8w..8w+7, the first in the high nibble
  __device__ static __forceinline__ uint32_t word(const uint32_t *r, uint32_t w) {
    const uint32_t *b = r + 1 + 4 * (w >> 2);
    uint32_t out = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e)
      out |= spread8((__brev(__ldg(b + e)) >> (24 - 8 * (w & 3u))) & 0xFFu) << e;
    return out;
  }
  uint32_t block = 0xFFFFFFFFu;
  uint32_t p0 = 0, p1 = 0, p2 = 0, p3 = 0;
  uint32_t kmer = 0;
  __device__ __forceinline__ uint32_t code(uint32_t pos) {
    const uint32_t blk = pos >> 5;
    if (blk != block) {
      const uint32_t *b = rec + 1 + 4 * blk;
      p0 = __ldg(b);
      p1 = __ldg(b + 1);
      p2 = __ldg(b + 2);
      p3 = __ldg(b + 3);
      block = blk;
    }
    const uint32_t s = pos & 31u;
    return ((p0 >> s) & 1u) | (((p1 >> s) & 1u) << 1) | (((p2 >> s) & 1u) << 2) |
           (((p3 >> s) & 1u) << 3);
  }
  __device__ __forceinline__ void start(uint32_t pb) {
    kmer = 0;
    for (uint32_t q = pb >= 7 ? pb - 7 : 0; q < pb; ++q) kmer = (kmer << 4) | code(q);
  }
  __device__ __forceinline__ uint32_t at(uint32_t p) {  // positions in increasing order
    kmer = (kmer << 4) | code(p);
    return kmer;
  }
};

// k-mers from the nibble layout (word k holds positions 8k..8k+7, first in the
// high nibble): the k-mer ending at p is the 32-bit window of the stream
// starting at position p - 7, one funnel shift.
struct NibbleKmers {
  const uint32_t *nib;  // the record's first code word
  __device__ static NibbleKmers make(const uint32_t *r) { return NibbleKmers{r + 1}; }
  __device__ static __forceinline__ uint32_t word(const uint32_t *r, uint32_t w) {
    return __ldg(r + 1 + w);
  }
  __device__ __forceinline__ void start(uint32_t) {}
  __device__ __forceinline__ uint32_t at(uint32_t p) {
    if (p < 7) return __ldg(nib) >> (28 - 4 * p);  // short record: codes 0..p
    const uint32_t s = p - 7, k = s >> 3, r = s & 7u;
    const uint32_t hi = __ldg(nib + k);
    return r ? __funnelshift_l(__ldg(nib + k + 1), hi, 4 * r) : hi;
  }
};

// More than 32 bands of a record by one warp, bands `lane` and `lane + 32` in each
// lane, every lane over all positions.  A tile of 256 positions at a time: the
// lanes load (or make) its code words, turn them into the positions' folded
// k-mers in shared memory, and then all read the same four k-mers per 16-byte
// load and hash them for their own bands.
//
// What bounds it: the logic pipe, ten operations a hash.  The positions are
// hashed as many times as there are, up to three more at a record's end, and
// nothing is combined across lanes; with a run of the positions per lane and
// all 64 minima in its registers a record of 333 positions took 352 (eleven in
// each lane), 64 reductions, and left room for 16 warps per multiprocessor:
// 20,000 proteins of 340 residues on average 244 us, so 234 (1.82e12 hashes/s;
// 1.97e12 without loads and tails).  A block per four records, not a grid that
// loops: the blocks follow one another as they end, longest first.  1, 2, 4, 8
// warps a block: 4,800 records 82, 82, 82, 103 us (eight of the longest on one
// multiprocessor), 20,000 242, 238, 234, 236.
constexpr uint32_t kSketchWarps = 4;  // per block
constexpr uint32_t kSketchTile = 256;

template <typename Source>
__global__ void __launch_bounds__(kSketchWarps * 32)
sketch_kernel(const uint32_t *__restrict__ words, const uint64_t *__restrict__ offs,
              uint32_t n, uint32_t *__restrict__ sigs, size_t stride, uint32_t bands) {
  __shared__ __align__(16) uint32_t kmers[kSketchWarps][kSketchTile];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t *km = kmers[threadIdx.x >> 5];
  const uint4 *km4 = reinterpret_cast<const uint4 *>(km);
  const uint32_t fold0 = band_seed_fold(lane), fold1 = band_seed_fold(lane + 32);
  const uint32_t i = blockIdx.x * kSketchWarps + (threadIdx.x >> 5);
  if (i < n) {
    const uint32_t *rec = words + offs[i];
    const uint32_t len = __ldg(rec);
    const uint32_t nw = (len + 7u) >> 3;  // code words
    const uint32_t span = len >= 8 ? len - 7 : (len ? 1u : 0u);  // signed positions
    uint32_t lo = kFull, hi = kFull;
    for (uint32_t s0 = 0; s0 < span; s0 += kSketchTile) {
      const uint32_t cnt = min(span - s0, kSketchTile);
      const uint32_t w0 = s0 >> 3;
      const uint32_t mine = w0 + lane < nw ? Source::word(rec, w0 + lane) : 0u;
      uint32_t after = w0 + 32 < nw ? Source::word(rec, w0 + 32) : 0u;
      const uint32_t next = __shfl_down_sync(kFull, mine, 1);
      if (lane < 31) after = next;
      // the lane's eight windows: the k-mer of window r starts at its residue r
      // (a record of fewer than eight residues has one, of all of them)
      __syncwarp();
#pragma unroll
      for (uint32_t r = 0; r < 8; ++r) {
        uint32_t k = __funnelshift_l(after, mine, 4 * r);
        if (len < 8) k = mine >> (4 * (8 - len));
        k ^= k >> 16;
        const uint32_t q = 8 * lane + r;
        if (q < cnt) km[q] = k;
        // the last group of four filled up with the last k-mer
        if (q == cnt - 1)
          for (uint32_t f = cnt; f & 3u; ++f) km[f] = k;
      }
      __syncwarp();
      const uint32_t groups = (cnt + 3) >> 2;
#pragma unroll 2
      for (uint32_t g = 0; g < groups; ++g) {
        const uint4 y = km4[g];
        lo = min(lo, band_hash_tail(y.x ^ fold0));
        hi = min(hi, band_hash_tail(y.x ^ fold1));
        lo = min(lo, band_hash_tail(y.y ^ fold0));
        hi = min(hi, band_hash_tail(y.y ^ fold1));
        lo = min(lo, band_hash_tail(y.z ^ fold0));
        hi = min(hi, band_hash_tail(y.z ^ fold1));
        lo = min(lo, band_hash_tail(y.w ^ fold0));
        hi = min(hi, band_hash_tail(y.w ^ fold1));
      }
    }
    if (lane < bands) sigs[lane * stride + i] = lo;
    if (lane + 32 < bands) sigs[(lane + 32) * stride + i] = hi;
  }
}

// Bands [NB * blockIdx.y, ...) below `bands` only, signatures at sigs[band *
// stride + i]: one warp per record and run of NB bands, the band seeds in
// registers.
template <typename Source, int NB>
__global__ void __launch_bounds__(256)
sketch_bands_kernel(const uint32_t *__restrict__ words, const uint64_t *__restrict__ offs,
                    uint32_t n, uint32_t *__restrict__ sigs, size_t stride, uint32_t bands) {
  static_assert(NB <= 32, "one lane per band writes");
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t band0 = blockIdx.y * NB;
  uint32_t fold[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k) fold[k] = band_seed_fold(band0 + (uint32_t)k);
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const uint32_t *rec = words + offs[i];
    const uint32_t len = __ldg(rec);
    const uint32_t first = len >= 8 ? 7u : (len > 0 ? len - 1 : 0u);
    const uint32_t per = (len - first + 31u) >> 5;
    const uint32_t pb = first + lane * per;
    const uint32_t pe = min(pb + per, len);
    uint32_t mn[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) mn[k] = kFull;
    if (pb < pe) {
      Source src = Source::make(rec);
      src.start(pb);
      for (uint32_t p = pb; p < pe; ++p) {
        const uint32_t kmer = src.at(p);
        const uint32_t y = kmer ^ (kmer >> 16);
#pragma unroll
        for (int k = 0; k < NB; ++k) mn[k] = min(mn[k], band_hash_tail(y ^ fold[k]));
      }
    }
    uint32_t mine = kFull;
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      const uint32_t r = __reduce_min_sync(kFull, mn[k]);
      if ((uint32_t)k == lane) mine = r;
    }
    if (lane < (uint32_t)NB && band0 + lane < bands) sigs[(band0 + lane) * stride + i] = mine;
  }
}

template <typename Source, int NB>
static int launch_bands(const uint32_t *words, const uint64_t *offs, uint32_t n, uint32_t *sigs,
                        size_t stride, uint32_t bands, uint32_t cap, cudaStream_t s) {
  const uint32_t want = ceil_div(n, 8u);  // 8 warps per block
  sketch_bands_kernel<Source, NB><<<dim3(want < cap ? want : cap, ceil_div(bands, (uint32_t)NB)),
                                    256, 0, s>>>(words, offs, n, sigs, stride, bands);
  NGIA_LAUNCHED();
  return NGIA_OK;
}

template <typename Source>
static int launch(const uint32_t *words, const uint64_t *offs, uint32_t n, uint32_t *sigs,
                  size_t stride, uint32_t bands, cudaStream_t s) {
  if (n == 0) return NGIA_OK;
  int dev = 0, sms = 0;
  NGIA_CUDA(cudaGetDevice(&dev));
  NGIA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint32_t cap = (uint32_t)sms * 16u;
  // Fewer bands than the file's 64 are hashed as such (400,009 proteins, 3
  // bands: 0.23 ms where 64 take 4.8).  All 64 of few records are split over
  // warps: a warp that hashes 64 bands of a record of 340 takes 8,300
  // instructions by itself, and fewer records than keep the device busy leave it
  // waiting for that.  Proteins, 16 and 8 bands a warp: 200 records 13.6, 12.6
  // us; 600: 20.8, 20.6; 2,400: 49, 54; 4,800: 87, 92 (every run of bands rolls
  // the k-mers again); all 64 a warp: 2,433 51 us, 4,800 82.  More than 32 bands
  // of many records are hashed as 64 (33 bands of 200,003 streamed proteins,
  // sketch pass: 2.83 ms in two runs of 32, 2.40 so).
  if (bands <= 4) return launch_bands<Source, 4>(words, offs, n, sigs, stride, bands, cap, s);
  if (bands <= 8 || n <= (uint32_t)sms * 2u)
    return launch_bands<Source, 8>(words, offs, n, sigs, stride, bands, cap, s);
  if (bands <= 32 || n <= (uint32_t)sms * 16u)
    return launch_bands<Source, 16>(words, offs, n, sigs, stride, bands, cap, s);
  sketch_kernel<Source><<<ceil_div(n, kSketchWarps), kSketchWarps * 32, 0, s>>>(
      words, offs, n, sigs, stride, bands);
  NGIA_LAUNCHED();
  return NGIA_OK;
}

int launch_sketch(const uint32_t *packed, const uint64_t *offs, uint32_t n, uint32_t *sigs,
                  cudaStream_t s) {
  return launch<PlaneKmers>(packed, offs, n, sigs, n, kBands, s);
}

int launch_sketch_nibbles(const uint32_t *nib, const uint64_t *offs, uint32_t n,
                          uint32_t *sigs, size_t stride, uint32_t bands, cudaStream_t s) {
  return launch<NibbleKmers>(nib, offs, n, sigs, stride, bands, s);
}

// ---- databases of at most four residue codes: tables of all 8-mers -------------
// With at most four codes (nucleotides) an 8-mer is one of 4^8 = 65,536
// values.  Entry idx of the tables (2 bits per position, the newest in the low
// bits; digit d is aligner code d + 1, i.e. the residue code in nibble d + 1
// of `inv`) stands for the k-mer kmer_of_index(idx), whose hashes are exactly
// those sketch_kernel computes, so the signatures are the same.  Two tables:
//
//  * the ranks: per band, the 65,536 entries in increasing order of that
//    band's hash.  A band's minimum over a record is the hash of the first
//    entry in this order that occurs in the record.  A warp marks the
//    record's 8-mers in a 65,536-bit set in shared memory, then each lane
//    walks the orders of two bands, 8 entries per 16-byte load, until each
//    has met an 8-mer of the record: ~45 bit tests per band for a record of
//    1,500 positions instead of 1,500 hashes per band (the warp waits for its
//    slowest lane, ~3x the mean).  The expected walk grows as
//    65,536 / positions, so
//  * short records (fewer than kRankMinSpan signed positions) take the hash
//    row table: bands [0, kTableBands) of every 8-mer, gathered with 16-byte
//    loads while the other bands are hashed as in sketch_kernel (gathering
//    all 64 is bound by L2 bandwidth, hashing all by the logic pipe).
#ifndef NGIA_SKETCH_TABLE_BANDS
#define NGIA_SKETCH_TABLE_BANDS 24  // multiple of 4
#endif
#ifndef NGIA_SKETCH_RANK_MIN_SPAN
#define NGIA_SKETCH_RANK_MIN_SPAN 512
#endif
constexpr int kTableBands = NGIA_SKETCH_TABLE_BANDS;
static_assert(kTableBands % 4 == 0 && kTableBands <= kBands, "table bands");
constexpr uint32_t kRankMinSpan = NGIA_SKETCH_RANK_MIN_SPAN;
constexpr uint32_t kBitsetWords = kSketchTableEntries / 32;
constexpr uint32_t kRankWarps = 4;  // warps per block, one 8 KB bit set each
constexpr size_t kRowTableBytes = (size_t)kSketchTableEntries * kTableBands * 4;
constexpr size_t kRankBytes = (size_t)kSketchTableEntries * kBands * 2;

__device__ __forceinline__ uint32_t kmer_of_index(uint32_t idx, uint64_t inv) {
  uint32_t kmer = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t d = (idx >> (2 * j)) & 3u;
    kmer |= ((uint32_t)(inv >> (4 * (d + 1))) & 15u) << (4 * j);
  }
  return kmer;
}

__device__ __forceinline__ uint32_t index_hash(uint32_t idx, uint64_t inv, uint32_t band) {
  const uint32_t kmer = kmer_of_index(idx, inv);
  return band_hash_tail((kmer ^ (kmer >> 16)) ^ band_seed_fold(band));
}

// rows[idx * kTableBands + band] for the first kTableBands bands
__global__ void __launch_bounds__(256)
sketch_rows_build_kernel(uint64_t inv, uint32_t *__restrict__ rows) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= kSketchTableEntries * (uint32_t)kTableBands) return;
  rows[t] = index_hash(t / kTableBands, inv, t % kTableBands);
}

// band-major (hash, entry) pairs of all 64 bands, to be sorted per band
__global__ void __launch_bounds__(256)
sketch_keys_build_kernel(uint64_t inv, uint32_t *__restrict__ keys,
                         uint32_t *__restrict__ vals) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= kSketchTableEntries * (uint32_t)kBands) return;
  const uint32_t idx = t % kSketchTableEntries;
  keys[t] = index_hash(idx, inv, t / kSketchTableEntries);
  vals[t] = idx;
}

__global__ void __launch_bounds__(256)
narrow_kernel(const uint32_t *__restrict__ in, uint16_t *__restrict__ out, uint32_t count) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < count) out[t] = (uint16_t)in[t];
}

// A word of eight 2-bit digits held one per nibble (first position in the
// high nibble) -> the table entry of that 8-mer (the newest digit lowest).
__device__ __forceinline__ uint32_t compress_digits(uint32_t t) {
  t = (t | (t >> 2)) & 0x0F0F0F0Fu;
  t = (t | (t >> 4)) & 0x00FF00FFu;
  return (t | (t >> 8)) & 0x0000FFFFu;
}

// Rolling 8-mer entry over positions [pb, pe) of a record in aligner codes
// (word k holds positions 8k..8k+7, first in the high nibble); f(p, idx).
template <typename F>
__device__ __forceinline__ void for_each_index(const uint32_t *w, uint32_t pb, uint32_t pe,
                                               F &&f) {
  uint32_t idx = 0;
  for (uint32_t q = pb - 7; q < pb; ++q)
    idx = (idx << 2) | (((__ldg(w + (q >> 3)) >> (28 - 4 * (q & 7u))) & 15u) - 1u);
  uint32_t word = __ldg(w + (pb >> 3));
  for (uint32_t p = pb; p < pe; ++p) {
    if ((p & 7u) == 0) word = __ldg(w + (p >> 3));
    idx = ((idx << 2) | (((word >> (28 - 4 * (p & 7u))) & 15u) - 1u)) & 0xFFFFu;
    f(p, idx);
  }
}

// Records with at least kRankMinSpan signed positions: the rank walk.
__global__ void __launch_bounds__(kRankWarps * 32)
sketch_rank_kernel(const uint32_t *__restrict__ dense, const uint64_t *__restrict__ offs,
                   uint32_t n, uint64_t words, uint64_t inv, const uint16_t *__restrict__ ranks,
                   uint32_t *__restrict__ sigs, uint32_t stride) {
  __shared__ __align__(16) uint32_t bitsets[kRankWarps * kBitsetWords];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t *bits = bitsets + (threadIdx.x >> 5) * kBitsetWords;
  uint4 *bits4 = reinterpret_cast<uint4 *>(bits);
#pragma unroll
  for (uint32_t k = 0; k < kBitsetWords / 128; ++k) bits4[k * 32 + lane] = make_uint4(0, 0, 0, 0);
  __syncwarp();
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const uint64_t o = offs[i];
    if (o >= words) continue;  // outside the layouts (flagged by their kernel)
    const uint32_t len = __ldg(dense + o);
    if (len < 7 + kRankMinSpan) continue;  // short: the row table kernel's
    if (o + 1 + 4ull * ((len + 31u) >> 5) > words) continue;
    // mark the 8-mers: lane l takes code words l, l + 32, ... (coalesced), the
    // entry rolling over the word's 8 positions from the previous word's last
    const uint32_t *w = dense + o + 1;
    const uint32_t words = (len + 7) >> 3;
    for (uint32_t k = lane; k < words; k += 32) {
      uint32_t cur = __ldg(w + k);
      const uint32_t valid = len - 8 * k;  // codes in this word (1..8 in the last)
      if (valid < 8) cur |= 0x11111111u >> (4 * valid);  // padding: any code, never read
      cur -= 0x11111111u;                  // digits 0..3, no borrows
      uint32_t idx = k ? compress_digits(__ldg(w + k - 1) - 0x11111111u) : 0u;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        idx = ((idx << 2) | ((cur >> (28 - 4 * r)) & 3u)) & 0xFFFFu;
        if (8 * k + r >= 7 && (uint32_t)r < valid)
          atomicOr(bits + (idx >> 5), 1u << (idx & 31u));
      }
    }
    __syncwarp();
    // walk: lane l finds the minima of bands l and l + 32 in turn, testing
    // 8 entries of the band's order per 16-byte load, two loads ahead
    uint32_t hit[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4 *row = reinterpret_cast<const uint4 *>(ranks) +
                         (size_t)(lane + 32 * h) * (kSketchTableEntries / 8);
      uint4 cur = __ldg(row), nxt = __ldg(row + 1);
      uint32_t found = kFull;
      // bounded: the record has an 8-mer, so every band's order meets it
      for (uint32_t step = 0; found == kFull && step < kSketchTableEntries / 8; ++step) {
        const uint4 v = cur;
        cur = nxt;
        nxt = __ldg(row + min(step + 2, kSketchTableEntries / 8 - 1));
        const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
        uint32_t hm = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const uint32_t e = (wv[q >> 1] >> (16 * (q & 1))) & 0xFFFFu;
          hm |= ((bits[e >> 5] >> (e & 31u)) & 1u) << q;
        }
        if (hm) {
          const int q = __ffs(hm) - 1;
          found = (wv[q >> 1] >> (16 * (q & 1))) & 0xFFFFu;
        }
      }
      hit[h] = found;
    }
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < kBitsetWords / 128; ++k)
      bits4[k * 32 + lane] = make_uint4(0, 0, 0, 0);
    const uint32_t lo = index_hash(hit[0], inv, lane);
    const uint32_t hi = index_hash(hit[1], inv, lane + 32);
    __syncwarp();
    sigs[(size_t)lane * stride + i] = lo;
    sigs[(size_t)(lane + 32) * stride + i] = hi;
  }
}

// Records with fewer than kRankMinSpan signed positions: row table + hashing.
// packed: the records' bit planes (residue codes for the hashed bands, and
// records shorter than 8, hashed directly); dense: the same records in
// aligner codes 1..4 (the table's index).
__global__ void __launch_bounds__(256)
sketch_table_kernel(const uint32_t *__restrict__ packed, const uint32_t *__restrict__ dense,
                    const uint64_t *__restrict__ offs, uint32_t n, uint64_t words,
                    const uint4 *__restrict__ table, uint32_t *__restrict__ sigs,
                    uint32_t stride) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const uint64_t o = offs[i];
    if (o >= words) continue;  // outside the layouts (flagged by their kernel)
    const uint32_t len = __ldg(packed + o);
    if (len >= 7 + kRankMinSpan) continue;  // the rank walk's
    if (o + 1 + 4ull * ((len + 31u) >> 5) > words) continue;
    uint32_t mn[kBands];
#pragma unroll
    for (int k = 0; k < kBands; ++k) mn[k] = kFull;
    if (len >= 8) {
      const uint32_t span = len - 7;  // signed positions 7 .. len-1
      const uint32_t per = (span + 31u) >> 5;
      const uint32_t pb = 7 + lane * per;
      const uint32_t pe = min(pb + per, len);
      if (pb < pe) {
        PlaneKmers src = PlaneKmers::make(packed + o);  // rolled along the lane's run
        src.start(pb);
        for_each_index(dense + o + 1, pb, pe, [&](uint32_t p, uint32_t idx) {
          const uint4 *row = table + (size_t)idx * (kTableBands / 4);
          uint4 v[kTableBands / 4];
#pragma unroll
          for (int k = 0; k < kTableBands / 4; ++k) v[k] = __ldg(row + k);
          // the other bands are hashed while the row is on its way
          const uint32_t kmer = src.at(p);
          const uint32_t y = kmer ^ (kmer >> 16);
#pragma unroll
          for (int k = kTableBands; k < kBands; ++k)
            mn[k] = min(mn[k], band_hash_tail(y ^ band_seed_fold((uint32_t)k)));
#pragma unroll
          for (int k = 0; k < kTableBands / 4; ++k) {
            mn[4 * k] = min(mn[4 * k], v[k].x);
            mn[4 * k + 1] = min(mn[4 * k + 1], v[k].y);
            mn[4 * k + 2] = min(mn[4 * k + 2], v[k].z);
            mn[4 * k + 3] = min(mn[4 * k + 3], v[k].w);
          }
        });
      }
    } else if (len > 0 && lane == 0) {  // the one signed position: the whole record
      PlaneKmers src = PlaneKmers::make(packed + o);
      src.start(len - 1);
      const uint32_t kmer = src.at(len - 1);
      const uint32_t y = kmer ^ (kmer >> 16);
#pragma unroll
      for (int k = 0; k < kBands; ++k) mn[k] = band_hash_tail(y ^ band_seed_fold((uint32_t)k));
    }
    uint32_t lo = kFull, hi = kFull;
#pragma unroll
    for (int k = 0; k < kBands; ++k) {
      const uint32_t r = __reduce_min_sync(kFull, mn[k]);
      if ((uint32_t)(k & 31) == lane) {
        if (k < 32) lo = r;
        else hi = r;
      }
    }
    sigs[(size_t)lane * stride + i] = lo;
    sigs[(size_t)(lane + 32) * stride + i] = hi;
  }
}

size_t sketch_table_bytes() { return kRowTableBytes + kRankBytes; }

int build_sketch_table(uint64_t inv, void *table, cudaStream_t s) {
  uint8_t *base = static_cast<uint8_t *>(table);
  const uint32_t rows = kSketchTableEntries * (uint32_t)kTableBands;
  sketch_rows_build_kernel<<<ceil_div(rows, 256u), 256, 0, s>>>(
      inv, reinterpret_cast<uint32_t *>(base));
  NGIA_LAUNCHED();
  // the ranks: sort (hash, entry) per band, keep the entries as 16 bits
  const uint32_t total = kSketchTableEntries * (uint32_t)kBands;
  const size_t sort_bytes = radix_sort_scratch_bytes(kSketchTableEntries, kBands);
  void *tmp = nullptr;
  NGIA_CUDA(cudaMallocAsync(&tmp, (size_t)total * 16 + sort_bytes, s));
  uint32_t *keys = static_cast<uint32_t *>(tmp), *vals = keys + total;
  uint32_t *keys_out = vals + total, *vals_out = keys_out + total;
  sketch_keys_build_kernel<<<ceil_div(total, 256u), 256, 0, s>>>(inv, keys, vals);
  NGIA_LAUNCHED();
  int rc = radix_sort_pairs(keys, vals, keys_out, vals_out, kSketchTableEntries, kBands, 0,
                            32, vals_out + total, s);
  if (rc == NGIA_OK) {
    narrow_kernel<<<ceil_div(total, 256u), 256, 0, s>>>(
        vals_out, reinterpret_cast<uint16_t *>(base + kRowTableBytes), total);
    NGIA_LAUNCHED();
  }
  NGIA_CUDA(cudaFreeAsync(tmp, s));
  return rc;
}

int launch_sketch_table(const uint32_t *packed, const uint32_t *dense, const uint64_t *offs,
                        uint32_t n, uint64_t words, uint64_t inv, const void *table,
                        uint32_t *sigs, uint32_t stride, cudaStream_t s, cudaStream_t side,
                        cudaEvent_t fork, cudaEvent_t join) {
  if (n == 0) return NGIA_OK;
  int dev = 0, sms = 0;
  NGIA_CUDA(cudaGetDevice(&dev));
  NGIA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint8_t *base = static_cast<const uint8_t *>(table);
  // Both kernels' grids by the one lookup that, per device, also asks for the
  // most shared memory: a multiprocessor's split between L1 and shared memory
  // changes only while it is empty, and without that wish the short records'
  // kernel, which uses no shared memory, keeps the rank walk's blocks out until
  // it ends (200,000 nucleotide reads: 1.55 ms one after the other, 1.24 beside
  // each other).
  uint32_t rank_grid = 0, table_grid = 0;
  NGIA_TRY(persistent_grid(reinterpret_cast<const void *>(sketch_rank_kernel), kRankWarps * 32, 0,
                           ceil_div(n, (uint32_t)kRankWarps), &rank_grid));
  NGIA_TRY(persistent_grid(reinterpret_cast<const void *>(sketch_table_kernel), 256, 0,
                           std::min(ceil_div(n, 8u), (uint32_t)sms), &table_grid));
  // The rank walk's residency is bound by its bit sets (shared memory), which
  // leaves each SM room in threads and registers for one block of the short
  // records' kernel (no shared memory): one block per SM, beside it.
  NGIA_CUDA(cudaEventRecord(fork, s));
  NGIA_CUDA(cudaStreamWaitEvent(side, fork, 0));
  sketch_table_kernel<<<table_grid, 256, 0, side>>>(
      packed, dense, offs, n, words, reinterpret_cast<const uint4 *>(base), sigs, stride);
  NGIA_LAUNCHED();
  sketch_rank_kernel<<<rank_grid, kRankWarps * 32, 0, s>>>(
      dense, offs, n, words, inv, reinterpret_cast<const uint16_t *>(base + kRowTableBytes),
      sigs, stride);
  NGIA_LAUNCHED();
  if (join) {
    NGIA_CUDA(cudaEventRecord(join, side));
    NGIA_CUDA(cudaStreamWaitEvent(s, join, 0));
  }
  return NGIA_OK;
}

}  // namespace ngia

extern "C" int ngia_sketch_table_bands(void) { return ngia::kTableBands; }

extern "C" int ngia_sketch(const uint32_t *d_packed, const uint64_t *d_rec_offsets,
                           uint32_t n, uint32_t *d_sigs, void *stream) {
  if (n == 0) return NGIA_OK;
  if (!d_packed || !d_rec_offsets || !d_sigs) return NGIA_ERR_ARG;
  return ngia::launch_sketch(d_packed, d_rec_offsets, n, d_sigs, ngia::as_stream(stream));
}
