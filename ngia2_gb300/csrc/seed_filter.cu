// seed_filter.cu -- pairs that cannot reach the identity, told by the short
// words their sequences share (no counterpart in the reference, which aligns
// every candidate).
//
// Cut the rep into blocks of q residues.  A block whose word does not occur in
// the target costs any common subsequence of the two at least one unmatched
// residue: either one of the block's own, or one of the target's between the
// partners of two neighbours of the block, and no two blocks share one.  So
// with E such blocks  (Lr - lcs) + (Lt - lcs) >= E,  and the banded LCS, a
// common subsequence, is at most (Lr + Lt - E) / 2.  Once that fails the
// identity test the pair's score is 0 and it leaves the round before it is
// aligned; a pair that stays is aligned as before.
//
// A warp takes runs of the pairs in their order, in which a graph build's are
// grouped by target.  It marks the target's words in a set of 65,536 bits in
// shared memory (q = 4 residue codes are the 16 bits themselves, q = 8 aligner
// codes of a recoded database are hashed to them; a chance hit only loses
// evidence), and then counts the rep's words that miss the set until the count
// decides: four pairs of the target at a time, eight lanes each, or a single
// one by the whole warp, four code words per lane between two looks at the
// count and the next four on their way.
//
// What bounds it: the shared-memory pipe (random bits, 3.4 wavefronts a test or
// mark; 70 % of its rate) and issue slots (60 %), some 80 warp instructions a
// pair.  200,000 nucleotide reads at identity 95, 9.4 million pairs: 1.2 ms,
// after which 0.53 ms of alignment are left of 3.12.  A set of 8,192 bytes,
// marked without atomics, was no faster and told fewer pairs; four-byte loads
// took 1.4 times as long.
#include "align.cuh"
#include "kernels.cuh"

namespace ngia {

constexpr uint32_t kSeedWarps = 4;           // per block
constexpr uint32_t kSeedWords = 65536 / 32;  // the set

// The bit of a word (in the top 4Q bits of w) in the set.
template <int Q>
__device__ __forceinline__ uint32_t seed_index(uint32_t w) {
  return Q == 4 ? w >> 16 : (w * 0x9E3779B1u) >> 16;
}

// Makes the set that of the words starting in code words [first, end) of a
// target of n code words at w (the warp together).
template <int Q>
__device__ __forceinline__ void seed_mark(uint32_t *set, const uint32_t *w, uint32_t first,
                                          uint32_t end, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u;
  uint4 *set4 = reinterpret_cast<uint4 *>(set);
  __syncwarp();
#pragma unroll
  for (uint32_t s = 0; s < kSeedWords / 128; ++s)
    set4[s * 32 + lane] = make_uint4(s == 0 && lane == 0 ? 1u : 0u, 0, 0, 0);
  __syncwarp();
#pragma unroll 2
  for (uint32_t i = first + lane; i < end; i += 32) {
    const uint32_t a = __ldg(w + i), b = i + 1 < n ? __ldg(w + i + 1) : 0u;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const uint32_t e = seed_index<Q>(__funnelshift_l(b, a, 4 * r));
      atomicOr(set + (e >> 5), 1u << (e & 31u));
    }
  }
  __syncwarp();
}

// Least evidence E that settles the pair: (lr + lt - E) / 2 fails the test.
__device__ __forceinline__ uint32_t seed_need(uint32_t lr, uint32_t lt, float t) {
  const uint32_t sum = lr + lt, cap = lr < lt ? lr : lt;
  const float guess = (1.0f - t) / (1.0f + t) * (float)sum;
  uint32_t e = guess > 3.0f ? (uint32_t)guess - 3u : 0u;
  while (e <= sum && score_positive(min((sum - e) / 2, cap), lr, lt, t)) ++e;
  return e;
}

__device__ __forceinline__ uint64_t shfl64(uint64_t v, uint32_t src) {
  const uint32_t lo = __shfl_sync(kFull, (uint32_t)v, src);
  const uint32_t hi = __shfl_sync(kFull, (uint32_t)(v >> 32), src);
  return ((uint64_t)hi << 32) | lo;
}

// How many words of a rep miss the set, counted until they are `goal` or what
// is left cannot make them so.  The rep's `blocks` code words at nib + at, from
// the first 16-byte boundary on in whole groups of four, are tested by P lanes
// (a group of the warp; the whole warp calls, groups with nothing to test with
// blocks = 0): one 16-byte load per lane in place of four of four bytes, which
// cost the load pipe three times as much.  A place past the end is the zero
// word, which every set holds.
template <int Q, int P>
__device__ __forceinline__ uint32_t seed_count(const uint32_t *set, const uint32_t *nib,
                                               uint64_t at, uint32_t blocks, uint32_t goal) {
  constexpr uint32_t kPer = 8 / Q;          // tests per code word
  constexpr uint32_t kStep = 4 * P * kPer;  // per pass of the P lanes
  const uint32_t i0 = threadIdx.x & (uint32_t)(P - 1), skip = (uint32_t)(0 - at) & 3u;
  const int32_t groups = blocks > skip ? (int32_t)((blocks - skip) >> 2) : 0;
  const uint4 *w = reinterpret_cast<const uint4 *>(nib + at + skip) + i0;
  int32_t left = groups - (int32_t)i0;  // this lane's groups are those of every P-th place
  uint32_t found = 0, tested = 0;
  uint4 next = left > 0 ? __ldg(w) : make_uint4(0, 0, 0, 0);
  bool have = true;
  for (;;) {
    uint4 cur = next;
    if (!have && left > 0) cur = __ldg(w);
    w += P;
    left -= P;
    tested += kStep;
    // the next group is on its way meanwhile, unless this pass should do
    have = tested < goal + (goal >> 3);
    next = left > 0 && have ? __ldg(w) : make_uint4(0, 0, 0, 0);
    const uint32_t word[4] = {cur.x, cur.y, cur.z, cur.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (uint32_t h = 0; h < kPer; ++h) {
        const uint32_t x = seed_index<Q>(word[j] << (16 * h));
        found += (set[x >> 5] >> (x & 31u)) & 1u;
      }
    const int32_t rest = left + (int32_t)i0;  // groups after this pass
    // looked at once the words tested could settle a pair, or none is left
    if (!__any_sync(kFull, tested >= goal || rest <= 0)) continue;
    uint32_t f = found;
    if constexpr (P == 32) {
      f = __reduce_add_sync(kFull, f);
    } else {
#pragma unroll
      for (int o = 1; o < P; o <<= 1) f += __shfl_xor_sync(kFull, f, o);
    }
    const uint32_t missed = tested - f;  // (places past the end count as found)
    if (__all_sync(kFull, missed >= goal || rest <= 0 || missed + 4 * kPer * rest < goal))
      return missed;
  }
}

// The same for a long target, a window of the rep at a time: a common
// subsequence inside the band pairs row r only with columns of blocks r / 32 -
// rs + 1 .. r / 32 + ls, so a word of the rep's window counts as missing when it
// does not start in the columns that the window reaches.  Windows as long as
// the band is wide mark each of the target's words about twice.
template <int Q>
__device__ __forceinline__ bool seed_windows(uint32_t *set, const uint32_t *nib, uint64_t rep_at,
                                             uint32_t blocks, uint64_t tar_at, uint32_t tar_words,
                                             uint32_t ls, uint32_t rs, uint32_t goal) {
  constexpr uint32_t kPer = 8 / Q;
  const uint32_t size = 4u * max(ls + rs, 64u);  // code words of a window (four per row block)
  uint32_t missed = 0;
  for (uint32_t s = 0; s < blocks; s += size) {
    const uint32_t n = min(size, blocks - s);
    const uint32_t row0 = s >> 2, row1 = (s + n - 1) >> 2;  // row blocks
    const uint32_t from = row0 + 1 > rs ? 4 * (row0 + 1 - rs) : 0u;
    seed_mark<Q>(set, nib + tar_at, min(from, tar_words), min(4 * (row1 + ls + 1), tar_words),
                 tar_words);
    missed += seed_count<Q, 32>(set, nib, rep_at + s, n, goal - missed);
    const uint32_t left = kPer * (blocks - s - n);
    if (missed >= goal || missed + left < goal) break;
  }
  return missed >= goal;
}

template <int Q>
__global__ void __launch_bounds__(kSeedWarps * 32)
seed_filter_kernel(const uint32_t *__restrict__ nib, const uint64_t *__restrict__ offs,
                   const uint32_t *__restrict__ lens, const uint2 *__restrict__ pairs,
                   uint32_t m, float t, int fma_mode, uint8_t *__restrict__ keys,
                   unsigned int *__restrict__ key_count, unsigned int *__restrict__ cursor,
                   uint32_t run) {
  __shared__ __align__(16) uint32_t sets[kSeedWarps][kSeedWords];
  __shared__ unsigned int out[kQueueKeys];
  constexpr uint32_t kPer = 8 / Q;  // tests per code word
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t *set = sets[threadIdx.x >> 5];
  for (uint32_t k = threadIdx.x; k < kQueueKeys; k += kSeedWarps * 32) out[k] = 0;
  __syncthreads();
  uint32_t target = kFull;  // whose words the set holds
  for (;;) {
    // runs are counted, not pairs: a sum past m could wrap at 2^32
    uint32_t claim = 0;
    if (lane == 0) claim = atomicAdd(cursor, 1u);
    const uint64_t at = (uint64_t)__shfl_sync(kFull, claim, 0) * run;
    if (at >= m) break;
    const uint32_t first = (uint32_t)at, size = min(run, m - first);
    for (uint32_t base = 0; base < size; base += 32) {
      const uint32_t p = first + base + lane;
      const uint32_t key = base + lane < size ? keys[p] : skip_sort_key();
      uint2 pr = make_uint2(0u, 0u);
      uint32_t lr = 0, lt = 0, need = kFull;
      uint64_t ro = 0, to = 0;
      bool eligible = key >> 3 != (uint32_t)kSkipClass;
      if (eligible) {
        pr = pairs[p];
        lr = __ldg(lens + pr.x);
        lt = __ldg(lens + pr.y);
        ro = offs[pr.x];
        to = offs[pr.y];
        need = seed_need(lr, lt, t);
      }
      // Worth it where the test costs less than the alignment it may save, both
      // in warp instructions: the target's words marked (lt / 4, and its loads
      // waited for, shared by the pairs of these 32 that have it) and about
      // need words tested, against the columns an unrelated pair takes before
      // its exit times its window (a group of lanes takes twice as long).  The
      // factors where they measured best: 200,000 nucleotide reads at 95, whose
      // targets have 47 pairs each, binning and align 3.57 ms without the
      // filter, 2.17 / 2.05 / 2.07 at 1.25 / 0.8 / 0.5; 2 million unordered
      // protein pairs at 90 7.98 ms without, 5.5 / 6.0 at 1.25 / 0.8.
      const uint32_t peers = __match_any_sync(kFull, eligible ? pr.y : kFull - 1u);
      uint32_t ls = 0, rs = 0;
      if (eligible) {
        const Band b = make_band(lr, lt, t, fma_mode);
        ls = b.ls;
        rs = b.rs;
        const uint32_t words = stream_width(b);
        const uint32_t sharers = __popc(peers);
        const float shared = 1.0f / (float)sharers;
        const float align = (float)(need + 64) * (float)(words + 3) * (words > 28 ? 0.25f : 0.125f);
        const float test = ((float)lt * 0.25f + 400.0f) * shared + 40.0f + 0.65f * (float)need;
        eligible = need <= kPer * (lr >> 3) && align > (sharers >= 4 ? 0.8f : 1.25f) * test;
      }
      // The band lets a rep's word meet the target's only within its own reach,
      // so a long target's words are marked a window at a time.
      const bool windows = lt > 4096u + 64u * (ls + rs);
      uint32_t todo = __ballot_sync(kFull, eligible);
      bool drop = false;
      while (todo) {
        const uint32_t k0 = __ffs(todo) - 1;
        const uint32_t tar = __shfl_sync(kFull, pr.y, k0);
        const uint64_t tar_at = shfl64(to, k0) + 1;
        const uint32_t tar_words = (__shfl_sync(kFull, lt, k0) + 7) >> 3;
        if (__shfl_sync(kFull, windows, k0)) {
          const uint32_t hit =
              seed_windows<Q>(set, nib, shfl64(ro, k0) + 1, __shfl_sync(kFull, lr, k0) >> 3,
                              tar_at, tar_words, __shfl_sync(kFull, ls, k0),
                              __shfl_sync(kFull, rs, k0), __shfl_sync(kFull, need, k0));
          if (lane == k0) drop = hit;
          target = kFull;
          todo &= todo - 1;
          continue;
        }
        if (tar != target) {
          target = tar;
          seed_mark<Q>(set, nib + tar_at, 0, tar_words, tar_words);
        }
        uint32_t same = __ballot_sync(kFull, pr.y == tar) & todo;
        if (same & (same - 1)) {  // two pairs of this target or more
          uint32_t k = k0, taken = 0;
          const uint32_t sub = lane >> 3;
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j) {
            if (same) {
              const uint32_t kj = __ffs(same) - 1;
              if (sub == j) k = kj;
              taken |= 1u << kj;
              same &= same - 1;
            }
          }
          const bool mine = sub < (uint32_t)__popc(taken);
          const uint32_t blocks = __shfl_sync(kFull, lr, k) >> 3;
          const uint32_t goal = __shfl_sync(kFull, need, k);
          const uint64_t at = shfl64(ro, k) + 1;
          const bool hit = seed_count<Q, 8>(set, nib, at, mine ? blocks : 0u, goal) >= goal;
          const uint32_t hits = __ballot_sync(kFull, mine && hit);
          // lane l's pair is the rank-th taken, on lanes 8 rank ..
          if (taken >> lane & 1u)
            drop = hits >> (8 * __popc(taken & ((1u << lane) - 1u))) & 1u;
          todo &= ~taken;
        } else {
          const uint32_t blocks = __shfl_sync(kFull, lr, k0) >> 3;
          const uint32_t goal = __shfl_sync(kFull, need, k0);
          const uint64_t at = shfl64(ro, k0) + 1;
          const bool hit = seed_count<Q, 32>(set, nib, at, blocks, goal) >= goal;
          if (lane == k0) drop = hit;
          todo &= todo - 1;
        }
      }
      const uint32_t dropped = __match_any_sync(kFull, drop ? key : kFull);
      if (drop) {
        if ((dropped & ((1u << lane) - 1u)) == 0)
          atomicAdd(&out[key], (unsigned int)__popc(dropped));
        keys[p] = (uint8_t)skip_sort_key();
      }
    }
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < kQueueKeys; k += kSeedWarps * 32)
    if (out[k]) atomicSub(key_count + k, out[k]);
}

int seed_filter(const uint32_t *nib, int K, const uint64_t *offs, const uint32_t *lens,
                const uint2 *pairs, uint32_t m, uint32_t identity, uint8_t *keys,
                unsigned int *key_count, unsigned int *cursor, cudaStream_t s) {
  const uint32_t q = K == 16 ? 4 : 8;
  // every rep of Lr residues has Lr / q blocks, and a pair passes the length
  // filter with at least (1 - t) Lr unmatched to spare: below 1 - 1 / q no
  // pair can be told
  if (m == 0 || identity * q <= 100 * (q - 1)) return NGIA_OK;
  // few pairs of a large alphabet, mostly relatives, are aligned in less than
  // the filter's own latency (38,873 protein pairs: align 59 us without, 55
  // with it, after 24 us of filter)
  if (q == 4 && m < 65536u) return NGIA_OK;
  const float t = identity_threshold(identity);
  const void *func = q == 4 ? reinterpret_cast<const void *>(seed_filter_kernel<4>)
                            : reinterpret_cast<const void *>(seed_filter_kernel<8>);
  uint32_t grid = 0;
  NGIA_TRY(persistent_grid(func, kSeedWarps * 32, 0, ceil_div(m, 32 * kSeedWarps), &grid));
  // pairs claimed at a time: enough claims per warp to even out their lengths,
  // long enough runs that a target is marked by few warps
  uint32_t run = m / (grid * kSeedWarps * 8u) / 32u * 32u;
  run = run < 32u ? 32u : run > 256u ? 256u : run;
  if (q == 4)
    seed_filter_kernel<4><<<grid, kSeedWarps * 32, 0, s>>>(
        nib, offs, lens, pairs, m, t, round_mode(), keys, key_count, cursor, run);
  else
    seed_filter_kernel<8><<<grid, kSeedWarps * 32, 0, s>>>(
        nib, offs, lens, pairs, m, t, round_mode(), keys, key_count, cursor, run);
  NGIA_LAUNCHED();
  return NGIA_OK;
}

}  // namespace ngia
