// align_window.cuh -- the batched aligner's kernel body for bands of up to 28
// row words: each lane of a warp aligns its own stream of pairs, the band's
// row words in registers, match masks from its table in shared memory
// (align_lds.cuh; internal header).
//
// Sliding window (kSlide).  At column block i a lane holds rows i - lv .. i -
// lv + W - 1, lv = W - min(rs, nr), so the row that enters the band always
// takes the top word.  Every step the whole warp slides its windows by one
// word: the bottom word's zeros are counted and the registers move down one
// place (W moves against 3 ALU operations per word and column, 32 columns).
// The tables do not move: they hold NS > W slots and the window starts at slot
// `base`, the same in every lane, which advances with it; when the window
// reaches the last slot its masks are copied down to slot 0.  So one copy of
// the column code, its eight columns of a code word unrolled, serves every
// position of the window.  Covers pairs with ls + min(rs, nr) <= W.
//
// Fixed window.  A rep of at most W row words is held whole, row r in word r.
// Nothing slides; covers pairs with nr <= W whatever their band, which at low
// identities is narrower than ls + min(rs, nr).
//
// Words outside the band cost no table writes where that can be had.  Rows
// below 0 are words of zeros: they match nothing (V & M = 0), so they stay
// zero and pass a zero carry, whatever their masks hold; their zeros are taken
// off the count.  Words above the rows that have entered hold anything -- no
// carry comes down from them -- and are set to all ones when their row enters
// and not counted before.  Only a row that has left the band while its word is
// still held (lv > ls, or a fixed window) has its masks cleared, after which
// the word keeps its zeros and passes the zero carry below it.
//
// What bounds it: the integer ALU, 3 operations per word and column at 64
// lanes/clk/SM (6.2e12 word steps/s).  The column loop alone reaches 5.0e12
// word steps/s at 8 warps per SM and 4.6e12 at 4 (W = 8, 8 columns unrolled;
// 4.4e12 and 3.4e12 with 2 unrolled), which is why code for one window
// position with 8 columns unrolled is worth the register moves and the copied
// masks over code per position with 2, and why windows of 18 to 28 words,
// whose tables leave room for 4 warps per SM, still beat a group of lanes per
// pair (align_group.cuh: a carry popped and pushed per column and slice, and
// 58-67 % of lanes live).
//
// Streams.  A lane whose pair ends (last column block, or a score of 0 already
// certain) writes the score and takes the next pair of its warp's chunk (32
// pairs claimed from the class's queue with one atomic), so the lanes stay
// busy until the queue drains.  Pairs are queued longest first.
#pragma once

#include "align_lds.cuh"
#include "kernels.cuh"

namespace ngia {

// A queued pair, as staged for a refill.
struct PairDesc {
  uint32_t p, len, band;  // pair index; lr, lt and ls, rs as 16-bit halves
  uint64_t ro, to;        // record offsets of rep and target
};

__device__ __forceinline__ uint64_t shfl64(uint64_t v, uint32_t src) {
  const uint32_t lo = __shfl_sync(kFull, (uint32_t)v, src);
  const uint32_t hi = __shfl_sync(kFull, (uint32_t)(v >> 32), src);
  return ((uint64_t)hi << 32) | lo;
}

// One lane's pair.
struct WindowPair {
  const uint32_t *rep;  // rep record (length word, then bit planes)
  const uint32_t *tar;  // target's nibble code words
  uint32_t p;           // pair index (score slot)
  uint32_t i;           // current column block
  uint32_t nc, nr, rs, ls;
  uint32_t act;         // rows entered so far
  int32_t lcs;          // zeros of the words slid out, less 32 per row below 0
  uint32_t lr, lt;
  uint4 cur;            // code words of block i
  uint4 pf;             // planes of row pf_row, loaded one block ahead
  uint32_t pf_row;
  bool active;
};

// 32 column steps of one column block; tab: the window's first slot.
template <int W, int NS>
__device__ __forceinline__ void window_columns(uint32_t (&V)[W], const uint32_t *tab,
                                               const uint4 &nib) {
  uint32_t w0 = nib.x, w1 = nib.y, w2 = nib.z, w3 = nib.w;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    uint32_t x = w0;
    w0 = w1;
    w1 = w2;
    w2 = w3;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t *row = tab + (x >> 28) * (uint32_t)(NS * 32);
      x <<= 4;
      uint32_t t[W], s[W];
#pragma unroll
      for (int m = 0; m < W; ++m) t[m] = V[m] & row[m * 32];
      add_run<W>(s, V, t);
#pragma unroll
      for (int m = 0; m < W; ++m) V[m] = s[m] | (V[m] ^ t[m]);
    }
  }
}

// One column block of the warp's pairs (the tables already at `base`): slide,
// let the next rows enter, 32 column steps, then for a lane with a pair
//   total = the LCS so far, ub = an upper bound of the pair's final LCS.
// kPlanes: the target's words are bit planes, made into codes here.
//
// The early exit (see align.cuh): the banded LCS is the best monotone path
// through the matrix counting matches in band cells only (rows below the band
// hold their values, rows above it enter all ones with empty masks).  Such a
// path crosses the last column done at some row j, so the final LCS is at
// most  L(j) + min(columns left, Lr - j)  with L(j) the zeros of rows 0..j
// now; taken at word granularity (zeros through a word's end, rows above its
// start) and over the retired rows.
template <int W, int NS, int K, bool kSlide, bool kPlanes>
__device__ __forceinline__ void window_block(uint32_t (&V)[W], WindowPair &sp,
                                             const LdsTable<NS, K> &tab, uint32_t base,
                                             int32_t &total, int32_t &ub) {
  const uint32_t lv = kSlide ? W - min(sp.rs, sp.nr) : 0u;
  uint32_t j1 = 0;
  uint4 nxt = sp.cur, pfn = sp.pf;
  uint32_t pfn_row = sp.pf_row;
  if (sp.active) {
    if constexpr (kSlide) {
      // the word sliding out is row i - lv - 1; past the rep's end it holds
      // nothing to count
      if ((int32_t)(sp.i - lv - 1) < (int32_t)sp.nr) sp.lcs += __popc(~V[0]);
#pragma unroll
      for (int m = 0; m + 1 < W; ++m) V[m] = V[m + 1];
      V[W - 1] = kFull;
    }
    // the next block's code words and entering row (J1 moves up at most one
    // row per block), loaded now so that their latency hides behind this block
    const bool more = sp.i + 1 < sp.nc;
    if (more) nxt = load4(sp.tar + 4 * (sp.i + 1));
    j1 = sp.i + sp.rs < sp.nr ? sp.i + sp.rs : sp.nr;
    const uint32_t j1n = sp.i + 1 + sp.rs < sp.nr ? sp.i + 1 + sp.rs : sp.nr;
    if (more && j1n > j1) {
      pfn_row = j1n - 1;
      pfn = load4(sp.rep + 1 + 4 * pfn_row);
    }
    // slot of row r: base + (r - (i - lv)) sliding, r fixed
    const uint32_t slot0 = kSlide ? base + lv - sp.i : 0u;
    if (sp.i > sp.ls && sp.i - sp.ls <= sp.nr && (!kSlide || lv > sp.ls))
      tab.clear(slot0 + sp.i - sp.ls - 1);  // the row leaving the band
    if constexpr (!kSlide) {
#pragma unroll
      for (int m = 0; m < W; ++m)
        if ((uint32_t)m >= sp.act) V[m] = kFull;
    }
    while (sp.act < j1) {
      if (sp.act == sp.pf_row) {
        tab.fill(slot0 + sp.act, sp.pf);
        ++sp.act;
      } else {  // a pair's first block: four rows' loads together
        uint4 r[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
          if (sp.act + k < j1) r[k] = load4(sp.rep + 1 + 4 * (sp.act + k));
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
          if (sp.act + k < j1) tab.fill(slot0 + sp.act + k, r[k]);
        sp.act = min(sp.act + 4, j1);
      }
    }
  }
  // the whole warp together (a lane without a pair steps on what its words
  // and masks hold, which its next start replaces)
  __syncwarp();
  window_columns<W, NS>(V, tab.base + base * 32, kPlanes ? planes_to_nibbles(sp.cur) : sp.cur);
  if (sp.active) {
    ++sp.i;
    const int32_t cols = 32 * (int32_t)sp.i;
    const int32_t left = (int32_t)sp.lt > cols ? (int32_t)sp.lt - cols : 0;
    // rows above the first row of word 0
    const int32_t above0 =
        (int32_t)sp.lr - (kSlide ? 32 * ((int32_t)sp.i - 1 - (int32_t)lv) : 0);
    total = kSlide ? sp.lcs : 0;
    ub = max(total, 0) + min(left, (int32_t)sp.lr);
#pragma unroll
    for (int m = 0; m < W; ++m) {
      const int32_t above = above0 - 32 * m;
      if (kSlide ? above > 0 : (uint32_t)m < j1) {
        total += __popc(~V[m]);
        ub = max(ub, total + min(left, above));
      }
    }
    sp.cur = nxt;
    sp.pf = pfn;
    sp.pf_row = pfn_row;
  }
}

// Advances the tables of a sliding window by one slot.
template <int W, int NS, int K>
__device__ __forceinline__ void window_advance(const LdsTable<NS, K> &tab, uint32_t &base) {
  if (base + W == NS) {
#pragma unroll 1
    for (uint32_t s = 0; s + 1 < (uint32_t)W; ++s) tab.move(s, base + 1 + s);
    base = 0;
  } else {
    ++base;
  }
}

// A sliding window's words before a pair's first block (and its slide): rows
// below 0 are zeros, taken off the count.
template <int W>
__device__ __forceinline__ void window_start(uint32_t (&V)[W], WindowPair &sp) {
  const uint32_t lv = W - min(sp.rs, sp.nr);
  sp.lcs = -32 * (int32_t)(lv + 1);
#pragma unroll
  for (int m = 0; m < W; ++m) V[m] = (uint32_t)m <= lv ? 0u : kFull;
}

// One class of the round on this warp: takes pairs from order[bounds[cls],
// bounds[cls + 1]) until the queue is empty.  col: the lane's column of the
// warp's table of NS slots, whose code-0 row holds zeros.  Returns the lane's
// column blocks x W.
//
// Lanes start new pairs only every kStartEvery-th step (or when no lane has
// one).  A start costs the warp the new rows' loads and table writes whatever
// the lanes that start, so with 16-entry tables fewer, fuller starts are worth
// the idle steps (1,000,003 proteins at identity 50, align: 9.74 ms starting
// at every step, 9.48 at every second, 9.29 third, 9.37 fourth); with 5 and 8
// entries they are not (200,000 nucleotide reads: 3.26, every second 3.31).
template <int W, int NS, int K, bool kSlide>
__device__ __forceinline__ uint32_t align_window(const RoundArgs &a, int cls, uint32_t *col) {
  static_assert(kSlide ? NS > W : NS >= W, "slots");
  constexpr uint32_t kStartEvery = K == 16 ? 3 : 1;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t begin = a.bounds[cls], size = a.bounds[cls + 1] - begin;
  if (size == 0) return 0;
  const LdsTable<NS, K> tab{col};
  uint32_t V[W];
#pragma unroll
  for (int m = 0; m < W; ++m) V[m] = kFull;
  WindowPair sp{};
  // Pair descriptors, staged per warp: lane l of A holds the l-th pair of the
  // warp's current chunk of 32, so a refill waits on global memory once per
  // 32 pairs.
  PairDesc A{};
  uint32_t a_count = 0, a_used = 0;  // warp-uniform
  bool queue_empty = false;
  uint32_t done = 0, base = 0, step = 0;
  for (;; ++step) {
    // lanes without a pair take the next descriptors of A, a new chunk being
    // claimed when A runs out
    uint32_t need = __ballot_sync(kFull, !sp.active);
    if (step % kStartEvery != 0 && need != kFull) need = 0;
    while (need) {
      if (a_used == a_count) {
        if (queue_empty) break;
        uint32_t first = 0;
        if (lane == 0) first = atomicAdd(a.cursors + cls, 32u);
        first = __shfl_sync(kFull, first, 0);
        a_count = first < size ? min(size - first, 32u) : 0u;
        a_used = 0;
        if (a_count == 0) {
          queue_empty = true;
          break;
        }
        if (lane < a_count) {
          A.p = a.order[begin + first + lane];
          const uint2 pr = a.pairs[A.p];
          A.ro = a.offs[pr.x];
          A.to = a.offs[pr.y];
          const uint32_t lr = __ldg(a.lens + pr.x), lt = __ldg(a.lens + pr.y);
          const Band b = make_band(lr, lt, a.t, a.fm);
          A.len = lr | lt << 16;
          A.band = b.ls | b.rs << 16;
        }
      }
      const uint32_t rank = __popc(need & ((1u << lane) - 1u));
      const uint32_t take = min((uint32_t)__popc(need), a_count - a_used);
      const uint32_t src = a_used + (rank < take ? rank : 0u);
      const uint32_t p = __shfl_sync(kFull, A.p, src);
      const uint32_t len = __shfl_sync(kFull, A.len, src);
      const uint32_t band = __shfl_sync(kFull, A.band, src);
      const uint64_t ro = shfl64(A.ro, src), to = shfl64(A.to, src);
      const bool mine = (need >> lane & 1u) && rank < take;
      if (mine) {
        sp.lr = len & 0xFFFFu;
        sp.lt = len >> 16;
        // no columns, or no row to enter the window (a sliding window's words
        // below row 0 assume one does)
        if (sp.lt == 0 || sp.lr == 0) {
          a.scores[p] = identity_score(0u, sp.lr, sp.lt, a.t);
        } else {
          sp.rep = a.rows + ro;
          sp.tar = a.nib + to + 1;
          sp.cur = load4(sp.tar);
          sp.p = p;
          sp.i = 0;
          sp.nc = (sp.lt + 31u) >> 5;
          sp.nr = (sp.lr + 31u) >> 5;
          sp.rs = band >> 16;
          sp.ls = band & 0xFFFFu;
          sp.act = 0;
          sp.pf_row = kFull;
          sp.active = true;
          if constexpr (kSlide) window_start(V, sp);
        }
      }
      a_used += take;
      need &= ~__ballot_sync(kFull, mine);
      // lanes whose pair needed no alignment ask again
      need |= __ballot_sync(kFull, mine && !sp.active);
    }
    if (!__any_sync(kFull, sp.active)) {
      if (queue_empty) break;
      continue;
    }
    // every lane, with or without a pair
    if constexpr (kSlide) window_advance<W>(tab, base);
    int32_t total = 0, ub = 0;
    window_block<W, NS, K, kSlide, false>(V, sp, tab, base, total, ub);
    if (sp.active) {
      done += W;
      const bool last = sp.i >= sp.nc;
      if (last || !lcs_may_reach((uint32_t)ub, sp.lr, sp.lt, a.t)) {
        a.scores[sp.p] = last ? identity_score((uint32_t)total, sp.lr, sp.lt, a.t) : 0u;
        sp.active = false;
      }
    }
  }
  return done;
}

}  // namespace ngia
