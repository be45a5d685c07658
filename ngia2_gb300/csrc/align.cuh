// align.cuh -- banded bit-parallel LCS of one (rep, tar) pair (internal header).
//
// Restates BuildGraph::kernel_dynamic (src/buildGraph.hpp:192-253), identical
// to FastClustering::kernel_dynamic (src/fastClustering.hpp:183-244).
//
// Recurrence.  Rows are the representative's residues, columns the target's.
// A row bit is 1 while the row is unmatched.  One column step with match mask
// M (rows whose 4-bit code equals the column's code; code 0 matches nothing)
// is the bit-parallel LCS update
//     V' = (V + (V & M) + carry_in) | (V & ~M)
// applied to the multi-word vector of the rows inside the band, the carry
// rippling upward from the band's lowest row block (carry 0 there).  The
// reference applies it block by block (32 columns x 32 rows, column carries
// kept in a shift register); here one column step updates every live row
// word at once, which is the same set of dependencies evaluated in another
// order, and the word-to-word carry is the hardware carry flag.
//
// The live row blocks are at most min(ls + rs, nr) words and both ends advance
// by at most one block per column block.  A row block above them is all ones
// with empty masks -- the "not yet visited" state of the reference -- and only
// passes a carry; one below is frozen.  The batched and drop-in kernels hold
// them in registers (align_window.cuh) or over a group of lanes
// (align_group.cuh); the general form below holds any number in local memory.
//
// The general form computes match masks from the bit planes:
//   u = (P0 & T0) | (~P0 & B);  u &= ~(Pe ^ Te) for e = 1..3;  t = V & u
// where Te = all-ones if bit e of the column code is set, B = ~T0 & (T1|T2|T3)
// (so a zero column code gives u = 0).  Since t = V & M is a subset of V,
// V & ~M = V ^ t and the update is V' = (V + t + c) | (V ^ t).
#pragma once

#include "carry_chain.cuh"
#include "common.cuh"

namespace ngia {

// Column-code masks of a target block, one column per step.  The four planes
// are bit-reversed once per block so that column k's bits sit in bit 31 after
// k left shifts; Te = arithmetic shift of that sign bit across the word.
struct ColMask {
  uint32_t T0, T1, T2, T3, B;
};
struct ColumnPlanes {
  uint32_t r0, r1, r2, r3;
  __device__ __forceinline__ explicit ColumnPlanes(const uint32_t *tb) {
#ifdef __CUDA_ARCH__
    r0 = __brev(__ldg(tb));
    r1 = __brev(__ldg(tb + 1));
    r2 = __brev(__ldg(tb + 2));
    r3 = __brev(__ldg(tb + 3));
#endif
  }
  // masks of the next column, then advance
  __device__ __forceinline__ ColMask next() {
    ColMask m;
    m.T0 = (uint32_t)((int32_t)r0 >> 31);
    m.T1 = (uint32_t)((int32_t)r1 >> 31);
    m.T2 = (uint32_t)((int32_t)r2 >> 31);
    m.T3 = (uint32_t)((int32_t)r3 >> 31);
    m.B = ~m.T0 & (m.T1 | m.T2 | m.T3);
    r0 <<= 1;
    r1 <<= 1;
    r2 <<= 1;
    r3 <<= 1;
    return m;
  }
};

__device__ __forceinline__ uint32_t match_and(uint32_t v, uint32_t p0, uint32_t p1,
                                              uint32_t p2, uint32_t p3,
                                              const ColMask &c) {
  uint32_t u = (p0 & c.T0) | (~p0 & c.B);
  u &= ~(p1 ^ c.T1);
  u &= ~(p2 ^ c.T2);
  u &= ~(p3 ^ c.T3);
  return v & u;
}

// General form for any band width: per column block the live rows are
// processed in chunks of 8 words held in `lines` (the row vector, one word per
// row block), with the 32 column carries between chunks kept as one word
// (bit k = carry of column k), like the reference's carry register.
constexpr uint32_t kMaxRowBlocks = (NGIA_MAX_READ + 31) / 32;  // 2048

__device__ inline uint32_t lcs_general(const uint32_t *__restrict__ rep,
                                const uint32_t *__restrict__ tar, const Band &b,
                                uint32_t *lines, uint32_t &blocks) {
  for (uint32_t w = 0; w < b.nr; ++w) lines[w] = kFull;
  uint32_t zeros = 0;  // running LCS: zero bits over all row blocks
  for (uint32_t i = 0; i < b.nc; ++i) {
    const uint32_t j0 = i > b.ls ? i - b.ls : 0;
    const uint32_t j1 = (i + b.rs < b.nr) ? i + b.rs : b.nr;
    const uint32_t *tb = tar + 1 + 4 * i;
    if (i > 0 && !may_reach_threshold(zeros, 32 * i, b)) {  // score 0 certain
      blocks = i;
      return 0;
    }
    uint32_t cin_word = 0;  // carries into the current chunk, bit k = column k
    for (uint32_t j = j0; j < j1; j += 8) {
      uint32_t V[8], P0[8], P1[8], P2[8], P3[8];
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const uint32_t r = j + m;
        if (r < j1) {
          const uint32_t *rb = rep + 1 + 4 * r;
          V[m] = lines[r];
          P0[m] = __ldg(rb);
          P1[m] = __ldg(rb + 1);
          P2[m] = __ldg(rb + 2);
          P3[m] = __ldg(rb + 3);
        } else {
          V[m] = kFull;
          P0[m] = P1[m] = P2[m] = P3[m] = 0;
        }
      }
      uint32_t cout_word = 0;
      ColumnPlanes col(tb);
#pragma unroll 4
      for (int k = 0; k < 32; ++k) {
        const ColMask c = col.next();
        uint32_t t[8], s[8], co;
#pragma unroll
        for (int m = 0; m < 8; ++m) t[m] = match_and(V[m], P0[m], P1[m], P2[m], P3[m], c);
        add_chain8_cc(s, V, t, cin_word & 1u, co);
        cin_word >>= 1;
        cout_word |= co << k;
#pragma unroll
        for (int m = 0; m < 8; ++m) V[m] = s[m] | (V[m] ^ t[m]);
      }
#pragma unroll
      for (int m = 0; m < 8; ++m)
        if (j + m < j1) {
          zeros += __popc(~V[m]) - __popc(~lines[j + m]);
          lines[j + m] = V[m];
        }
      cin_word = cout_word;
    }
  }
  blocks = b.nc;
  return zeros;
}

// Width classes of the batched aligner.  The plan's ladder (width_class):
//   0..10  one pair per lane in a sliding window (align_window.cuh), W = 4, 5,
//          ..., 12, 14, 16 words by stream_width (every width up to 12: a
//          window word above the band costs as much as a live one, and bands
//          of equal ls + rs - 1 are common)
//   11..18 group kernel (align_group.cuh), one pair per group of G lanes with
//          K words per lane: (8,3) (8,4) (16,4) (16,6) (32,4) (32,6) (32,8)
//          (32,16).  A column step costs a lane 3 ops per word plus a fixed
//          ~6 (carry pop and push, code, table row), and a band of span S
//          keeps about S / (K + 1) of the G lanes live, so the ladder takes
//          each span to the shape with the fewest issue slots per cell: eight
//          lanes of three or four words for the 17-36-word bands of medium
//          proteins rather than sixteen lanes of one or two
//   19     general kernel, one pair per thread (any width)
//   20     pairs failing the length filter (score 0, not launched)
// and, with a plan that sends every window of 16 words to the lanes, the
// further one-pair-per-lane classes that round_class prefers:
//   21..24 sliding windows of 18, 20, 24, 28 words
//   25..31 fixed windows (the whole rep) of 8, 10, 12, 14, 16, 20, 24 words
constexpr int kNumLdsClasses = 11;
constexpr int kFirstGroupClass = 11;
constexpr int kNumGroupClasses = 8;
constexpr int kGeneralClass = kFirstGroupClass + kNumGroupClasses;
constexpr int kSkipClass = kGeneralClass + 1;
constexpr int kNumClasses = kSkipClass + 1;
constexpr int kFirstWideClass = kNumClasses, kNumWideClasses = 4;
constexpr int kFirstFixedClass = kFirstWideClass + kNumWideClasses, kNumFixedClasses = 7;
constexpr int kNumRoundClasses = kFirstFixedClass + kNumFixedClasses;

struct GroupShape {
  int G, K;
};
__host__ __device__ constexpr GroupShape group_shape(int c) {
  return c == kFirstGroupClass ? GroupShape{8, 3}
       : c == kFirstGroupClass + 1 ? GroupShape{8, 4}
       : c == kFirstGroupClass + 2 ? GroupShape{16, 4}
       : c == kFirstGroupClass + 3 ? GroupShape{16, 6}
       : c == kFirstGroupClass + 4 ? GroupShape{32, 4}
       : c == kFirstGroupClass + 5 ? GroupShape{32, 6}
       : c == kFirstGroupClass + 6 ? GroupShape{32, 8}
                                   : GroupShape{32, 16};
}

__host__ __device__ constexpr int class_width(int c) {
  return c < 9 ? 4 + c : c == 9 ? 14 : c == 10 ? 16 : 0;
}

// Window words of the further classes.
__host__ __device__ constexpr int wide_width(int k) {
  return k == 0 ? 18 : k == 1 ? 20 : k == 2 ? 24 : 28;
}
__host__ __device__ constexpr int fixed_width(int k) {
  return k < 5 ? 8 + 2 * k : k == 5 ? 20 : 24;
}

constexpr uint32_t kWidestWindow = 28;

// The widest sliding window for tables of K entries per row word: a 28-word
// window of 16-entry tables would leave a multiprocessor's shared memory to
// three warps, which is no faster than the groups (1,000,003 proteins at
// identity 50, align: 9.24 ms with, 9.26 without it; 2 million heavy-tailed
// pairs: 6.7 and 6.0).
__host__ __device__ constexpr uint32_t widest_window(int K) {
  return K > 8 ? 24u : kWidestWindow;
}

// Window a streaming kernel needs for a pair: the live rows of block i,
// [max(i - ls, 0), min(i + rs, nr)), inside [i - ls, i - ls + W).
__host__ __device__ inline uint32_t stream_width(const Band &b) {
  return b.ls + (b.rs < b.nr ? b.rs : b.nr);
}

// A group of G lanes with K words per lane holds at most one live slice per
// lane when the rep has at most G slices or ls + rs <= (G - 1)K + G.
__host__ __device__ inline bool group_fits(const Band &b, int G, int K) {
  const uint32_t ns = (b.nr + K - 1) / K;
  return ns <= (uint32_t)G || b.ls + b.rs <= (uint32_t)((G - 1) * K + G);
}

// Largest ls + rs a group class can hold with one live slice per lane.
__host__ __device__ constexpr uint32_t group_span_limit(int c) {
  return (uint32_t)((group_shape(c).G - 1) * group_shape(c).K + group_shape(c).G);
}

// The binning plan (what an autotuner picks): the widest window sent to the
// one-pair-per-lane kernels, and per group class the widest band (ls + rs) it
// takes (0: class unused; never above group_span_limit).  A pair goes to the
// first class that takes it; reps of at most G slices fit a group class of G
// lanes whatever the band (each slice has its own lane).
struct ClassPlan {
  uint32_t stream_max;
  uint32_t group_limit[kNumGroupClasses];
};

__host__ __device__ inline ClassPlan default_plan() {
  ClassPlan p{16, {}};
  for (int g = 0; g < kNumGroupClasses; ++g) p.group_limit[g] = group_span_limit(kFirstGroupClass + g);
  return p;
}

__host__ __device__ inline int width_class(const Band &b, const ClassPlan &plan) {
  if (!b.pass) return kSkipClass;
  const uint32_t ws = stream_width(b);
  if (ws <= plan.stream_max) return ws <= 4 ? 0 : ws <= 12 ? (int)ws - 4 : ws <= 14 ? 9 : 10;
  for (int g = 0; g < kNumGroupClasses; ++g) {
    const uint32_t lim = plan.group_limit[g];
    if (lim == 0) continue;
    const GroupShape sh = group_shape(kFirstGroupClass + g);
    const uint32_t ns = (b.nr + sh.K - 1) / sh.K;
    if (ns <= (uint32_t)sh.G || b.ls + b.rs <= lim) return kFirstGroupClass + g;
  }
  return kGeneralClass;
}

__host__ __device__ inline int width_class(const Band &b) {
  return width_class(b, default_plan());
}

// The class a round runs a pair in.  It is width_class's, except that with
// stream_max 16 (every window the ladder has) a pair also has the classes
// above: sliding windows up to `widest` words instead of a group of lanes, and
// a fixed window where the rep is short enough for a narrower one than the
// sliding window would be.  Fewest window words wins: the lanes run 3 ALU
// operations per window word and column, so a pair's time is its words.
// Align phase without and with these classes: 1,000,003 proteins at identity
// 50 12.9 -> 9.6 ms, 25,013 nucleotide reads with N at 85 6.4 -> 3.5 ms, 2
// million heavy-tailed protein pairs at 90 8.7 -> 7.8 ms.
__host__ __device__ inline int round_class(const Band &b, const ClassPlan &plan,
                                           uint32_t widest) {
  const int c = width_class(b, plan);
  if (c == kSkipClass || plan.stream_max < 16) return c;
  const uint32_t ws = stream_width(b);
  int slide = c < kNumLdsClasses ? c : -1;
  uint32_t words = slide >= 0 ? (uint32_t)class_width(c) : kFull;
  if (slide < 0 && ws <= widest) {
    slide = ws <= 18 ? 0 : ws <= 20 ? 1 : ws <= 24 ? 2 : 3;
    words = (uint32_t)wide_width(slide);
    slide += kFirstWideClass;
  }
  if (b.nr <= (widest < 24u ? widest : 24u)) {
    const int f = b.nr <= 8 ? 0 : b.nr <= 16 ? (int)(b.nr - 7) / 2 : b.nr <= 20 ? 5 : 6;
    if ((uint32_t)fixed_width(f) < words) return kFirstFixedClass + f;
  }
  return slide >= 0 ? slide : c;
}

// Whether a round over records of at most `longest` residues can have pairs of
// the general class.  A rep of at most G slices goes to a group class of G
// lanes that the plan uses, whatever its band (16,384 residues with the default
// plan), and so does a band within the class's limit: ls + rs is about
// (lr + lt (1 - 2t)) / 32 words, most at the shortest target the length filter
// lets through (t lr) for t > 1/2 and at the longest for less, and up to four
// words more by its roundings.  (An empty launch of the class at identity 90
// cost a round of 2 million pairs of up to 35,000 residues 60 us of 5.88 ms.)
__host__ __device__ inline bool general_possible(const ClassPlan &plan, uint32_t longest,
                                                 float t) {
  const float spread = t > 0.5f ? 1.0f + t - 2.0f * t * t : 2.0f - 2.0f * t;
  const uint32_t rep = (longest + 31) / 32;
  const uint32_t band = (uint32_t)((float)longest * spread / 32.0f) + 5;
  for (int g = 0; g < kNumGroupClasses; ++g) {
    const GroupShape sh = group_shape(kFirstGroupClass + g);
    const uint32_t lim = plan.group_limit[g];
    if (lim && (rep <= (uint32_t)(sh.G * sh.K) || band <= lim)) return false;
  }
  return true;
}

// Queue order inside a class: longest targets first.  The sort key of a pair
// is class-major, then 7 - floor(log2 nc) (column blocks in octaves, capped
// at 7), in eight bits.
__host__ __device__ inline uint32_t class_sort_key(int cls, const Band &b) {
  uint32_t h = 0;  // floor(log2 nc)
  if (b.nc > 1) {
#ifdef __CUDA_ARCH__
    h = 31u - (uint32_t)__clz(b.nc);
#else
    h = 31u - (uint32_t)__builtin_clz(b.nc);
#endif
  }
  return ((uint32_t)cls << 3) | (7u - (h < 7u ? h : 7u));
}
constexpr uint32_t kQueueKeys = 256;
static_assert(kNumRoundClasses <= 32, "class sort key: 5 class bits");
__host__ __device__ constexpr uint32_t skip_sort_key() { return ((uint32_t)kSkipClass << 3) | 7u; }

}  // namespace ngia
