// align_round.cuh -- the batched round's kernels and their launches for tables
// of K entries (internal header; instantiated by align_k5.cu, align_k8.cu and
// align_k16.cu, one translation unit each so that they compile side by side).
#pragma once

#include "align_group.cuh"
#include "align_window.cuh"
#include "kernels.cuh"

namespace ngia {

// The batched kernels read their classes' ranges of the queue order from
// device memory (bounds[cls] .. bounds[cls + 1], written by the classifier),
// so that a round needs no host round trip and can be captured as a graph.
// Classes share launches by the shared memory they need: a warp goes through
// its kernel's classes, widest first, taking pairs from each until its queue
// is empty (an empty class costs a load).  One launch per class, 20 a round,
// cost the small rounds more than their work: 600 proteins at identity 50
// spent 0.14 ms aligning 1,176 pairs.

// One group class: the block's warps take its pairs (align_group.cuh).
template <int C, int KC>
__device__ __forceinline__ uint32_t group_class(const RoundArgs &a, uint32_t *smem) {
  if (a.bounds[C] == a.bounds[C + 1]) return 0;
  constexpr GroupShape sh = group_shape(C);
  return align_group<sh.G, sh.K, KC>(a.rows, a.nib, a.offs, a.pairs, a.order, a.bounds[C],
                                     a.bounds[C + 1], a.cursors + C, a.scores, a.t, a.fm, smem);
}

// The classes of 32 lanes, widest first: few and long pairs, at most seven warps
// of them per multiprocessor, so that a pair of 30,000 residues does not share
// its scheduler with three others and end the round alone (2 million heavy-tailed
// pairs after the seed filter: 6.3 ms in one kernel with the classes of 8 and 16
// lanes at 14 warps, 4.7 ms here).  Twenty blocks are asked of the registers (96
// a thread): the windows' and groups' warps share the multiprocessor (at 108 and
// 115 registers 2 million pairs lose 2 and 6 %), and as many without the ask gave
// 2,425 pairs at identity 88, one chain of 32 lanes, 823 us instead of 812.
template <int KC>
__global__ void __launch_bounds__(32, 20)
align_wide_kernel(const __grid_constant__ RoundArgs a) {
  extern __shared__ uint32_t smem[];
  uint32_t done = group_class<kFirstGroupClass + 7, KC>(a, smem);
  done += group_class<kFirstGroupClass + 6, KC>(a, smem);
  done += group_class<kFirstGroupClass + 5, KC>(a, smem);
  done += group_class<kFirstGroupClass + 4, KC>(a, smem);
  count_work(done, a.work);
}

// The classes of 16 and 8 lanes, widest first.
template <int KC>
__global__ void __launch_bounds__(kGroupThreads)
align_group_kernel(const __grid_constant__ RoundArgs a) {
  extern __shared__ uint32_t smem[];
  uint32_t *mine = smem + (threadIdx.x >> 5) * (KC * 6 * 32);
  uint32_t done = group_class<kFirstGroupClass + 3, KC>(a, mine);
  done += group_class<kFirstGroupClass + 2, KC>(a, mine);
  done += group_class<kFirstGroupClass + 1, KC>(a, mine);
  done += group_class<kFirstGroupClass, KC>(a, mine);
  count_work(done, a.work);
}

// The one-pair-per-lane classes in kernels by width, one warp per block, a
// table of window_slots(K, tier) slots each: tier 0 windows of 4-8 words, 1 of
// 9-16 (rounds of few pairs), 2 of 18-28, and for other rounds 9-12 and 14-16 by
// themselves (3 and 4), whose tables leave room for eight and six warps per
// multiprocessor with 16 entries (1,000,003 proteins at
// identity 50, align: 9.28 ms as one tier of six, 8.96 so).
__host__ __device__ constexpr int window_slots(int K, int tier) {
  return K == 16 ? (tier == 0 ? 12 : tier == 2 ? 27 : tier == 3 ? 14 : 18)
                 : (tier == 0 ? 16 : tier == 2 ? 36 : tier == 3 ? 18 : 24);
}

// The classes of a tier, widest first.
struct WindowClass {
  int words, cls;
  bool slide;
};
__host__ __device__ constexpr int window_classes(int K, int T) {
  return T == 0 ? 6 : T == 1 ? 10 : T == 3 ? 6 : T == 4 ? 4 : widest_window(K) == 28 ? 6 : 5;
}
__host__ __device__ constexpr WindowClass window_class(int T, int k) {
  constexpr int w = kFirstWideClass, f = kFirstFixedClass;
  constexpr WindowClass t0[] = {{8, 4, true}, {8, f, false}, {7, 3, true},
                                {6, 2, true}, {5, 1, true},  {4, 0, true}};
  constexpr WindowClass t1[] = {{16, 10, true},    {16, f + 4, false}, {14, 9, true},
                                {14, f + 3, false}, {12, 8, true},      {12, f + 2, false},
                                {11, 7, true},      {10, 6, true},      {10, f + 1, false},
                                {9, 5, true}};
  constexpr WindowClass t2[] = {{24, w + 2, true},  {24, f + 6, false}, {20, w + 1, true},
                                {20, f + 5, false}, {18, w, true},      {28, w + 3, true}};
  return T == 0 ? t0[k] : T == 2 ? t2[k] : T == 3 ? t1[4 + k] : t1[k];
}

// The classes from `first` on (kFrom) or those before it, one after another.
template <int K, int T, bool kFrom, int C = 0>
__device__ __forceinline__ uint32_t window_run(const RoundArgs &a, int first, uint32_t *col) {
  if constexpr (C < window_classes(K, T)) {
    constexpr WindowClass w = window_class(T, C);
    uint32_t done = 0;
    if ((C >= first) == kFrom)
      done = align_window<w.words, window_slots(K, T), K, w.slide>(a, w.cls, col);
    return done + window_run<K, T, kFrom, C + 1>(a, first, col);
  }
  return 0;
}

template <int K, int T>
__global__ void __launch_bounds__(32)
align_window_kernel(const __grid_constant__ RoundArgs a) {
  extern __shared__ uint32_t smem[];
  constexpr int NS = window_slots(K, T);
  uint32_t *col = smem + threadIdx.x;
#pragma unroll 1
  for (int s = 0; s < NS; ++s) col[s * 32] = 0u;  // code 0 matches nothing
  // Where this multiprocessor begins: the classes' shares of the tier's work
  // (pairs x window words squared: a pair's columns grow with its window too)
  // laid end to end over the multiprocessors, which then help with the rest.
  // A warp that goes through every class idles its early finishers at the end
  // of each, waiting for its longest pair (200,000 nucleotide reads, 11
  // classes: 19-22 of 32 lanes with a pair on average), and warps of one
  // multiprocessor in different classes evict each other's column loops from
  // the instruction caches (1,000,003 proteins: 9.7 -> 16.9 ms with the classes
  // dealt to warps).  By multiprocessor, against every warp from the widest
  // class on: nucleotide reads at 95 3.24 -> 3.10 ms, reads with N at 85 3.90
  // -> 3.48, 2 million protein pairs at 90 8.47 -> 7.83, proteins at 50 9.4 ->
  // 9.6.
  constexpr int n = window_classes(K, T);
  uint64_t share[n], total = 0;
#pragma unroll
  for (int k = 0; k < n; ++k) {
    const WindowClass w = window_class(T, k);
    total += share[k] = (uint64_t)(a.bounds[w.cls + 1] - a.bounds[w.cls]) *
                         (uint32_t)(w.words * w.words);
  }
  uint32_t sm, sms;
  asm("mov.u32 %0, %%smid;" : "=r"(sm));
  asm("mov.u32 %0, %%nsmid;" : "=r"(sms));
  const uint64_t at = total * sm / sms;
  int first = 0;
  uint64_t before = 0;
#pragma unroll
  for (int k = 0; k < n; ++k) {
    if (share[k] && at >= before) first = k;
    before += share[k];
  }
  uint32_t done = window_run<K, T, true>(a, first, col);
  done += window_run<K, T, false>(a, first, col);
  count_work(done, a.work);
}

template <typename F>
static int launch_round(F func, int threads, size_t smem, uint32_t want, const RoundArgs &a,
                        cudaStream_t s) {
  uint32_t grid = 0;
  NGIA_TRY(persistent_grid(reinterpret_cast<const void *>(func), threads, smem, want, &grid));
  func<<<grid, threads, smem, s>>>(a);
  NGIA_LAUNCHED();
  return NGIA_OK;
}

template <int K>
int launch_align_k(int kernel, const RoundArgs &a, uint32_t m, cudaStream_t s) {
  constexpr int KC = K <= 8 ? 8 : 16;
  // no more warps than the pairs could occupy if all were of one class
  const uint32_t lanes = ceil_div(m, 32u), warps = ceil_div(m, (uint32_t)kGroupThreads / 32u);
  constexpr auto slots = [](int tier) { return (size_t)K * window_slots(K, tier) * 32 * 4; };
  switch (kernel) {
    case 0:
      return launch_round(align_wide_kernel<KC>, 32, (size_t)KC * 16 * 32 * 4, m, a, s);
    case 2:
      return launch_round(align_group_kernel<KC>, kGroupThreads, group_smem_bytes(6, KC), warps,
                          a, s);
    case 1: return launch_round(align_window_kernel<K, 2>, 32, slots(2), lanes, a, s);
    case 3: return launch_round(align_window_kernel<K, 4>, 32, slots(4), lanes, a, s);
    case 4: return launch_round(align_window_kernel<K, 3>, 32, slots(3), lanes, a, s);
    case 5: return launch_round(align_window_kernel<K, 1>, 32, slots(1), lanes, a, s);
    case 6: return launch_round(align_window_kernel<K, 0>, 32, slots(0), lanes, a, s);
    default: return NGIA_ERR_ARG;
  }
}

}  // namespace ngia
