// align_jobs.cu -- the drop-in job-triple kernel: the reference's
// one-launch-per-band kernel_dynamic<<<ceil(count/64), 64>>> (launch at
// src/buildGraph.hpp:323), on the packed records alone and without scratch.
//
// A warp takes 32 jobs in job order, one pair per lane, in the windows of the
// batched aligner (align_window.cuh): the lanes whose pairs fit 4, 8, 12, 16
// and 24 words (the whole rep, or the sliding band) run together, the rest
// through the general form.  Many jobs take a launch each for narrow, medium and
// wide pairs.  Match masks come from tables in shared memory, as there; the
// target's codes are made from its bit planes, block by block.
//
// What bounds it at the reference's launch sizes (a band's few thousand jobs):
// the longest pair of a warp, a serial chain of 32 columns a block.  With the
// masks computed from the bit planes in every column, 12 ALU operations a word
// instead of 3, 6,000 jobs of 20,000 proteins at identity 90 took 107 us, with
// the tables 75 us.
#include <algorithm>

#include "align_window.cuh"
#include "kernels.cuh"

namespace ngia {

constexpr uint32_t kJobWords = 24;  // the widest window
constexpr int kJobSlots = 27;       // table slots: room for it to slide
constexpr int kNarrowSlots = 9;     // the same for 8 words

// The lanes of the warp with `run` align their pairs; returns the score.
template <int NS, int W, bool kSlide>
__device__ __forceinline__ void job_window(bool run, const uint32_t *rep, const uint32_t *tar,
                                           const Band &b, uint32_t *col, uint32_t &score) {
  if (!__any_sync(kFull, run)) return;
  const LdsTable<NS, 16> tab{col};
  uint32_t V[W];
#pragma unroll
  for (int m = 0; m < W; ++m) V[m] = kFull;
  WindowPair sp{};
  if (run) {
    sp.rep = rep;
    sp.tar = tar + 1;
    sp.lr = b.lr;
    sp.lt = b.lt;
    sp.nc = b.nc;
    sp.nr = b.nr;
    sp.rs = b.rs;
    sp.ls = b.ls;
    sp.pf_row = kFull;
    sp.cur = load4(sp.tar);
    sp.active = true;
    if constexpr (kSlide) window_start(V, sp);
  }
  uint32_t base = 0;
  while (__any_sync(kFull, sp.active)) {
    if constexpr (kSlide) window_advance<W>(tab, base);
    int32_t total = 0, ub = 0;
    window_block<W, NS, 16, kSlide, true>(V, sp, tab, base, total, ub);
    if (sp.active) {
      const bool last = sp.i >= sp.nc;
      if (last || !lcs_may_reach((uint32_t)ub, sp.lr, sp.lt, b.t)) {
        score = last ? identity_score((uint32_t)total, sp.lr, sp.lt, b.t) : 0u;
        sp.active = false;
      }
    }
  }
}

// A job, and how it is aligned.
struct Job {
  const uint32_t *rep, *tar;
  Band b;
  bool mine, empty;  // to be scored; no columns
  bool fixed;        // the whole rep is narrower than the sliding window
  uint32_t words;    // of the narrower of the two (0: nothing to align)
};

__device__ __forceinline__ Job load_job(const uint32_t *packed, const uint64_t *offs,
                                        const uint32_t *jobs, uint32_t j, uint32_t count,
                                        float t, int fma_mode) {
  Job w{packed, packed, {}, false, true, false, 0u};
  if (j >= count) return w;
  w.rep = packed + offs[jobs[3 * (size_t)j]];
  w.tar = packed + offs[jobs[3 * (size_t)j + 1]];
  w.b = make_band(__ldg(w.rep), __ldg(w.tar), t, fma_mode);
  w.mine = w.b.pass;  // else the reference leaves the score word as it was
  w.empty = w.b.nc == 0;
  const uint32_t ws = stream_width(w.b);
  w.fixed = w.b.nr < ws;
  w.words = w.mine && !w.empty ? (w.fixed ? w.b.nr : ws) : 0u;
  return w;
}

// In the general form, for any width.
__device__ __forceinline__ uint32_t job_general(const Job &w, float t) {
  uint32_t lines[kMaxRowBlocks];
  uint32_t blocks;
  return identity_score(lcs_general(w.rep, w.tar, w.b, lines, blocks), w.b.lr, w.b.lt, t);
}

// Jobs by the width of their windows: up to 8 words, 9-24, more (general form).
constexpr int kNarrow = 1, kMid = 2, kWide = 4;

// The jobs of the widths in kSet.
template <int NS, int kSet>
__global__ void __launch_bounds__(32)
align_jobs_kernel(const uint32_t *__restrict__ packed, const uint64_t *__restrict__ offs,
                  uint32_t *__restrict__ jobs, uint32_t count, float t, int fma_mode) {
  extern __shared__ uint32_t smem[];
  const uint32_t j = blockIdx.x * 32u + threadIdx.x;
  const Job w = load_job(packed, offs, jobs, j, count, t, fma_mode);
  const uint32_t *rep = w.rep, *tar = w.tar, words = w.words;
  const Band &b = w.b;
  const bool fixed = w.fixed;
  const int kind = words <= 8 ? kNarrow : words <= kJobWords ? kMid : kWide;
  const bool mine = w.mine && (kind & kSet);
  if (!__any_sync(kFull, mine)) return;
  [[maybe_unused]] uint32_t *col = smem + threadIdx.x;
  if constexpr (NS > 0) {
#pragma unroll 1
    for (int s = 0; s < NS; ++s) col[s * 32] = 0u;  // code 0 matches nothing
  }
  uint32_t score = 0;
  if constexpr (kSet & kNarrow) {
    job_window<NS, 4, true>(!fixed && words - 1u < 4u, rep, tar, b, col, score);
    job_window<NS, 8, true>(!fixed && words - 5u < 4u, rep, tar, b, col, score);
    job_window<NS, 8, false>(fixed && words - 1u < 8u, rep, tar, b, col, score);
  }
  if constexpr (kSet & kMid) {
    job_window<NS, 12, true>(!fixed && words - 9u < 4u, rep, tar, b, col, score);
    job_window<NS, 16, true>(!fixed && words - 13u < 4u, rep, tar, b, col, score);
    job_window<NS, 24, true>(!fixed && words - 17u < 8u, rep, tar, b, col, score);
    job_window<NS, 16, false>(fixed && words - 9u < 8u, rep, tar, b, col, score);
    job_window<NS, 24, false>(fixed && words - 17u < 8u, rep, tar, b, col, score);
  }
  if constexpr (kSet & kWide) {
    if (words > kJobWords) score = job_general(w, t);
  }
  if (mine) jobs[3 * (size_t)j + 2] = w.empty ? identity_score(0u, b.lr, b.lt, t) : score;
}

constexpr size_t job_smem(int slots) { return (size_t)slots * 16 * 32 * 4; }

int launch_align_jobs(const uint32_t *packed, const uint64_t *offs, uint32_t *jobs,
                      uint32_t count, uint32_t identity, cudaStream_t s) {
  if (count == 0) return NGIA_OK;
  const float t = identity_threshold(identity);
  const uint32_t warps = ceil_div(count, 32u);
  constexpr auto all = align_jobs_kernel<kJobSlots, kNarrow | kMid | kWide>;
  constexpr auto mid = align_jobs_kernel<kJobSlots, kMid>;
  constexpr auto narrow = align_jobs_kernel<kNarrowSlots, kNarrow>;
  uint32_t grid = 0;
  NGIA_TRY(persistent_grid(reinterpret_cast<const void *>(all), 32, job_smem(kJobSlots), warps,
                           &grid));
  if (grid == warps) {
    // as much of the L1 for the tables as these warps need and no more: what is
    // left holds the row words of pairs over kJobWords words (all for the tables,
    // so: 1,000 of 60,000 residues at identity 90 231, 213 ms; 6,000 of 1,500 at 50
    // 0.67, 0.62; 6,000 narrow ones no different)
    int dev = 0, sms = 0;
    NGIA_CUDA(cudaGetDevice(&dev));
    NGIA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const uint32_t kib = ceil_div(warps, (uint32_t)sms) * (job_smem(kJobSlots) / 1024 + 1);
    cudaLaunchAttribute split{};
    split.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    split.val.sharedMemCarveout = std::min(kib * 100 / 228 + 1, 100u);  // of 228 KB, percent
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(warps);
    cfg.blockDim = dim3(32);
    cfg.dynamicSmemBytes = job_smem(kJobSlots);
    cfg.stream = s;
    cfg.attrs = &split;
    cfg.numAttrs = 1;
    NGIA_CUDA(cudaLaunchKernelEx(&cfg, all, packed, offs, jobs, count, t, round_mode()));
    NGIA_LAUNCHED();
    return NGIA_OK;
  }
  // More jobs than fit on the device at once: the widest windows' tables leave a
  // multiprocessor four warps, so the pairs that do with less have launches with
  // smaller tables (eleven warps) and with none (twenty), which cost the others a
  // pass over their jobs.  In one launch, in two (the pairs over kJobWords words
  // apart), in three, and with masks from the bit planes throughout:
  // 1,000,000 of 300 residues at identity 90 244, 258, 201, 205 us; 200,000 65, 71,
  // 66, 60; 200,000 of 400 at 50 253, 271, 281, 439; 100,000 of 3,000 at 90 533, 549,
  // 555, 1,076; 100,000 of 1,500 at 50 3.56, 2.69, 2.64, 2.54 ms; 2 million
  // heavy-tailed pairs at 90 in 64 calls 3,655, 3,545, 3,498, 3,416.
  NGIA_TRY(persistent_grid(reinterpret_cast<const void *>(narrow), 32, job_smem(kNarrowSlots),
                           warps, &grid));  // (sets its shared memory)
  narrow<<<warps, 32, job_smem(kNarrowSlots), s>>>(packed, offs, jobs, count, t, round_mode());
  NGIA_LAUNCHED();
  NGIA_TRY(persistent_grid(reinterpret_cast<const void *>(mid), 32, job_smem(kJobSlots), warps,
                           &grid));
  mid<<<warps, 32, job_smem(kJobSlots), s>>>(packed, offs, jobs, count, t, round_mode());
  NGIA_LAUNCHED();
  // (no wish for shared memory: the row words of the general form live in L1;
  // with it 100,000 of 1,500 residues take 3.66 ms)
  align_jobs_kernel<0, kWide><<<warps, 32, 0, s>>>(packed, offs, jobs, count, t, round_mode());
  NGIA_LAUNCHED();
  return NGIA_OK;
}

}  // namespace ngia

extern "C" int ngia_align_pairs(const uint32_t *d_packed, const uint64_t *d_rec_offsets,
                                uint32_t *d_jobs, uint32_t count, uint32_t identity,
                                void *stream) {
  if (identity < 1 || identity > 99) return NGIA_ERR_ARG;
  if (count == 0) return NGIA_OK;
  if (!d_packed || !d_rec_offsets || !d_jobs) return NGIA_ERR_ARG;
  return ngia::launch_align_jobs(d_packed, d_rec_offsets, d_jobs, count, identity,
                                 ngia::as_stream(stream));
}
