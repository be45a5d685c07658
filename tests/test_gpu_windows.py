"""The one-pair-per-lane classes of the batched round (align_window.cuh):
sliding windows of 4-28 row words and fixed windows of 8-24, at the edges of
their widths, for tables of 5, 8 and 16 entries.  The round's binning
(align.cuh round_class) is compiled on the host and checked to put every pair
in a class that holds it; on the GPU the scores equal the oracle's."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import ngia2_gb300 as ng
import oracle
from ngia2_gb300 import synth

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r'''
#include <cstdio>
#include "align.cuh"
using namespace ngia;
int main() {
  long bad = 0, seen[kNumRoundClasses] = {};
  ClassPlan narrow = default_plan();
  narrow.stream_max = 12;
  for (uint32_t id = 5; id <= 95; id += 5)
    for (uint32_t lr = 1; lr < 4000; lr += 1 + lr / 37)
      for (uint32_t lt = 1; lt <= 4000; lt += 1 + lt / 29)
        for (uint32_t widest = 16; widest <= kWidestWindow; widest += 12) {
          const Band b = make_band(lr, lt, identity_threshold(id), NGIA_ROUND_FMA);
          const uint32_t ws = stream_width(b);
          const int c = round_class(b, default_plan(), widest);
          const int base = width_class(b, default_plan());
          bool ok = c >= 0 && c < kNumRoundClasses && (class_sort_key(c, b) >> 3) == (uint32_t)c;
          if (c >= kFirstFixedClass)
            ok = ok && (int)b.nr <= fixed_width(c - kFirstFixedClass) &&
                 (widest > 16 || fixed_width(c - kFirstFixedClass) <= 16);
          else if (c >= kFirstWideClass)
            ok = ok && (int)ws <= wide_width(c - kFirstWideClass) &&
                 wide_width(c - kFirstWideClass) <= (int)widest;
          else ok = ok && c == base;
          ok = ok && (c == kSkipClass) == !b.pass;
          ok = ok && round_class(b, narrow, widest) == width_class(b, narrow);
          if (!ok && bad++ < 5) printf("lr %u lt %u id %u widest %u class %d\n", lr, lt, id, widest, c);
          ++seen[c];
        }
  for (int c = kFirstWideClass; c < kNumRoundClasses; ++c) bad += seen[c] == 0;
  printf("bad %ld\n", bad);
  return bad != 0;
}
'''


def test_round_classes_hold_their_pairs(tmp_path, built):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "round.cu", tmp_path / "round"
    src.write_text(PROGRAM)
    build = subprocess.run(
        [nvcc, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
         "--expt-relaxed-constexpr", "-I", str(ROOT / "ngia2_gb300" / "csrc"),
         "-I", str(ROOT / "include"), str(src), "-o", str(exe)],
        capture_output=True, text=True, timeout=600)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stdout[-2000:]


def window_pairs(alphabet: bytes, identity: int, seed: int):
    """Reps of whole, just over and just under 1-30 row words; targets are
    suffixes, prefixes and mutated copies around the identity cut, copies of a
    few hundred columns less, and unrelated sequences."""
    rng = np.random.default_rng(seed)
    letters = np.frombuffer(alphabet, np.uint8)

    def draw(n):
        return letters[rng.integers(0, len(letters), n)]

    seqs, pairs = [], []
    for words in (1, 2, 4, 7, 8, 9, 10, 12, 14, 16, 17, 18, 20, 21, 24, 25, 28, 29, 30):
        for length in (32 * words - 31, 32 * words - 1, 32 * words):
            for k in range(4):
                rep = draw(length)
                if k == 3:
                    tar = draw(max(1, int(length * rng.uniform(0.8, 1.0))))
                else:
                    keep = int(np.ceil(length * (1.0, identity / 100 * 1.03,
                                                 rng.uniform(identity / 100, 1.0))[k]))
                    keep = max(1, min(length, keep))
                    cut = 0 if rng.random() < 0.5 else length - keep
                    tar = rep[cut:cut + keep].copy()
                    flip = rng.random(len(tar)) < rng.uniform(0, 1.2) * (1 - identity / 100) / 2
                    tar[flip] = draw(int(flip.sum()))
                seqs += [rep.tobytes(), tar.tobytes()]
                pairs.append((len(seqs) - 2, len(seqs) - 1))
    pairs = np.array(pairs, np.uint32)
    return seqs, np.concatenate([pairs[rng.permutation(len(pairs))] for _ in range(6)])


@pytest.mark.gpu
@pytest.mark.parametrize("alphabet", [b"ACGT", b"ACGTN", bytes(synth.AMINO)],
                         ids=["five", "eight", "sixteen"])
@pytest.mark.parametrize("identity", [20, 50, 70, 88, 96])
def test_windows_match_oracle(cuda, built, alphabet, identity):
    from gpu_util import build_db
    seqs, pairs = window_pairs(alphabet, identity, 7000 + identity)
    packed, offs, lens = build_db(seqs)
    want = oracle.align_pairs(packed, offs, pairs, identity, oracle.ROUND_FMA)
    assert (want > 0).any() and (want == 0).any()
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        for repeat in (1, 7):  # a round of few pairs, and of more than 8,192
            many = np.tile(pairs, (repeat, 1))
            got, _ = ctx.align_pairs(many, identity)
            bad = np.flatnonzero(got != np.tile(want, repeat))
            assert len(bad) == 0, [(int(lens[many[i, 0]]), int(lens[many[i, 1]]), int(got[i]),
                                    int(want[i % len(want)])) for i in bad[:8]]
