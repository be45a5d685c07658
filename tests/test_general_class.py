"""The general class's own launch: left out of rounds whose longest read rules
the class out under the plan (general_possible in align.cuh, compiled on the
host and checked against the binning), and part of the captured round's key."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import ngia2_gb300 as ng
import oracle

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r'''
#include <cstdio>
#include "align.cuh"
using namespace ngia;
int main() {
  ClassPlan plans[5];
  for (auto &p : plans) p = default_plan();
  plans[1].stream_max = 4;
  plans[2].group_limit[7] = 0;
  for (int g = 0; g < kNumGroupClasses; ++g) plans[3].group_limit[g] = 0;
  plans[4].stream_max = 8;
  for (int g = 1; g < kNumGroupClasses; ++g) plans[4].group_limit[g] = 0;
  long bad = 0, out = 0, seen = 0;
  const uint32_t steps[] = {31, 32, 33, 767, 768, 769, 8191, 8192, 8193, 16383, 16384, 16385,
                            16416, 17000, 20000, 25000, 30000, 35000, 40000, 47000, 55000, 60000,
                            65000, 65533, 65534};
  for (const ClassPlan &p : plans)
    for (uint32_t lr : steps)
      for (uint32_t lt : steps)
        for (uint32_t id = 1; id <= 99; ++id) {
          const Band b = make_band(lr, lt, identity_threshold(id), NGIA_ROUND_FMA);
          const bool may = general_possible(p, lr > lt ? lr : lt, identity_threshold(id));
          out += !may;
          for (uint32_t widest = 16; widest <= kWidestWindow; widest += 12) {
            const int c = round_class(b, p, widest);
            seen += c == kGeneralClass;
            bad += c == kGeneralClass && !may;
          }
        }
  // the default plan leaves it out up to 16,384 residues, beyond that by the band
  bad += general_possible(plans[0], 16384, 0.3f) || !general_possible(plans[0], 16385, 0.3f);
  bad += general_possible(plans[0], 35000, 0.9f) || !general_possible(plans[0], 65534, 0.5f);
  bad += !general_possible(plans[3], 1, 0.9f) || general_possible(plans[4], 768, 0.3f);
  printf("bad %ld out %ld seen %ld\n", bad, out, seen);
  return bad != 0 || !out || !seen;
}
'''


def test_rule_never_leaves_a_general_pair_out(tmp_path, built):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "general.cu", tmp_path / "general"
    src.write_text(PROGRAM)
    build = subprocess.run(
        [nvcc, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
         "--expt-relaxed-constexpr", "-I", str(ROOT / "ngia2_gb300" / "csrc"),
         "-I", str(ROOT / "include"), str(src), "-o", str(exe)],
        capture_output=True, text=True, timeout=600)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stdout[-2000:]


@pytest.mark.gpu
def test_longer_reads_in_the_same_buffers(cuda, built):
    """A round captured for short reads is not replayed for a database with
    pairs of the general class, loaded into the same buffers."""
    from gpu_util import build_db
    rng = np.random.default_rng(71)
    letters = np.frombuffer(b"ACGT", np.uint8)

    def reads(lengths):
        root = letters[rng.integers(0, 4, max(lengths))]
        out = []
        for k in lengths:
            a = root[:k].copy()
            flip = rng.random(k) < 0.2
            a[flip] = letters[rng.integers(0, 4, int(flip.sum()))]
            out.append(a.tobytes())
        return build_db(out)

    short, long_ = reads([16_300 - 20 * k for k in range(8)]), reads([17_400, 17_000, 16_900] +
                                                                     [9_000] * 5)
    assert short[0].size >= long_[0].size
    pairs = np.array([(i, j) for i in range(8) for j in range(i, 8)], np.uint32)
    with ng.Context() as ctx:
        for packed, offs, lens in (short, long_, short):
            ctx.load(packed, offs, lens)
            got, _ = ctx.align_pairs(pairs, 30)
            want = oracle.align_pairs(packed, offs, pairs, 30, oracle.ROUND_FMA)
            assert (want > 0).any()
            assert np.array_equal(got, want)
