"""Launch sizes up to the 2^32 - 1 pairs a build accepts: ceil_div does not
wrap (compiled on the host)."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r'''
#include <cstdio>
#include "common.cuh"
using namespace ngia;
int main() {
  long bad = 0;
  const uint32_t counts[] = {0u, 1u, 31u, 32u, 33u, 4096u, 0x7FFFFFFFu, 0xFFFFEFFFu, 0xFFFFF001u,
                             0xFFFFFF00u, 0xFFFFFF01u, 0xFFFFFFFEu, 0xFFFFFFFFu};
  for (uint32_t a : counts)
    for (uint32_t b : {1u, 2u, 32u, 128u, 256u, 2048u, 4096u}) {
      const uint64_t want = ((uint64_t)a + b - 1) / b;
      bad += ceil_div(a, b) != want;
    }
  bad += ceil_div<uint64_t>(~0ull, 2048) != (~0ull / 2048) + 1;
  printf("bad %ld\n", bad);
  return bad != 0;
}
'''


def test_ceil_div_does_not_wrap(tmp_path, built):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "range.cu", tmp_path / "range"
    src.write_text(PROGRAM)
    build = subprocess.run(
        [nvcc, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
         "--expt-relaxed-constexpr", "-I", str(ROOT / "ngia2_gb300" / "csrc"),
         "-I", str(ROOT / "include"), str(src), "-o", str(exe)],
        capture_output=True, text=True, timeout=600)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stdout[-2000:]
