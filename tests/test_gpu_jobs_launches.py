"""ngia_align_pairs on both sides of the job count from which the pairs wider
than its tables take a launch of their own: narrow, wide and refused pairs
mixed in every warp, against the oracle, eagerly and replayed from a capture."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import ngia2_gb300 as ng
import oracle
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 33, 15_000, 60_001])
@pytest.mark.parametrize("identity", [40, 90])
def test_jobs_of_all_widths(cuda, built, count, identity):
    from gpu_util import build_db, from_dev, to_dev
    rng = np.random.default_rng(81)
    letters = np.frombuffer(bytes(synth.AMINO), np.uint8)
    root = letters[rng.integers(0, len(letters), 9_000)]
    seqs = []
    for k in (9_000, 8_900, 1_200, 1_150, 780, 760, 300, 290, 40, 33, 32, 1, 0, 0):
        a = root[:k].copy()
        flip = rng.random(k) < 0.03
        a[flip] = letters[rng.integers(0, len(letters), int(flip.sum()))]
        seqs.append(a.tobytes())
    packed, offs, lens = build_db(seqs)
    n = len(seqs)
    few = np.array([(a, b) for a in range(n) for b in range(n)], np.uint32)
    want = oracle.align_pairs(packed, offs, few, identity, oracle.ROUND_FMA)
    l32 = lens.astype(np.float32)
    t = np.float32(identity) / np.float32(100)
    refused = l32[few[:, 1]] < l32[few[:, 0]] * t
    want[refused] = 77  # a failing length filter leaves the score word as it was
    pick = rng.integers(0, len(few), count)
    jobs = np.full((count, 3), 77, np.uint32)
    jobs[:, :2] = few[pick]
    d_packed, d_offs, d_jobs = to_dev(packed), to_dev(offs), to_dev(jobs)
    fresh = d_jobs.clone()

    def call(stream):
        ng.align_pairs(d_packed.data_ptr(), d_offs.data_ptr(), d_jobs.data_ptr(), count,
                       identity, stream.cuda_stream)

    call(torch.cuda.current_stream())
    assert np.array_equal(from_dev(d_jobs, np.uint32).reshape(-1, 3)[:, 2], want[pick])
    d_jobs.copy_(fresh)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(torch.cuda.current_stream())
    graph.replay()
    assert np.array_equal(from_dev(d_jobs, np.uint32).reshape(-1, 3)[:, 2], want[pick])
