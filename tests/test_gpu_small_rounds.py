"""The single-launch forms for small sizes, on both sides of each limit: the
bucketing of up to 4,096 records (bucket.cu), the binning of up to 8,192 pairs
and the emission of up to 4,096 (pairs.cu)."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
import oracle
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 512, 513, 1025, 4095, 4096, 4097])
@pytest.mark.parametrize("bands", [1, 64])
def test_small_bucket_matches_grouping(cuda, built, n, bands):
    from gpu_util import dev_empty, from_dev, stream, to_dev
    rng = np.random.default_rng(n * 64 + bands)
    pool = rng.integers(0, 2**32, size=max(1, n // 4), dtype=np.uint64).astype(np.uint32)
    sigs = pool[rng.integers(0, len(pool), size=(bands, n))]
    sigs[:, rng.random(n) < 0.1] = 0xFFFFFFFF  # what an empty record signs
    sigs[0] = sigs[0, 0]  # one bucket of every record
    want = np.stack([oracle.bucket_band(s) for s in sigs])
    d_sigs, d_rep = to_dev(sigs), dev_empty(bands * n * 4)
    ng.bucket(d_sigs.data_ptr(), n, bands, d_rep.data_ptr(), stream())
    assert np.array_equal(from_dev(d_rep, np.uint32, bands * n).reshape(bands, n), want)
    ng.bucket_noalloc(d_sigs.data_ptr(), n, bands, d_rep.data_ptr(), stream())
    assert np.array_equal(from_dev(d_rep, np.uint32, bands * n).reshape(bands, n), want)


@pytest.mark.parametrize("count", [1, 8191, 8192, 8193])
def test_round_sizes_match_oracle(cuda, built, count):
    from gpu_util import build_db
    s = synth.protein_families(400, 40, seed=41)
    order = np.argsort(-s.lens, kind="stable")
    packed, offs, lens = build_db([s.seq(int(i)) for i in order])
    rng = np.random.default_rng(count)
    few = np.sort(rng.integers(0, 400, (1500, 2)), axis=1).astype(np.uint32)
    want = oracle.align_pairs(packed, offs, few, 60, oracle.ROUND_FMA)
    pick = rng.integers(0, len(few), count)
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        got, st = ctx.align_pairs(few[pick], 60)
        ctx.use_graphs(False)
        eager, st_eager = ctx.align_pairs(few[pick], 60)
    assert np.array_equal(got, want[pick]) and np.array_equal(eager, got)
    assert st["aligned_cells"] == st_eager["aligned_cells"]
    assert st["aligned_cells"] == 1024 * sum(
        oracle.band_blocks(int(lens[r]), int(lens[t]), 60) for r, t in few[pick])


@pytest.mark.parametrize("n,identity", [(60, 50), (900, 50), (2300, 40)])
def test_graphs_around_the_small_emission_match_oracle(cuda, built, n, identity):
    from gpu_util import build_db
    s = synth.protein_families(n, max(1, n // 12), seed=43)
    order = np.argsort(-s.lens, kind="stable")
    packed, offs, lens = build_db([s.seq(int(i)) for i in order])
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        m, st = ctx.group_align(identity, 64)
        edges, rep = ctx.edges(m), ctx.rep_rows(64)
    want, total = oracle.graph_edges(packed, offs, lens, rep, identity, 64)
    got = np.stack([edges["rep"], edges["tar"],
                    np.rint(edges["weight"].astype(np.float64) * 100)], axis=1).astype(np.int64)
    assert np.array_equal(got, want) and st["candidate_pairs"] == total
    assert (st["unique_pairs"] <= 4096) == (n < 2000)
