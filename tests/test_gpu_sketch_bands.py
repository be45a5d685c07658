"""The hashing sketch's runs of bands (sketch.cu): few records split over warps,
and fewer bands than 64 -- record counts on both sides of each rule, band
counts around each run's width, against the oracle and the resident path."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
import oracle
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu


def short_proteins(n: int, seed: int):
    from gpu_util import build_db
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 60, n)  # empty, one k-mer, a few
    return build_db([synth._draw(rng, synth.AMINO, synth.AMINO_FREQ, int(k)).tobytes()
                     for k in lens])


@pytest.mark.parametrize("n", [1, 304, 305, 2432, 2433])
def test_sketch_split_over_warps_matches_oracle(cuda, built, n):
    from gpu_util import dev_empty, from_dev, stream, to_dev
    packed, offs, lens = short_proteins(n, n)
    want = oracle.sketch_all(packed, offs, lens)
    d_packed, d_offs, d_sigs = to_dev(packed), to_dev(offs), dev_empty(64 * n * 4)
    ng.sketch(d_packed.data_ptr(), d_offs.data_ptr(), n, d_sigs.data_ptr(), stream())
    assert np.array_equal(from_dev(d_sigs, np.uint32, 64 * n).reshape(64, n), want)
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        ctx.sketch_bucket(64)
        assert np.array_equal(ctx.sigs(), want)


@pytest.mark.parametrize("bands", [1, 4, 5, 8, 9, 16, 17, 32, 33, 63, 64])
def test_stream_hashes_only_its_bands(cuda, built, bands):
    from gpu_util import build_db
    s = synth.protein_families(600, 60, seed=31)
    order = np.argsort(-s.lens, kind="stable")
    packed, offs, lens = build_db([s.seq(int(i)) for i in order])
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        m, _ = ctx.group_align(50, bands)
        want = ctx.edges(m)
    got, st = ng.stream_graph(packed, offs, lens, 50, bands, packed.size * 4 * 3)
    assert st["chunks"] > 1
    assert np.array_equal(got, want)
