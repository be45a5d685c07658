"""Fast mode in runs of bands (pairs.cu, ctx_fast_cluster): at band counts on
both sides of each run's end the clusters equal the oracle's band-by-band
assignment."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
import oracle
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,identity", [("protein", 60), ("close", 90), ("dna", 88)])
def test_fast_runs_of_bands_match_oracle(cuda, built, kind, identity):
    from gpu_util import build_db
    if kind == "dna":
        s = synth.dna_families(700, 70, seed=21)
    elif kind == "close":  # families of fifty near copies
        s = synth.families(800, 16, synth.AMINO, synth.AMINO_FREQ,
                           synth._lognormal_roots(200, 0.5, 40, 900), 0.0, 0.05, 0.005, 2.0, 22)
    else:
        s = synth.protein_families(900, 90, seed=23)
    order = np.argsort(-s.lens, kind="stable")
    packed, offs, lens = build_db([s.seq(int(i)) for i in order])
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        ctx.sketch_bucket(64)
        rep = ctx.rep_rows(64)
        merged = 0
        for bands in (1, 3, 4, 5, 15, 16, 17, 63, 64):
            got = ctx.fast_cluster(identity, bands)
            want = oracle.fast_cluster(packed, offs, rep, identity, bands)
            assert np.array_equal(got, want), bands
            merged += int((want != np.arange(len(want))).sum())
    assert merged > 0
