"""Graph emission on both sides of the hits that one block sorts (4,096), with
more pairs than that: the edges are the pairs that score, by (rep, tar)."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng

pytestmark = pytest.mark.gpu

N = 9_000


@pytest.mark.parametrize("hits", [0, 1, 4_095, 4_096, 4_097, N - 2])
def test_edges_at_the_limit(cuda, built, hits):
    from gpu_util import build_db
    kinds = [b"ACDEFGHIKL" * 4, b"MNPQRSTVWY" * 4]  # no residue in common
    packed, offs, lens = build_db([kinds[i & 1] for i in range(N)])
    # band 0 names for `hits` records one of the same kind, else one of the other
    tar = np.arange(N, dtype=np.uint32)
    rng = np.random.default_rng(5)
    same = np.zeros(N, bool)
    same[2 + rng.permutation(N - 2)[:hits]] = True
    rep = np.where(same, tar - 2, tar - 1)
    rep[0] = 0
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens, rep.astype(np.uint32), bands=1)
        for _ in range(2):
            edges, st = ctx.graph(90, 1)
            assert st["unique_pairs"] == N - 1 and st["edges"] == hits
            want = np.flatnonzero(same)
            assert np.array_equal(edges["rep"], want - 2) and np.array_equal(edges["tar"], want)
            assert (edges["weight"] == 1.0).all()


def test_load_refuses_missing_rep_rows(cuda, built):
    """Fewer rep rows than bands: refused before the copy reads past them."""
    from gpu_util import build_db
    packed, offs, lens = build_db([b"ACDEFGHIKL"] * 3)
    with ng.Context() as ctx:
        with pytest.raises(ValueError):
            ctx.load(packed, offs, lens, np.zeros((1, 3), np.uint32))
        ctx.load(packed, offs, lens, np.zeros((1, 3), np.uint32), bands=1)
