"""Streaming's chunk slots (stream.cu): from one chunk to more than the slots
hold, with every block populated and with the far blocks empty (where an outer
chunk is not the one that the row before it left in its slot), the edges equal
the resident path's and no chunk is loaded more often than the blocks ask for."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,identity", [("protein", 50), ("protein", 93), ("dna", 88)])
@pytest.mark.parametrize("pieces", [1, 2, 3, 4, 13])
def test_streamed_edges_for_any_number_of_chunks(cuda, built, kind, identity, pieces):
    from gpu_util import build_db
    s = (synth.dna_families(900, 90, seed=81) if kind == "dna"
         else synth.families(1_500, 150, synth.AMINO, synth.AMINO_FREQ,
                             synth._lognormal_roots(200, 0.6, 40, 1_500), 0.0, 0.2, 0.01, 2.0, 82))
    packed, offs, lens = build_db([s.seq(int(i)) for i in np.argsort(-s.lens, kind="stable")])
    words = len(packed) if pieces == 1 else len(packed) // pieces + 400
    got, st = ng.stream_graph(packed, offs, lens, identity, 16, 36 * words)
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        m, rst = ctx.group_align(identity, 16)
        want = ctx.edges(m)
    chunks = st["chunks"]
    assert (chunks == pieces) if pieces < 3 else (chunks >= 3)
    assert np.array_equal(got, want) and len(want) > 0
    assert st["unique_pairs"] == rst["unique_pairs"]
    assert st["aligned_cells"] == rst["aligned_cells"]
    assert st["chunk_loads"] <= 2 * chunks + chunks * (chunks - 1) // 2
