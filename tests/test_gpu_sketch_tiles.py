"""The hashing sketch with two bands per lane (sketch_kernel in sketch.cu), which
takes databases of more than 2,432 records: record lengths around one k-mer, a
code word, a group of four positions, a row block and a tile of 256 positions,
and past it, from planes and from nibble codes, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
import oracle
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu

EDGES = [*range(0, 18), 31, 32, 33, 39, 40, 41, 255, 256, 257, *range(260, 268), 270, 271, 272,
         511, 512, 518, 519, 520, 1_030, 1_031, 1_032, 2_000]


@pytest.mark.parametrize("alphabet", [bytes(synth.AMINO), b"ACGTN"], ids=["protein", "five"])
def test_sketch_at_tile_edges_matches_oracle(cuda, built, alphabet):
    from gpu_util import build_db, dev_empty, from_dev, stream, to_dev
    rng = np.random.default_rng(len(alphabet))
    letters = np.frombuffer(alphabet, np.uint8)
    lens = np.concatenate([np.array(EDGES * 3), rng.integers(0, 40, 2_440)])
    seqs = sorted((letters[rng.integers(0, len(letters), int(k))].tobytes() for k in lens),
                  key=len, reverse=True)
    seqs[5] = alphabet[:1] * len(seqs[5])  # one residue only
    packed, offs, lens = build_db(seqs)
    n = len(lens)
    assert n > 2_432 and n % 4  # a last block that is not full
    want = oracle.sketch_all(packed, offs, lens)
    d_packed, d_offs, d_sigs = to_dev(packed), to_dev(offs), dev_empty(64 * n * 4)
    ng.sketch(d_packed.data_ptr(), d_offs.data_ptr(), n, d_sigs.data_ptr(), stream())
    assert np.array_equal(from_dev(d_sigs, np.uint32, 64 * n).reshape(64, n), want)
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        ctx.sketch_bucket(64)
        assert np.array_equal(ctx.sigs(), want)


@pytest.mark.parametrize("bands", [33, 63, 64])
def test_streamed_chunks_of_many_bands(cuda, built, bands):
    """More than 32 bands of chunks of more than 2,432 records, whose rows are
    further apart than the chunk is long."""
    from gpu_util import build_db
    s = synth.families(9_000, 900, synth.AMINO, synth.AMINO_FREQ,
                       synth._lognormal_roots(40, 0.3, 8, 90), 0.0, 0.2, 0.01, 2.0, 91)
    packed, offs, lens = build_db([s.seq(int(i)) for i in np.argsort(-s.lens, kind="stable")])
    got, st = ng.stream_graph(packed, offs, lens, 60, bands, 36 * (len(packed) // 3 + 400))
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        m, rst = ctx.group_align(60, bands)
        want = ctx.edges(m)
    assert 2 <= st["chunks"] <= 3 and len(want) > 0
    assert np.array_equal(got, want) and st["unique_pairs"] == rst["unique_pairs"]
