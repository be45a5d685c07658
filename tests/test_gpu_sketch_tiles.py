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
