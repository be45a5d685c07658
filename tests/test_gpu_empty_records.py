"""Pairs with an empty record in the batched round: no residue can match, so
the score is 0 whichever of the two is empty and whatever class the pair falls
in (the rep of a pair given by its caller may be the shorter record)."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
import oracle
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu

LENGTHS = (0, 0, 1, 10, 31, 32, 33, 64, 400, 8_000)


@pytest.mark.parametrize("alphabet", [b"ACGT", b"ACGTN", bytes(synth.AMINO)],
                         ids=["five", "eight", "sixteen"])
@pytest.mark.parametrize("identity", [5, 50, 90, 99])
@pytest.mark.parametrize("stream_max", [16, 4])
def test_empty_records_score_zero(cuda, built, alphabet, identity, stream_max):
    from gpu_util import build_db
    rng = np.random.default_rng(91)
    letters = np.frombuffer(alphabet, np.uint8)
    # every letter present, so that the tables are the alphabet's
    seqs = [alphabet * 3] + [letters[rng.integers(0, len(letters), k)].tobytes()
                             for k in LENGTHS]
    packed, offs, lens = build_db(seqs)
    n = len(seqs)
    few = np.array([(a, b) for a in range(n) for b in range(n)], np.uint32)
    want = oracle.align_pairs(packed, offs, few, identity, oracle.ROUND_FMA)
    empty = (lens[few[:, 0]] == 0) | (lens[few[:, 1]] == 0)
    assert not want[empty].any() and want[~empty].any()
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        ctx.set_plan({**ctx.plan(), "stream_max": stream_max})
        for repeat in (1, 100):  # a round of few pairs, and of more than 8,192
            pick = rng.permutation(np.tile(np.arange(len(few)), repeat))
            got, _ = ctx.align_pairs(few[pick], identity)
            bad = np.flatnonzero(got != want[pick])
            assert len(bad) == 0, [(int(lens[few[i, 0]]), int(lens[few[i, 1]]), int(g),
                                    int(want[i])) for i, g in zip(pick[bad[:8]], got[bad[:8]])]
