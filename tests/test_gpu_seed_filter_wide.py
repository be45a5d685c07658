"""The seed filter's form for large alphabets (four residue codes a word), which
rounds of fewer than 65,536 such pairs do not run: rounds above that, of pairs
around the identity cut, against the oracle, and a check that the filter ran on
the same kinds of pairs -- targets marked whole, shared and single, and a window
at a time."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
import oracle
from ngia2_gb300 import synth
from test_gpu_seed_filter import relatives

pytestmark = pytest.mark.gpu

ROUND = 70_000  # pairs
AMINO = bytes(synth.AMINO)


def rounds(few, rng):
    """The pairs often enough for a round, grouped by target and shuffled."""
    pick = np.repeat(np.arange(len(few)), -(-ROUND // len(few)))
    return pick, rng.permutation(pick)


@pytest.mark.parametrize("identity", [76, 85, 95, 99])
def test_filtered_protein_rounds_match_oracle(cuda, built, identity):
    from gpu_util import build_db
    lengths = [7, 8, 33, 200, 512, 1_000, 1_777, 3_000, 4_500]
    seqs = relatives(AMINO, lengths, 12, 51) + relatives(AMINO, [9_001, 16_000], 5, 52)
    seqs.sort(key=len, reverse=True)
    packed, offs, lens = build_db(seqs)
    rep, tar = np.triu_indices(len(seqs), 1)
    near = lens[tar] >= 0.6 * lens[rep]
    few = np.stack([rep[near], tar[near]], 1).astype(np.uint32)
    few = few[np.argsort(few[:, 1], kind="stable")]
    want = oracle.align_pairs(packed, offs, few, identity, oracle.ROUND_FMA)
    assert (want > 0).any() and (want == 0).any()
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        for order in rounds(few, np.random.default_rng(53)):
            got, _ = ctx.align_pairs(few[order], identity)
            bad = np.flatnonzero(got != want[order])
            assert len(bad) == 0, [(int(lens[few[order[i], 0]]), int(lens[few[order[i], 1]]),
                                    int(got[i]), int(want[order[i]])) for i in bad[:8]]


@pytest.mark.parametrize("length,count,shuffled", [(1_000, 60, False), (12_000, 12, False),
                                                   (12_000, 12, True)])
def test_filter_drops_unrelated_proteins(cuda, built, length, count, shuffled):
    """75 is below the least identity that the filter serves here; at 95 the
    same unrelated pairs leave the round before they are aligned.  (Short
    proteins in random order do not: by the filter's rule marking a target of
    1,000 for one pair, 723 instructions, costs more than the 101 of aligning
    it to its exit.)"""
    from gpu_util import build_db
    rng = np.random.default_rng(length)
    letters = np.frombuffer(AMINO, np.uint8)
    seqs = sorted((letters[rng.integers(0, len(letters), int(k))].tobytes()
                   for k in rng.integers(int(length * 0.97), length, count)),
                  key=len, reverse=True)
    packed, offs, lens = build_db(seqs)
    rep, tar = np.triu_indices(count, 1)
    few = np.stack([rep, tar], 1).astype(np.uint32)
    few = few[np.argsort(few[:, 1], kind="stable")]
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        order = rounds(few, rng)[shuffled]
        got, st = ctx.align_pairs(few[order], 95)
        _, low = ctx.align_pairs(few[order], 75)
    assert not got.any() and low["computed_cells"] > 0
    assert st["computed_cells"] < low["computed_cells"] // 100
