"""The seed filter (seed_filter.cu): rounds large enough to run it, of pairs
around the identity cut, where a pair wrongly told apart would lose its score,
against the oracle -- grouped by target as a graph build's are and in random
order, targets short, long and long enough to be marked a window at a time,
identities on both sides of the least the filter serves."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
import oracle
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu


def relatives(alphabet: bytes, lengths, copies: int, seed: int):
    """Records of each length with copies at 0-30 % substitutions and a few
    indels, and blocks moved far from the diagonal; index order."""
    rng = np.random.default_rng(seed)
    letters = np.frombuffer(alphabet, np.uint8)
    seqs = []
    for length in lengths:
        root = letters[rng.integers(0, len(letters), length)]
        for k in range(copies):
            a = root.copy()
            flip = rng.random(length) < rng.uniform(0.0, 0.3) * (k > 0)
            a[flip] = letters[rng.integers(0, len(letters), int(flip.sum()))]
            if k % 3 == 1:  # an insertion and a deletion
                p, q = sorted(rng.integers(0, length, 2))
                a = np.concatenate([a[:p], letters[rng.integers(0, len(letters), 3)], a[p:q],
                                    a[q + 2:]])
            if k % 5 == 4:  # words the target holds, out of the band's reach
                a = np.roll(a, length // 3)
            seqs.append(a.tobytes())
    return sorted(seqs, key=len, reverse=True)


@pytest.mark.parametrize("alphabet,identities", [
    (b"ACGT", (87, 88, 95, 99)), (b"ACGTN", (89, 96)), (bytes(synth.AMINO), (75, 76, 85, 95))],
    ids=["five", "eight", "sixteen"])
def test_filtered_rounds_match_oracle(cuda, built, alphabet, identities):
    from gpu_util import build_db, to_dev
    lengths = [7, 8, 33, 200, 512, 1_000, 1_777, 3_000, 4_500]
    seqs = relatives(alphabet, lengths, 12, 51)
    seqs += relatives(alphabet, [9_001, 16_000], 5, 52)
    seqs.sort(key=len, reverse=True)
    packed, offs, lens = build_db(seqs)
    n = len(seqs)
    rep, tar = np.triu_indices(n, 1)
    near = lens[tar] >= 0.6 * lens[rep]
    few = np.stack([rep[near], tar[near]], 1).astype(np.uint32)
    few = few[np.argsort(few[:, 1], kind="stable")]  # grouped by target
    rng = np.random.default_rng(53)
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        for identity in identities:
            want = oracle.align_pairs(packed, offs, few, identity, oracle.ROUND_FMA)
            assert (want > 0).any() and (want == 0).any()
            # each pair often enough that the round is not a small one
            pick = np.repeat(np.arange(len(few)), -(-9_000 // len(few)))
            for order in (pick, rng.permutation(pick)):
                got, _ = ctx.align_pairs(few[order], identity)
                bad = np.flatnonzero(got != want[order])
                assert len(bad) == 0, (identity, [
                    (int(lens[few[order[i], 0]]), int(lens[few[order[i], 1]]), int(got[i]),
                     int(want[order[i]])) for i in bad[:8]])


def test_filter_tells_unrelated_pairs_apart(cuda, built):
    """The filter runs: a nucleotide graph of unrelated reads computes a small
    part of the cells that the same round computes at an identity below the
    filter's least, for the same candidates."""
    from gpu_util import build_db
    rng = np.random.default_rng(54)
    letters = np.frombuffer(b"ACGT", np.uint8)
    seqs = sorted((letters[rng.integers(0, 4, int(k))].tobytes()
                   for k in rng.integers(900, 1_100, 1_200)), key=len, reverse=True)
    packed, offs, lens = build_db(seqs)
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        ctx.sketch_bucket(64)
        _, st = ctx.build_graph(95, 64)
        _, low = ctx.build_graph(85, 64)
    assert st["unique_pairs"] > 8_192 and low["computed_cells"] > 0
    assert st["computed_cells"] < low["computed_cells"] // 20
