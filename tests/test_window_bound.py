"""The one-pair-per-lane windows (align_window.cuh) restated, sliding and fixed:
window_start, the slide, the rows' entry and exit, the table slots with their
moves, and the exit bound -- pair after pair on one lane, so that every pair
meets the words and masks the last one left, over tables that begin with
garbage in every code but 0.  At the last block the total equals the banded LCS
(the reference's recurrence, test_exit_bound.run), and no block's bound is
below it.  Rows of the narrowest and the widest kind, and reps and targets of
one residue, are among them; an empty record never reaches the window.  No GPU."""
from __future__ import annotations

import numpy as np
import pytest

from test_exit_bound import FULL, band, mutate, run


class Lane:
    """One lane's words, table and window base (slots as in window_slots)."""

    def __init__(self, W: int, NS: int, codes: int, slide: bool, rng):
        self.W, self.NS, self.slide = W, NS, slide
        self.base = 0
        self.V = [FULL] * W
        self.tab = [[int(rng.integers(0, 1 << 32)) if c else 0 for _ in range(NS)]
                    for c in range(codes)]

    def fill(self, slot, rep, row):
        for c in range(1, len(self.tab)):
            bits = rep[32 * row:32 * row + 32] == c
            self.tab[c][slot] = sum(1 << k for k in np.flatnonzero(bits))

    def clear(self, slot):
        for c in range(1, len(self.tab)):
            self.tab[c][slot] = 0

    def advance(self):
        if self.base + self.W == self.NS:
            for s in range(self.W - 1):
                for c in range(1, len(self.tab)):
                    self.tab[c][s] = self.tab[c][self.base + 1 + s]
            self.base = 0
        else:
            self.base += 1

    def idle(self):
        if self.slide:
            self.advance()

    def columns(self, cols):
        for code in cols:
            carry = 0
            for m in range(self.W):
                t = self.V[m] & self.tab[code][self.base + m]
                s = self.V[m] + t + carry
                carry, s = s >> 32, s & FULL
                self.V[m] = s | (self.V[m] ^ t)

    def align(self, rep, tar, t):
        """(total, ub) after every column block."""
        W, lr, lt = self.W, len(rep), len(tar)
        ls, rs, nr, nc = band(lr, lt, t)
        lv = W - min(rs, nr) if self.slide else 0
        act = lcs = 0
        if self.slide:
            lcs = -32 * (lv + 1)
            self.V = [0 if m <= lv else FULL for m in range(W)]
        out = []
        for i in range(nc):
            if self.slide:
                self.advance()
                if i - lv - 1 < nr:
                    lcs += 32 - bin(self.V[0]).count("1")
                self.V = self.V[1:] + [FULL]
            j1 = min(i + rs, nr)
            slot0 = self.base + lv - i if self.slide else 0
            if ls < i <= ls + nr and (not self.slide or lv > ls):
                self.clear(slot0 + i - ls - 1)
            if not self.slide:
                self.V = [v if m < act else FULL for m, v in enumerate(self.V)]
            for row in range(act, j1):
                self.fill(slot0 + row, rep, row)
            act = max(act, j1)
            cols = [int(c) for c in tar[32 * i:32 * i + 32]]
            self.columns(cols + [0] * (32 - len(cols)))
            left = max(lt - 32 * (i + 1), 0)
            above0 = lr - (32 * (i - lv) if self.slide else 0)
            total = lcs if self.slide else 0
            ub = max(total, 0) + min(left, lr)
            for m in range(W):
                above = above0 - 32 * m
                if above > 0 if self.slide else m < j1:
                    total += 32 - bin(self.V[m]).count("1")
                    ub = max(ub, total + min(left, above))
            out.append((total, ub))
        return out


def pairs(rng, W, slide, t):
    """Pairs of every size that the window takes, the extremes first."""
    sizes = [1, 1, 2, 31, 32, 33, 32 * W, 32 * W - 31]
    for k in range(24):
        n = sizes[k] if k < len(sizes) else int(rng.integers(1, 32 * W + (600 if slide else 1)))
        a = rng.integers(1, 5, size=n)
        kind = k % 3
        if kind == 0:
            b = a.copy()
        elif kind == 1:
            b = mutate(rng, a, rng.uniform(0, 0.2), 0.02)
        else:
            b = rng.integers(1, 5, size=max(1, int(n * rng.uniform(t, 1.3))))
        if len(b) == 0:
            continue
        # either order: a caller's rep may be the shorter one
        for rep, tar in ((a, b), (b, a)):
            ls, rs, nr, _ = band(len(rep), len(tar), t)
            fits = ls + min(rs, nr) <= W if slide else nr <= W
            if fits and not np.float32(len(tar)) < np.float32(len(rep)) * np.float32(t):
                yield rep, tar


@pytest.mark.parametrize("slide", [True, False], ids=["sliding", "fixed"])
@pytest.mark.parametrize("W,NS", [(4, 12), (4, 16), (5, 12), (8, 12), (8, 16), (9, 14), (12, 18),
                                  (16, 18), (24, 27), (28, 36)])
def test_window_total_and_bound(slide, W, NS):
    rng = np.random.default_rng(W * 100 + NS + slide)
    checked = short = 0
    for t in (0.5, 0.9) if W > 12 else (0.3, 0.6, 0.9, 0.95):
        lane = Lane(W, NS, 5, slide, rng)
        for rep, tar in pairs(rng, W, slide, t):
            final = run(rep, tar, t)[0]
            blocks = lane.align(rep, tar, t)
            assert blocks[-1][0] == final, (len(rep), len(tar), t)
            assert all(ub >= final for _, ub in blocks), (len(rep), len(tar), t)
            checked += 1
            short += min(len(rep), len(tar)) == 1
            for _ in range(int(rng.integers(0, 4))):
                lane.idle()
    assert checked > 10 and short > 0
