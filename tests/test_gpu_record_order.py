"""ngia_ctx_run_host on records whose offsets are not in index order, after a
database of another layout has left its words on the device: the pieced upload
meets records outside their pieces, discards the step before anything is
aligned, and the plain load gives the resident path's edges."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
from test_gpu_load_pipeline import dna, host_edges, resident_edges

pytestmark = pytest.mark.gpu


def moved(db, order):
    """The records of db in memory in the order `order`, their indices kept."""
    packed, offs, lens = db
    words = 1 + 4 * ((lens.astype(np.int64) + 31) // 32)
    out_offs = np.zeros(len(lens), np.uint64)
    out, at = np.empty(int(words.sum()), np.uint32), 0
    for i in order:
        out[at:at + words[i]] = packed[int(offs[i]):int(offs[i]) + words[i]]
        out_offs[i] = at
        at += int(words[i])
    return out, out_offs, lens


def swapped(n):
    """Two records of the first piece and of the last one trade places."""
    order = np.arange(n)
    order[[n // 100, n - 2]] = order[[n - 2, n // 100]]
    return order


def test_offsets_out_of_order(cuda, built):
    other = dna(16_000, 800, 61)  # what the device holds before
    db = dna(12_000, 1_200, 62)
    want = resident_edges(db, 90)
    assert len(want) > 0
    db = moved(db, swapped(len(db[2])))
    with ng.Context() as ctx:
        host_edges(ctx, other, 90)
        _, st = host_edges(ctx, other, 90)
        assert st["load_pipelined"] == 1
        got, st = host_edges(ctx, db, 90)
        assert st["load_pipelined"] == 0
        assert np.array_equal(got, want)


@pytest.mark.parametrize("name", ["reversed", "rotated", "random"])
def test_any_order_is_served(cuda, built, name):
    """Whatever the order: the pieces' bounds are looked up as if the offsets
    ascended, and may then not ascend themselves (random order)."""
    db = dna(12_000, 1_200, 64)
    n = len(db[2])
    want = resident_edges(db, 90)
    order = {"reversed": np.arange(n)[::-1], "rotated": np.roll(np.arange(n), n // 3),
             "random": np.random.default_rng(65).permutation(n)}[name]
    with ng.Context() as ctx:
        host_edges(ctx, dna(16_000, 800, 61), 90)
        got, _ = host_edges(ctx, moved(db, order), 90)
    assert np.array_equal(got, want)


def test_a_refused_step_leaves_the_database(cuda, built):
    """A pieced upload whose records pass its check stays loaded when the graph
    build refuses its arguments."""
    db = dna(12_000, 1_200, 63)
    want = resident_edges(db, 90)
    with ng.Context() as ctx:
        host_edges(ctx, db, 90)
        with pytest.raises(ng.NgiaError) as err:
            host_edges(ctx, db, 100)
        assert err.value.status == ng.ERR_ARG
        m, _ = ctx.group_align(90, 64)
        e = ctx.edges(m)
    assert np.array_equal(e["rep"], want[:, 0]) and np.array_equal(e["tar"], want[:, 1])
