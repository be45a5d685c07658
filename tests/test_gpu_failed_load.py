"""A load that fails half way leaves no database: the buffers it has already
given up are not read by later calls, which report the missing database until
the next load."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import ngia2_gb300 as ng
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu


def test_no_database_after_a_refused_reservation(cuda, built):
    from gpu_util import build_db
    s = synth.protein_families(400, 40, seed=9)
    order = np.argsort(-s.lens, kind="stable")
    packed, offs, lens = build_db([s.seq(int(i)) for i in order])
    packed, offs = np.ascontiguousarray(packed, np.uint32), np.ascontiguousarray(offs, np.uint64)
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        ctx.sketch_bucket(64)
        want, _ = ctx.graph(60)
        # a region of 2^44 words: the reservation fails before anything is copied
        rc = ng.lib().ngia_ctx_load(ctx._h, packed.ctypes.data, 1 << 44, offs.ctypes.data,
                                    lens.ctypes.data, lens.size, None, 64)
        assert rc == ng.ERR_NOMEM
        edges = C.c_uint64()
        assert ng.lib().ngia_ctx_build_graph(ctx._h, 60, 64, C.byref(edges),
                                             None) == ng.ERR_STATE
        assert ng.lib().ngia_ctx_sketch_bucket(ctx._h, 64) == ng.ERR_STATE
        ctx.load(packed, offs, lens)
        ctx.sketch_bucket(64)
        got, _ = ctx.graph(60)
    assert len(want) > 0 and np.array_equal(got, want)
