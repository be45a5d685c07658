"""Fast mode where a run's pairs do not fit: runs halved down to one band give
the same clusters, and a band that does not fit is an out-of-memory error that
leaves the context usable.  The refusals come from the test limit, not from a
full device."""
from __future__ import annotations

import numpy as np
import pytest

import ngia2_gb300 as ng
from ngia2_gb300 import synth

pytestmark = pytest.mark.gpu


def test_shorter_runs_give_the_same_clusters(cuda, built):
    from gpu_util import build_db
    s = synth.families(2_000, 40, synth.AMINO, synth.AMINO_FREQ,
                       synth._lognormal_roots(200, 0.5, 40, 900), 0.0, 0.08, 0.005, 2.0, 24)
    order = np.argsort(-s.lens, kind="stable")
    packed, offs, lens = build_db([s.seq(int(i)) for i in order])
    n = len(lens)
    with ng.Context() as ctx:
        ctx.load(packed, offs, lens)
        ctx.sketch_bucket(64)
        want = ctx.fast_cluster(85, 64)
        assert (want != np.arange(n)).sum() > n // 2

        # a run holds 8 bytes a record and band, then 9 more a pair: refused at
        # the slots, at the pairs, and not at all
        for room in (17 * n, 20 * n, 32 * n, 96 * n, 200 * n, 2_000 * n):
            assert ng.lib().ngia_ctx_test_fast_room(ctx._h, room) == ng.OK
            assert np.array_equal(ctx.fast_cluster(85, 64), want), room // n
        for room in (8 * n - 1, 8 * n):
            assert ng.lib().ngia_ctx_test_fast_room(ctx._h, room) == ng.OK
            with pytest.raises(ng.NgiaError) as err:
                ctx.fast_cluster(85, 64)
            assert err.value.status == ng.ERR_NOMEM
        assert ng.lib().ngia_ctx_test_fast_room(ctx._h, 0) == ng.OK
        assert np.array_equal(ctx.fast_cluster(85, 64), want)
