"""The autotuner on radius tables for which every schedule runs the same kernels:
one trial, the static schedule; other tables are timed schedule by schedule."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [nat.INDEX_GRID, nat.INDEX_MORTON, nat.INDEX_LEARNED])
def test_autotune_where_schedules_do_not_differ(ctx, kind):
    p, h = nat.gen_clustered_particles(41, 120000), nat.gen_clustered_halos(42, 2500)
    r2 = nat.radius_table(0.01, 15.0, 40)
    idx = ctx.build_index(p, radius_hint=15.0, kind=kind)
    q = ctx.query(h, r2)
    res = ctx.autotune(q, idx)
    assert len(res["trial_ms"]) == 6 and len(set(res["trial_ms"])) == 1 and res["trial_ms"][0] > 0
    assert res["chosen"]["mode"] == nat.SCHED_STATIC
    q.count(idx)
    assert np.array_equal(q.read_counts(), oracle.count(p, h, r2))
    q.destroy()
    q = ctx.query(h, nat.radius_table(0.01, 15.0, 129))
    assert len(set(ctx.autotune(q, idx)["trial_ms"])) > 1  # timed one by one
    q.destroy()
    idx.destroy()
