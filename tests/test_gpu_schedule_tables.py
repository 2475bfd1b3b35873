"""Schedules on radius tables that the lane-per-halo count does not take (129 to
300 increasing shells; a repeated edge): the work queue for every kind of index, the
static kernel over several files.  Counts are integers and must equal the
oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import _native as nat
from test_gpu_schedule import QUEUES

pytestmark = pytest.mark.gpu

KINDS = [nat.INDEX_GRID, nat.INDEX_MORTON, nat.INDEX_LEARNED]


def _table(name):
    if name == "repeated":
        r2 = nat.radius_table(0.01, 15.0, 40)
        r2[20] = r2[19]
        return r2
    return nat.radius_table(0.01, 15.0, int(name))


@pytest.fixture(scope="module")
def data():
    p = nat.gen_clustered_particles(41, 120000)
    h = nat.gen_clustered_halos(42, 2500)
    h["point"][:30] = np.random.default_rng(43).choice([0.0, 1000.0, 2.0, 998.0], size=(30, 3))
    want = {(t, per): oracle.count(p, h, _table(t), periodic=per)
            for t in ("129", "300", "repeated") for per in (True, False)}
    return p, h, want


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("qs", QUEUES)
@pytest.mark.parametrize("table", ["129", "300", "repeated"])
def test_queue(ctx, data, kind, qs, table):
    p, h, want = data
    idx = ctx.build_index(p, radius_hint=15.0, kind=kind)
    for per in (True, False):
        q = ctx.query(h, _table(table), periodic=per)
        q.set_schedule(nat.SCHED_QUEUE, **qs)
        q.count(idx)
        assert np.array_equal(q.read_counts(), want[table, per])
        q.destroy()
    idx.destroy()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("table", ["129", "300", "repeated"])
def test_static_over_several_files(ctx, data, kind, table):
    p, h, want = data
    files = [p[:50000], p[50000:50000], p[50000:]]
    q = ctx.query(h, _table(table))
    q.set_schedule(nat.SCHED_STATIC)
    # one grid for all files, so that they are counted in one pass
    idx = [ctx.build_index(f, radius_hint=15.0, grid=(110, 44, 44) if kind == nat.INDEX_GRID else None, kind=kind)
           for f in files]
    q.count_many(idx)
    assert np.array_equal(q.read_counts(), want[table, True])
    for o in [q] + idx:
        o.destroy()
