"""The lane-per-halo count (csrc/lane_count.cu) against the oracle where its
paths change: batches of 32, boxes of up to and beyond 5 x 5 rows, halos with
more candidates than a lane walks, many periodic images, a full item list,
distances in the zone below the largest radius, values that are not finite.
Counts are integers and must be equal."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu


def _count(ctx, files, h, r2, periodic=True, hint=0.0, grid=None, sched=nat.SCHED_AUTO, kind=nat.INDEX_GRID, level=0):
    q = ctx.query(h, r2, periodic=periodic)
    q.set_schedule(sched)
    idx = [ctx.build_index(f, radius_hint=hint, grid=grid, kind=kind, level=level) for f in files]
    q.count_many(idx)
    out = q.read_counts()
    for i in idx:
        i.destroy()
    q.destroy()
    return out


def _want(files, h, r2, periodic=True):
    return sum(oracle.count(f, h, r2, periodic=periodic) for f in files)


def _uniform(seed, n):
    return np.random.default_rng(seed).uniform(0, 1000, (n, 3)).astype(np.float32)


@pytest.mark.parametrize("m", [1, 31, 32, 33, 515, 4770])
@pytest.mark.parametrize("periodic", [True, False])
def test_batch_edges(ctx, m, periodic):
    files = [_uniform(900 + f, 60000) for f in range(2)]
    h = _uniform(910 + m, m)
    h[: min(m, 8)] = np.array(np.meshgrid([0.5, 999.0], [3.0, 998.0], [1.0, 996.0])).reshape(3, -1).T[: min(m, 8)]
    r2 = nat.radius_table(0.01, 18.0, 23)
    assert np.array_equal(_count(ctx, files, h, r2, periodic, 18.0), _want(files, h, r2, periodic))


@pytest.mark.parametrize("grid", [(400, 160, 160), (37, 41, 43), (1, 1, 1), (1000, 7, 300)])
@pytest.mark.parametrize("shells", [1, 40, 127])
def test_rows_of_any_grid(ctx, grid, shells):
    """Boxes of fewer and of more than 25 rows, cells of every shape."""
    p, h = _uniform(920, 30000), _uniform(921, 700)
    r2 = nat.radius_table(0.5, 20.0, shells) if shells > 1 else np.array([400.0], np.float32)
    assert np.array_equal(_count(ctx, [p], h, r2, grid=grid), _want([p], h, r2))


@pytest.mark.parametrize("sched", [nat.SCHED_STATIC, nat.SCHED_QUEUE])
@pytest.mark.parametrize("grid", [None, (100, 40, 40)])
def test_heavy_halos(ctx, sched, grid):
    """Halos in a dense clump beside light ones: lanes whose rows are listed,
    rows of more than 65535 candidates and items that are split."""
    rng = np.random.default_rng(930)
    clump = (np.array([500.0, 3.0, 997.0]) + rng.normal(0, 1.5, (150000, 3))) % 1000.0
    p = np.concatenate([clump, rng.uniform(0, 1000, (20000, 3))]).astype(np.float32)
    at = (np.array([500.0, 3.0, 997.0]) + rng.normal(0, 2.0, (40, 3))) % 1000.0
    h = np.concatenate([at, rng.uniform(0, 1000, (300, 3))]).astype(np.float32)
    r2 = nat.radius_table(0.01, 12.0, 40)
    assert np.array_equal(_count(ctx, [p], h, r2, hint=12.0, grid=grid, sched=sched), _want([p], h, r2))


def test_many_images_and_a_full_list(ctx):
    """Every halo in a corner (seven shifted images each); with fine cells all
    images are listed, more than the list holds."""
    rng = np.random.default_rng(940)
    p = (rng.normal(0, 40, (4000, 3)) % 1000.0).astype(np.float32)
    h = (rng.normal(0, 6, (4000, 3)) % 1000.0).astype(np.float32)
    r2 = nat.radius_table(0.5, 30.0, 20)
    want = _want([p], h, r2)
    for grid in [(50, 20, 20), (100, 100, 100)]:
        assert np.array_equal(_count(ctx, [p], h, r2, grid=grid), want)


@pytest.mark.parametrize("radius", [0.08, 5.0, 600.0])
def test_distances_around_the_largest_radius(ctx, radius):
    """Particles within a few ulps of the sphere and of the box faces, where
    the box test decides."""
    rng = np.random.default_rng(950)
    h = rng.uniform(0, 1000, (40, 3)).astype(np.float32)
    r2 = nat.radius_table(radius / 50, radius, 12)
    rr = np.float32(np.sqrt(np.float64(r2[-1])))
    pts = []
    for c in h:
        for a in range(3):
            for sgn in (-1, 1):
                v = c.copy()
                v[a] = np.float32(c[a] + np.float32(sgn) * rr)
                for _ in range(3):
                    pts.append(v.copy())
                    v[a] = np.nextafter(v[a], c[a])
        d = rng.normal(size=(60, 3))
        d *= (float(rr) * (1 + rng.uniform(-3e-6, 1e-6, (60, 1)))) / np.linalg.norm(d, axis=1, keepdims=True)
        pts += list((c + d).astype(np.float32))
    p = np.array(pts, np.float32)
    for periodic in (True, False):
        assert np.array_equal(_count(ctx, [p], h, r2, periodic, radius), _want([p], h, r2, periodic))


def test_values_that_are_not_finite(ctx):
    p, h = _uniform(960, 20000), _uniform(961, 200)
    p[:6] = [[np.nan, 1, 1], [np.inf, 2, 2], [3, -np.inf, 3], [-np.nan, np.nan, 4], [500, 500, np.inf], [-50, 1200, 3]]
    h[:6] = [[np.nan, 5, 5], [np.inf, 5, 5], [5, 5, -np.inf], [-40, 1190, 2], [5000, 5, 5], [1e30, 1, 1]]
    r2 = nat.radius_table(0.1, 25.0, 16)
    assert np.array_equal(_count(ctx, [p], h, r2, hint=25.0), _want([p], h, r2))


def test_wide_radius_ratio_and_close_shells(ctx):
    """Tables at the edge of the slot form: radii over many octaves, shells a
    part in 1e3 apart, and one a few ulps below the largest."""
    p, h = _uniform(970, 30000), _uniform(971, 300)
    last = np.float32(400.0)
    tables = [nat.radius_table(1e-15, 20.0, 60), (np.float32(20.0) * (1 - np.arange(40)[::-1] * 1e-3)).astype(np.float32) ** 2,
              np.array([1.0, np.nextafter(last, np.float32(0)), last], np.float32), np.array([0.0, 25.0, last], np.float32)]
    for r2 in tables:
        assert np.array_equal(_count(ctx, [p], h, r2, hint=20.0), _want([p], h, r2))


@pytest.mark.parametrize("kind", [nat.INDEX_MORTON, nat.INDEX_LEARNED])
@pytest.mark.parametrize("level", [1, 3, 5, 7])
@pytest.mark.parametrize("periodic", [True, False])
def test_morton_cells(ctx, kind, level, periodic):
    """Boxes of one cell to more than 400, dense and light halos together."""
    rng = np.random.default_rng(980)
    clump = (np.array([500.0, 3.0, 997.0]) + rng.normal(0, 2.0, (60000, 3))) % 1000.0
    p = np.concatenate([clump, rng.uniform(0, 1000, (20000, 3))]).astype(np.float32)
    at = (np.array([500.0, 3.0, 997.0]) + rng.normal(0, 2.0, (40, 3))) % 1000.0
    h = np.concatenate([at, rng.uniform(0, 1000, (600, 3))]).astype(np.float32)
    r2 = nat.radius_table(0.05, 25.0, 40)
    assert np.array_equal(_count(ctx, [p], h, r2, periodic, kind=kind, level=level), _want([p], h, r2, periodic))


@pytest.mark.parametrize("kind", [nat.INDEX_MORTON, nat.INDEX_LEARNED])
def test_morton_full_list_and_odd_values(ctx, kind):
    rng = np.random.default_rng(990)
    p = (rng.normal(0, 40, (4000, 3)) % 1000.0).astype(np.float32)
    p[:4] = [[np.nan, 1, 1], [np.inf, 2, 2], [3, -np.inf, 3], [-50, 1200, 3]]
    h = (rng.normal(0, 6, (3000, 3)) % 1000.0).astype(np.float32)
    h[:5] = [[np.nan, 5, 5], [np.inf, 5, 5], [-40, 1190, 2], [5000, 5, 5], [1e30, 1, 1]]
    r2 = nat.radius_table(0.5, 30.0, 20)
    assert np.array_equal(_count(ctx, [p], h, r2, kind=kind, level=6), _want([p], h, r2))


@pytest.mark.parametrize("kind,grid", [(nat.INDEX_GRID, (50, 20, 20)), (nat.INDEX_GRID, (100, 100, 100)),
                                       (nat.INDEX_MORTON, None), (nat.INDEX_LEARNED, None)])
@pytest.mark.parametrize("files,odd", [(1, 0), (3, 1)])
def test_more_items_than_the_list_holds(ctx, kind, grid, files, odd):
    """270000 halos in a corner, eight images each: with 1.5 items of room per
    halo most images are left to the count after the list.  Halos and particles
    outside the box among them (their images take the literal test)."""
    rng = np.random.default_rng(995)
    ps = [(rng.normal(0, 30, (900 + 7 * f, 3)) % 1000.0).astype(np.float32) for f in range(files)]
    h = (rng.normal(0, 6, (270000 + odd, 3)) % 1000.0).astype(np.float32)
    h[:400] = rng.normal(2100, 20, (400, 3)).astype(np.float32)
    ps[0][:100] = rng.normal(1100, 20, (100, 3)).astype(np.float32)
    r2 = nat.radius_table(0.5, 30.0, 9)
    level = 0 if grid else 7
    assert np.array_equal(_count(ctx, ps, h, r2, grid=grid, kind=kind, level=level), _want(ps, h, r2))
