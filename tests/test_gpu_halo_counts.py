"""Counts of few halos (a warp to a halo, heavy images left to a list) and of
many (a lane to a halo) against the oracle, on either side of where one takes
over from the other and where each can go wrong: the list full, images listed
from a later part of their box on, several counts of one query (they take the
list's control words in turn), grids of every shape, Morton cells.  Counts are
integers and must be equal."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu

KINDS = [nat.INDEX_GRID, nat.INDEX_MORTON, nat.INDEX_LEARNED]


def _count(ctx, files, h, r2, periodic=True, hint=0.0, grid=None, kind=nat.INDEX_GRID, level=0, times=1):
    q = ctx.query(h, r2, periodic=periodic)
    idx = [ctx.build_index(f, radius_hint=hint, grid=grid, kind=kind, level=level) for f in files]
    for _ in range(times):
        q.count_many(idx)
    out = q.read_counts()
    for i in idx:
        i.destroy()
    q.destroy()
    return out


def _mixed(rng, n, m):
    """Half the particles and a third of the halos in a clump near a corner."""
    centre = np.array([500.0, 3.0, 997.0])
    p = np.concatenate([(centre + rng.normal(0, 4, (n // 2, 3))) % 1000.0, rng.uniform(0, 1000, (n - n // 2, 3))])
    h = np.concatenate([(centre + rng.normal(0, 5, (m // 3, 3))) % 1000.0, rng.uniform(0, 1000, (m - m // 3, 3))])
    return p.astype(np.float32), h.astype(np.float32)


# 32 halos to a batch and five batches to an SM: 23680 halos on 148 SMs
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("m", [1, 4736, 4737, 23680, 23681])
@pytest.mark.parametrize("periodic", [True, False])
def test_either_side_of_the_lines(ctx, kind, m, periodic):
    p, h = _mixed(np.random.default_rng(1500 + m), 30000, m)
    r2 = nat.radius_table(0.05, 9.0, 30)
    want = oracle.count(p, h, r2, periodic=periodic)
    assert np.array_equal(_count(ctx, [p], h, r2, periodic, 9.0, kind=kind, times=3), 3 * want)


@pytest.mark.parametrize("grid", [(400, 160, 160), (37, 41, 43), (1, 1, 1), (1000, 7, 300)])
@pytest.mark.parametrize("m", [300, 24000])
def test_rows_of_any_grid(ctx, grid, m):
    """Boxes of up to hundreds of rows: images whose later rows are the heavy ones."""
    rng = np.random.default_rng(1510)
    p, h = _mixed(rng, 24000, m)
    h[-20:] = (np.array([500.0, 21.0, 1.0]) + rng.normal(0, 1, (20, 3))).astype(np.float32)
    r2 = nat.radius_table(0.5, 20.0, 40)
    assert np.array_equal(_count(ctx, [p], h, r2, grid=grid), oracle.count(p, h, r2))


@pytest.mark.parametrize("kind", KINDS)
def test_more_heavy_images_than_the_list_takes(ctx, kind):
    """8000 halos in a corner, eight images each, nearly all of them heavy."""
    rng = np.random.default_rng(1520)
    files = [(rng.normal(0, 8, (4000, 3)) % 1000.0).astype(np.float32) for _ in range(3)]
    h = (rng.normal(0, 4, (8000, 3)) % 1000.0).astype(np.float32)
    r2 = nat.radius_table(0.5, 20.0, 20)
    want = sum(oracle.count(f, h, r2) for f in files)
    assert np.array_equal(_count(ctx, files, h, r2, hint=20.0, kind=kind, times=2), 2 * want)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,radius", [(3000, 600.0), (20000, 250.0), (60000, 60.0)])
@pytest.mark.parametrize("m", [200, 24000])
def test_large_radii(ctx, kind, n, radius, m):
    """Two to eight images of nearly every halo, boxes of most of the volume."""
    rng = np.random.default_rng(1530)
    p, h = (rng.uniform(0, 1000, (k, 3)).astype(np.float32) for k in (n, m))
    keep = max(200, int(m * min(1.0, 2e8 / (n * m))))  # what the oracle counts in a few seconds
    r2 = nat.radius_table(radius / 40, radius, 12)
    got = _count(ctx, [p], h, r2, hint=radius, kind=kind)
    assert np.array_equal(got[:keep], oracle.count(p, h[:keep], r2))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("level", [1, 3, 5, 7])
def test_many_halos_on_cells_of_any_level(ctx, kind, level):
    rng = np.random.default_rng(1540)
    p, h = _mixed(rng, 16000, 24500)
    p[:4] = [[np.nan, 1, 1], [np.inf, 2, 2], [3, -np.inf, 3], [-50, 1200, 3]]
    h[:5] = [[np.nan, 5, 5], [np.inf, 5, 5], [-40, 1190, 2], [5000, 5, 5], [1e30, 1, 1]]
    r2 = nat.radius_table(0.05, 25.0, 40)
    grid = None if kind != nat.INDEX_GRID else (2**level,) * 3
    got = _count(ctx, [p], h, r2, kind=kind, grid=grid, level=0 if grid else level)
    assert np.array_equal(got, oracle.count(p, h, r2))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("data", ["uniform", "clumps", "few clumps"])
@pytest.mark.parametrize("files", [1, 3])
@pytest.mark.parametrize("m", [3000, 24100])
def test_full_boxes(ctx, kind, data, files, m):
    """More candidates to an ordinary box than a lane walks: of many halos a
    sample tells whether lanes or warps count them (clumps around most halos, or
    around 3 % of them).  Images listed from a later part of their box on."""
    rng = np.random.default_rng(1550)
    n, radius = 40000, 120.0
    ps = [rng.uniform(0, 1000, (n, 3)) for _ in range(files)]
    h = rng.uniform(0, 1000, (m, 3))
    if data != "uniform":
        centre = rng.uniform(0, 1000, (20, 3))
        for p in ps:
            p[: n // 2] = (centre[rng.integers(0, 20, n // 2)] + rng.normal(0, 25, (n // 2, 3))) % 1000.0
        k = m if data == "clumps" else m // 32
        h[:k] = (centre[rng.integers(0, 20, k)] + rng.normal(0, 20, (k, 3))) % 1000.0
        rng.shuffle(h)
    ps, h = [p.astype(np.float32) for p in ps], h.astype(np.float32)
    r2 = nat.radius_table(2.0, radius, 14)
    got = _count(ctx, ps, h, r2, hint=radius, kind=kind)
    assert np.array_equal(got[:6000], sum(oracle.count(p, h[:6000], r2) for p in ps))
