"""Morton cells fetched four at a time (csrc/lane_count.cu) against the oracle:
boxes that begin and end in either half of a quad, quads of which the sphere
leaves out one cell, ranges whose end lies past the last particle, cells of
many equal particles.  4770 halos, so that lanes walk; 300, so that all are
listed.  Counts are integers and must be equal."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu


def _particles(data, rng):
    if data == "uniform":
        return rng.uniform(0, 1000, (40000, 3))
    if data == "few":
        return rng.uniform(0, 1000, (3, 3))
    if data == "last":  # only the last cell, up to the largest coordinate
        return np.concatenate([rng.uniform(970, 1000, (3000, 3)), np.full((2, 3), 999.99994), np.full((1, 3), 1000.0)])
    p = rng.uniform(0, 1000, (5000, 3))  # equal keys among others
    p[100:3100] = [333.25, 666.5, 10.0]
    return p


@pytest.mark.parametrize("kind", [nat.INDEX_MORTON, nat.INDEX_LEARNED])
@pytest.mark.parametrize("data", ["uniform", "few", "last", "equal"])
@pytest.mark.parametrize("level,radius", [(1, 40.0), (4, 70.0), (5, 40.0), (6, 60.0)])
@pytest.mark.parametrize("halos,periodic", [(4770, True), (4770, False), (300, True)])
def test_quads(ctx, kind, data, level, radius, halos, periodic):
    rng = np.random.default_rng(1200 + level)
    p = _particles(data, rng).astype(np.float32)
    h = rng.uniform(0, 1000, (halos, 3)).astype(np.float32)
    # centres a radius from cell faces, so that boxes end at them
    cell = 1000.0 / 2**level
    near = np.round(rng.uniform(0, 1000, (halos // 4, 3)) / cell) * cell
    h[: halos // 4] = np.clip(near + rng.choice([-radius, radius], (halos // 4, 3)), 0, 1000).astype(np.float32)
    h[-40:] = p[rng.integers(0, len(p), 40)]
    r2 = nat.radius_table(0.5, radius, 20)
    q = ctx.query(h, r2, periodic=periodic)
    idx = ctx.build_index(p, radius_hint=radius, kind=kind, level=level)
    q.count(idx)
    out = q.read_counts()
    idx.destroy()
    q.destroy()
    assert np.array_equal(out, oracle.count(p, h, r2, periodic=periodic))


@pytest.mark.parametrize("kind,per_cell", [(nat.INDEX_MORTON, 1.0), (nat.INDEX_LEARNED, 2.4)])
@pytest.mark.parametrize("hint,below", [(5.0, 4), (40.0, 4), (60.0, 4), (0.0, 4)])
def test_automatic_level(ctx, kind, per_cell, hint, below):
    """The cells halve where the particles per cell allow it: one more or less
    particle than that, radii that allow the finer cells (40) and that do not
    (60: 0.7 R is more than 31.25), and no radius (four per cell)."""
    want = per_cell if hint else 4.0
    fine = below if hint == 60.0 else below + 1
    edge = int(np.ceil(8 ** (below + 1) * want))
    rng = np.random.default_rng(1300)
    h = rng.uniform(0, 1000, (300, 3)).astype(np.float32)
    r2 = nat.radius_table(0.5, hint or 25.0, 12)
    for n, level in ((edge - 1, below), (edge, fine)):
        p = rng.uniform(0, 1000, (n, 3)).astype(np.float32)
        idx = ctx.build_index(p, radius_hint=hint, kind=kind)
        q = ctx.query(h, r2)
        q.count(idx)
        out, got = q.read_counts(), idx.grid
        idx.destroy()
        q.destroy()
        assert tuple(got) == (2**level,) * 3
        assert np.array_equal(out, oracle.count(p, h, r2))
