"""Dense cells just outside a halo's box (csrc/lane_count.cu).  The lanes read a
quad of Morton cells from its first cell inside the box to its last, which can
take in a cell outside the box; what a lane may walk is decided on all it would
read, also when such a cell alone holds more than 16 bits' worth of particles.
Counts are integers and must equal the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu

LEVEL, RADIUS, CELL = 5, 40.0, 31.25


# The dense cell beside boxes that begin at an odd x (their quads hold cells 1
# and 3, and 2 lies between them) and beside boxes that end at an even x (0 and
# 2, and 1 lies between them).
@pytest.mark.parametrize("kind", [nat.INDEX_MORTON, nat.INDEX_LEARNED])
@pytest.mark.parametrize("dense", [(14, 15, 15), (15, 14, 15)])
@pytest.mark.parametrize("many", [65535, 65536, 70000, 131072])
def test_dense_cell_outside_the_box(ctx, kind, dense, many):
    rng = np.random.default_rng(1400)
    corner = np.array(dense) * CELL
    block = corner + rng.uniform(0.05, 0.95, (many, 3)) * CELL
    p = np.concatenate([block, rng.uniform(0, 1000, (20000, 3))]).astype(np.float32)
    # around the dense cell, where most warps hold a lane with more than 25
    # quads; more than five batches of 32 per SM, so that lanes walk
    h = rng.uniform(corner - 80, corner + 110, (25000, 3)).astype(np.float32)
    r2 = nat.radius_table(0.5, RADIUS, 12)
    idx = ctx.build_index(p, radius_hint=RADIUS, kind=kind, level=LEVEL)
    q = ctx.query(h, r2)
    q.count(idx)
    out = q.read_counts()
    idx.destroy()
    q.destroy()
    assert np.array_equal(out, oracle.count(p, h, r2))
