"""Index builds whose particles crowd into few cells: groups of 4096 cells with
more records than one block takes (32768 and a 100th of all, the edge; several
groups; all in one cell; pieces of one and of four tiles), grid and Morton table, and the allocation-free call.  Counts are integers and must equal
the oracle's."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu


def _crowd(rng, data, n):
    if data == "equal":
        return np.full((n, 3), 333.25)
    if data == "cells":  # a few cells of one group, and the last cell of all
        p = 500.0 + rng.uniform(0, 2.0, (n, 3))
        p[: n // 4] = 999.99
        return p
    if data == "many groups":  # 100 of them
        k = rng.integers(0, 100, (n, 1))
        return 5.0 + np.concatenate([200.0 * (k % 5), 240.0 * (k // 5 % 4), 240.0 * (k // 20)], 1) + rng.uniform(0, 0.5, (n, 3))
    p = rng.uniform(0, 1000, (n, 3))
    p[: n // 2] = 300.0 + rng.normal(0, 2, (n // 2, 3))
    return p


@pytest.mark.parametrize("kind", [nat.INDEX_GRID, nat.INDEX_MORTON])
@pytest.mark.parametrize("data,n", [("equal", 32767), ("equal", 32768), ("equal", 33099), ("equal", 33100), ("equal", 1000003), ("cells", 400001),
                                    ("half", 300007), ("half", 3000001), ("many groups", 4000000), ("half", 4500001)])
def test_crowded_particles(ctx, kind, data, n):
    rng = np.random.default_rng(1600)
    p = _crowd(rng, data, n).astype(np.float32)
    h = p[rng.integers(0, n, 12)] + rng.normal(0, 1.5, (12, 3)).astype(np.float32)
    h = np.concatenate([h, rng.uniform(0, 1000, (20, 3)).astype(np.float32)])
    r2 = nat.radius_table(0.05, 5.0, 20)
    idx = ctx.build_index(p, radius_hint=5.0, kind=kind)
    q = ctx.query(h, r2)
    q.count(idx)
    out = q.read_counts()
    q.destroy()
    idx.destroy()
    assert np.array_equal(out, oracle.count(p, h, r2))


@pytest.mark.parametrize("data", ["equal", "cells", "half"])
def test_crowded_particles_without_allocation(data):
    import torch
    rng = np.random.default_rng(1610)
    n, m = 131072, 200
    p = _crowd(rng, data, n).astype(np.float32)
    h = (p[rng.integers(0, n, m)] + rng.normal(0, 3, (m, 3))).astype(np.float32)
    r2 = nat.radius_table(0.05, 9.0, 20)
    dp, dh = torch.from_numpy(p).cuda(), torch.from_numpy(h).cuda()
    out = torch.zeros(m, 20, dtype=torch.int32, device="cuda")
    for _ in range(2):
        rc = nat.lib().sjcs_count_noalloc(
            ctypes.c_void_p(dp.data_ptr()), n, ctypes.c_void_p(dh.data_ptr()), 12, m, ctypes.c_void_p(r2.ctypes.data), 20, 1,
            ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0, nat.lib().sjcs_last_error()
    assert np.array_equal(out.cpu().numpy().astype(np.uint64), 2 * oracle.count(p, h, r2))
