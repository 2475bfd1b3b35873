"""A count when the device has hardly any memory left: its item list (12 bytes a
halo) is taken shorter, and what does not fit is counted without it."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import Context
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu


def test_count_with_little_memory_left(built):
    import torch
    rng = np.random.default_rng(1700)
    m = 6_000_000
    p = (rng.normal(0, 30, (300, 3)) % 1000.0).astype(np.float32)
    h = (rng.normal(0, 8, (m, 3)) % 1000.0).astype(np.float32)  # eight images each
    r2 = nat.radius_table(0.5, 30.0, 5)
    with Context(0) as ctx:
        idx = ctx.build_index(p, grid=(100, 100, 100))
        q = ctx.query(h, r2)
        idx.wait()
        ctx.sync()
        ctx.trim()
        torch.cuda.empty_cache()
        hog = []
        for size in (1 << 30, 64 << 20, 8 << 20):
            while torch.cuda.mem_get_info()[0] > size + (48 << 20):
                hog.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        try:
            q.count(idx)
            q.wait()
        finally:
            hog.clear()
            torch.cuda.empty_cache()
        got = q.read_counts()
        q.destroy()
        idx.destroy()
    part = slice(0, 200_000)
    assert np.array_equal(got[part], oracle.count(p, h[part], r2))
    # every halo's images were counted: the totals are those of a count with memory
    with Context(0) as ctx:
        idx = ctx.build_index(p, grid=(100, 100, 100))
        q = ctx.query(h, r2)
        q.count(idx)
        assert np.array_equal(got, q.read_counts())
        q.destroy()
        idx.destroy()
