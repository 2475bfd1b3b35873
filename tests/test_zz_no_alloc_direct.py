"""sjcs_count_noalloc on both sides of the line between testing every pair and
building an index (2^24 pairs), and at the ends of the direct count's groups
of four halos and runs of 32 particles, against the oracle."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(1, 1), (31, 3), (33, 4), (2003, 97), (4096, 4096), (4096, 4097), (131072, 128),
                                 (131072, 129)])
@pytest.mark.parametrize("kind", ["periodic", "nonperiodic", "first_match", "wide"])
def test_direct_and_indexed_calls(n, m, kind):
    import torch
    rng = np.random.default_rng(1000 + n + m)
    p = rng.uniform(0, 1000, (n, 3)).astype(np.float32)
    h = rng.uniform(0, 1000, (m, 3)).astype(np.float32)
    h[: m // 2] = (p[rng.integers(0, n, m // 2)] + rng.normal(0, 6, (m // 2, 3)).astype(np.float32)) % np.float32(1000)
    h[: min(m, 6)] = rng.choice([0.0, 999.9, 3.0, 500.0], (min(m, 6), 3))
    p[0] = [np.nan, 1, 1]
    r2 = nat.radius_table(0.5, 30.0, 256 if kind == "wide" else 24)
    if kind == "first_match":
        r2[[3, 11]] = r2[[11, 3]]
    periodic = kind != "nonperiodic"
    dp, dh = torch.from_numpy(p).cuda(), torch.from_numpy(h).cuda()
    out = torch.full((m, len(r2)), 5, dtype=torch.int32, device="cuda")
    rc = nat.lib().sjcs_count_noalloc(
        ctypes.c_void_p(dp.data_ptr()), n, ctypes.c_void_p(dh.data_ptr()), 12, m, ctypes.c_void_p(r2.ctypes.data),
        len(r2), 1 if periodic else 0, ctypes.c_void_p(out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, nat.lib().sjcs_last_error()
    want = oracle.count(p, h, r2, periodic=periodic)
    assert np.array_equal(out.cpu().numpy().astype(np.uint64), want + 5)
