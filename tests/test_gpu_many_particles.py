"""More than 2^29 particles in one index: lanes keep whole slot numbers and
lengths of their rows instead of packed ones.  The counts must equal those of
the same particles in two files, which lanes read packed."""
from __future__ import annotations

import numpy as np
import pytest

from spatialjoincountovershells_b200 import Context
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu


def test_counts_do_not_depend_on_how_rows_are_kept(built):
    import torch
    n = 2**29 + 1234
    g = torch.Generator(device="cuda").manual_seed(1800)
    p = torch.empty(n, 3, device="cuda")
    for part in p.split(1 << 27):
        part.uniform_(0, 1000, generator=g)
    p[: 3_000_000] = torch.remainder(torch.randn(3_000_000, 3, generator=g, device="cuda") * 3 + 500, 1000)  # a clump
    h = torch.rand(24_100, 3, generator=g, device="cuda") * 1000
    h[:300] = 500 + torch.randn(300, 3, generator=g, device="cuda") * 4
    h[300:600, 0] = 999.5
    r2 = nat.radius_table(0.01, 2.5, 24)
    with Context(0) as ctx:
        def count(files):
            q = ctx.query(h, r2)
            for f in files:
                idx = ctx.build_index(f, radius_hint=2.5)
                q.count(idx)
                q.wait()
                idx.destroy()
            out = q.read_counts()
            q.destroy()
            return out

        whole = count([p])
        halves = count([p[: n // 2], p[n // 2:]])
        ctx.trim()
    del p
    torch.cuda.empty_cache()
    assert whole.sum() > 20 * 24_100
    assert np.array_equal(whole, halves)
