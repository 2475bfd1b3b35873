"""Halo order (csrc/query_prep.cu): any order gives the same counts, so these
only have to reach its forms -- the plain copy up to 4096 halos, buckets of
every width, all halos in one bucket -- and every halo must be counted once.
Counts into pageable memory at the edges of the read-back's chunks."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [4096, 4097, 70_000, 600_000])
@pytest.mark.parametrize("crowded", [False, True])
def test_every_halo_is_counted_once(ctx, m, crowded):
    rng = np.random.default_rng(m)
    h = rng.uniform(0, 1000, (m, 3)).astype(np.float32)
    if crowded:
        h = (500 + rng.uniform(0, 1, (m, 3))).astype(np.float32)
    h[-1] = [np.nan, -5, 2000]
    p = h[rng.integers(0, m - 1, 20000)]
    r2 = np.array([0.04, 0.25], np.float32)
    q = ctx.query(h, r2)
    idx = ctx.build_index(p, radius_hint=0.5)
    q.count(idx)
    got = q.read_counts()
    idx.destroy()
    q.destroy()
    assert np.array_equal(got, oracle.count(p, h, r2))


@pytest.mark.parametrize("m", [1, 262143, 262144, 262145, 2 * 8 * 262144 + 77])
def test_read_back_chunks(ctx, m):
    """One shell per halo, so m counts: 2^18 of them fill a slot."""
    rng = np.random.default_rng(7)
    h = rng.uniform(0, 1000, (m, 3)).astype(np.float32)
    p = rng.uniform(0, 1000, (300, 3)).astype(np.float32)
    r2 = np.array([900.0], np.float32)
    q = ctx.query(h, r2)
    idx = ctx.build_index(p, radius_hint=30.0)
    q.count(idx)
    pinned = nat.PinnedBuffer((m, 1), np.uint64)
    q.read_counts(pinned.array)
    want = pinned.array.copy()
    assert np.array_equal(want[:2000], oracle.count(p, h[:2000], r2))
    assert np.array_equal(q.read_counts(), want)
    into = np.full((m, 1), 3, np.uint64)
    q.read_counts(into, accumulate=True)
    assert np.array_equal(into, want + 3)
    q.set_fold_limit(300)
    q.count(idx)  # folds: 64-bit values are read from here on
    assert q.folds == 1
    assert np.array_equal(q.read_counts(), 2 * want)
    idx.destroy()
    q.destroy()
    pinned.free()
