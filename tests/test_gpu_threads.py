"""Counts of different tables and sizes from several host threads, each with a
context of its own, and from the allocation-free call, which has none: they
launch the same kernels with different amounts of shared memory.  Counts are
integers and must equal the oracle's."""
from __future__ import annotations

import ctypes
import threading

import numpy as np
import pytest

from oracle import oracle
from spatialjoincountovershells_b200 import Context
from spatialjoincountovershells_b200 import _native as nat

pytestmark = pytest.mark.gpu


def _inputs(seed, halos):
    rng = np.random.default_rng(seed)
    return rng.uniform(0, 1000, (2000, 3)).astype(np.float32), rng.uniform(0, 1000, (halos, 3)).astype(np.float32)


def _context_worker(seed, shells, halos, calls, out):
    p, h = _inputs(seed, halos)
    r2 = nat.radius_table(0.5, 20.0, shells)
    with Context(0) as ctx:
        idx = ctx.build_index(p, radius_hint=20.0)
        q = ctx.query(h, r2)
        for _ in range(calls):
            q.count(idx)
        out[seed] = np.array_equal(q.read_counts(), calls * oracle.count(p, h, r2))
        q.destroy()
        idx.destroy()


def _noalloc_worker(seed, shells, halos, calls, out):
    import torch
    p, h = _inputs(seed, halos)
    r2 = nat.radius_table(0.5, 20.0, shells)
    dp, dh = torch.from_numpy(p).cuda(), torch.from_numpy(h).cuda()
    counts = torch.zeros(halos, shells, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    for _ in range(calls):
        rc = nat.lib().sjcs_count_noalloc(ctypes.c_void_p(dp.data_ptr()), len(p), ctypes.c_void_p(dh.data_ptr()), 12, halos,
                                          ctypes.c_void_p(r2.ctypes.data), shells, 1, ctypes.c_void_p(counts.data_ptr()),
                                          ctypes.c_void_p(s.cuda_stream))
        if rc:
            raise nat.SjcsError(rc, nat.lib().sjcs_last_error().decode())
    s.synchronize()
    out[seed] = np.array_equal(counts.cpu().numpy().astype(np.uint64), calls * oracle.count(p, h, r2))


def test_counts_from_several_threads(built):
    out, errors = {}, []

    def call(f, *args):
        try:
            f(*args, 300, out)
        except Exception as e:  # shown below: an exception in a thread fails no test by itself
            errors.append((f.__name__, args, str(e)))

    jobs = [(_context_worker, 1, 2, 40), (_context_worker, 2, 120, 80000), (_context_worker, 3, 1500, 300),
            (_context_worker, 4, 200, 3000), (_noalloc_worker, 5, 60, 20000)]
    threads = [threading.Thread(target=call, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert out == {1: True, 2: True, 3: True, 4: True, 5: True}
