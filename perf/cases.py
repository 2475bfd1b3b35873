"""Workloads whose speed is followed from change to change.

Each case is one thing a program does with this package: a whole particle-file
job (index build, query set-up, count), a request against resident indexes,
the same job from host buffers, or the allocation-free call.  Sizes and
radius schedules are those of the benchmark, the tests and the golden cases,
and sizes between them; inputs have the benchmark's distributions (uniform in
the periodic box, or 60 % of the particles in 1e4 Gaussian clumps with 70 % of
the halos at clump centres), drawn on the device from the seed.  Outputs are
the integer counts per halo and shell.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import spatialjoincountovershells_b200 as sjcs
from spatialjoincountovershells_b200 import _native as nat

BOX = 1000.0
KINDS = {"grid": nat.INDEX_GRID, "morton": nat.INDEX_MORTON, "learned": nat.INDEX_LEARNED}
SCHEDULES = {"auto": nat.SCHED_AUTO, "queue": nat.SCHED_QUEUE}


def _case(call, files, particles, halos, rmin, rmax, shells, data="uniform", index="grid", schedule="auto",
          periodic=True, **more):
    return dict(call=call, files=files, particles=particles, halos=halos, rmin=rmin, rmax=rmax, shells=shells,
                data=data, index=index, schedule=schedule, periodic=periodic, **more)


def listed():
    return [
        # The smallest call: a latency-critical loop counting a few halos
        # against a small particle set without any allocation.
        _case("noalloc", 1, 2003, 97, 0.5, 25.0, 17, periodic=False, name="noalloc_small"),
        # The allocation-free call at its particle limit (the size its tests use).
        _case("noalloc", 1, 131072, 20000, 0.01, 40.0, 40, name="noalloc_limit"),
        # The serving loop's smallest request: 100 clustered halos against
        # three resident particle files.
        _case("query", 3, 10_000_000, 100, 0.001, 5.0, 40, data="clustered", name="query_100"),
        # A mid-sized request of the serving mix (sizes 1e2..1e6, r_max up to 10, up to 64 shells).
        _case("query", 3, 20_000_000, 99_991, 0.001, 10.0, 64, data="clustered", name="query_1e5"),
        # A single small snapshot, the golden uniform case: 1e6 particles x 1.05e4 halos.
        _case("job", 1, 1_000_000, 10_500, 0.001, 5.0, 40, name="job_1e6x1e4"),
        # An ordinary file at the README's particles-to-halos ratio.
        _case("job", 1, 10_000_019, 1_000_003, 0.001, 5.0, 40, name="job_1e7x1e6"),
        # The README's run, the benchmark's step: 3 files of 1e8, 1e7 halos, 40 shells.
        _case("job", 3, 100_000_000, 10_000_000, 0.001, 5.0, 40, name="job_readme"),
        # Uneven load: clustered data under the default schedule.
        _case("job", 1, 30_000_000, 1_000_000, 0.001, 5.0, 40, data="clustered", name="job_clustered_r5"),
        # Heavy uneven load: large radii on clustered data, persistent queue.
        _case("job", 1, 50_000_000, 1_000_000, 0.01, 20.0, 64, data="clustered", schedule="queue",
              name="job_clustered_r20_queue"),
        # The other index forms: plain Morton table and the learned ranks.
        _case("job", 1, 20_000_000, 500_000, 0.001, 5.0, 40, data="clustered", index="morton", name="job_morton"),
        _case("job", 1, 20_000_000, 500_000, 0.001, 5.0, 40, data="clustered", index="learned", schedule="queue",
              name="job_learned"),
        # The driver's path: particles and halos in page-locked host memory,
        # 64-bit counts read back to the host.
        _case("host", 1, 5_000_011, 200_000, 0.001, 5.0, 40, name="host_5e6x2e5"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pairs(c):
    """Particles inside R of a halo, summed over halos and files, were the data uniform."""
    vol = min(4.0 / 3.0 * math.pi * c["rmax"] ** 3, BOX ** 3)
    return c["halos"] * c["files"] * c["particles"] * vol / BOX ** 3


def draw(rng):
    while True:
        call = rng.choice(["noalloc", "query", "job", "job", "job", "host"])
        shells = rng.randint(8, 64)
        if call == "noalloc":
            c = _case(call, 1, _log(rng, 1000, 131072), _log(rng, 50, 32768), 0.01, round(rng.uniform(5.0, 40.0), 2),
                      shells, periodic=rng.random() < 0.7)
        elif call == "query":
            c = _case(call, rng.randint(1, 3), _log(rng, 1e6, 3e7), _log(rng, 100, 1e6), 0.001,
                      round(rng.uniform(1.0, 10.0), 2), shells, data=rng.choice(["uniform", "clustered"]))
        elif call == "host":
            c = _case(call, 1, _log(rng, 1e5, 1e7), _log(rng, 1e3, 3e5), 0.001, round(rng.uniform(1.0, 10.0), 2), shells)
        else:
            data = rng.choice(["uniform", "clustered"])
            index = rng.choice(["grid", "grid", "grid", "morton", "learned"])
            top = 1e8 if index == "grid" else 3e7
            c = _case(call, rng.randint(1, 3), _log(rng, 1e5, top), _log(rng, 1e3, 1e7), 0.001,
                      round(rng.uniform(1.0, 20.0), 2), shells, data=data, index=index,
                      schedule=rng.choice(["auto", "queue"]), periodic=rng.random() < 0.8)
        heavy = (8.0 if c["data"] == "clustered" else 1.0) * (1.0 if c["index"] == "grid" else 3.0)
        if heavy * _pairs(c) <= 1.2e9 and c["halos"] * c["shells"] <= 4e8:
            return c


@functools.lru_cache(maxsize=1)
def _context():
    return sjcs.Context(0)  # a program opens one context


def _clumps(g):
    """1e4 clumps: centres, sigma log-uniform in [2, 20], weights lognormal(0, 1.5)."""
    k = 10_000
    centre = torch.rand(k, 3, generator=g, device="cuda") * BOX
    sigma = 2.0 * 10.0 ** torch.rand(k, 1, generator=g, device="cuda")
    weight = torch.exp(1.5 * torch.randn(k, generator=g, device="cuda"))
    return centre, sigma, torch.cumsum(weight.double(), 0)


def _in_box(x):
    x = torch.remainder(x, BOX)
    return torch.where(x >= BOX, torch.zeros_like(x), x)


def _pick(cum, m, g):
    u = torch.rand(m, generator=g, device="cuda", dtype=torch.float64) * cum[-1]
    return torch.searchsorted(cum, u).clamp_(max=cum.numel() - 1)


def _particles(data, n, g, clumps):
    p = torch.rand(n, 3, generator=g, device="cuda") * BOX
    if data == "clustered":
        centre, sigma, cum = clumps
        m = int(0.6 * n)
        k = _pick(cum, m, g)
        p[:m] = centre[k] + sigma[k] * torch.randn(m, 3, generator=g, device="cuda")
    return _in_box(p)


def _halos(data, m, g, clumps):
    h = torch.rand(m, 3, generator=g, device="cuda") * BOX
    if data == "clustered":
        centre, _, cum = clumps
        j = int(0.7 * m)
        h[:j] = centre[_pick(cum, j, g)] + torch.randn(j, 3, generator=g, device="cuda")
        h = h[torch.randperm(m, generator=g, device="cuda")].contiguous()
    return _in_box(h)


def _build(ctx, s, xyz):
    return ctx.build_index(xyz, radius_hint=s["case"]["rmax"], kind=KINDS[s["case"]["index"]])


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    clumps = _clumps(g) if case["data"] == "clustered" else None
    s = {"case": case, "r2": sjcs.radius_table(case["rmin"], case["rmax"], case["shells"]), "query": None}
    parts = [_particles(case["data"], case["particles"], g, clumps) for _ in range(case["files"])]
    halos = _halos(case["data"], case["halos"], g, clumps)
    if case["call"] == "noalloc":
        s["counts"] = torch.zeros(case["halos"], case["shells"], dtype=torch.int32, device="cuda")
    elif case["call"] == "query":
        s["index"] = [_build(_context(), s, p) for p in parts]  # resident: the requests come later
        for i in s["index"]:
            i.wait()
        parts = None
    elif case["call"] == "host":
        def pinned(t, dtype=np.float32):
            b = nat.PinnedBuffer(tuple(t.shape), dtype)
            b.array[...] = t.cpu().numpy()
            return b
        s["pinned"] = [pinned(p) for p in parts], pinned(halos)
        s["out"] = np.zeros((case["halos"], case["shells"]), np.uint64)
        parts = [b.array for b in s["pinned"][0]]
        halos = s["pinned"][1].array
    s["particles"], s["halos"] = parts, halos
    return s


class _DeviceCounts:
    """A query's device counts as a CUDA array that torch can view; it keeps the query alive."""

    def __init__(self, q):
        self.query = q
        self.__cuda_array_interface__ = {"shape": (q.nhalos, q.nrads), "typestr": "<i4",
                                         "data": (q.device_counts_ptr, False), "version": 3}


def _query(ctx, s):
    """A new query (the previous pass's is released: its counts have been used)."""
    if s["query"] is not None:
        s["query"].destroy()
    q = ctx.query(s["halos"], s["r2"], periodic=s["case"]["periodic"])
    q.set_schedule(SCHEDULES[s["case"]["schedule"]])
    s["query"] = q
    return q


def _device_counts(ctx, q):
    """The counts on the device, torch's work ordered after the count."""
    torch.cuda.current_stream().wait_stream(torch.cuda.ExternalStream(ctx.stream(1)))
    return torch.as_tensor(_DeviceCounts(q), device="cuda")


def run(state):
    s, case = state, state["case"]
    if case["call"] == "noalloc":
        p, h, r2, out = s["particles"][0], s["halos"], s["r2"], s["counts"]
        out.zero_()
        rc = nat.lib().sjcs_count_noalloc(
            ctypes.c_void_p(p.data_ptr()), p.shape[0], ctypes.c_void_p(h.data_ptr()), 12, h.shape[0],
            ctypes.c_void_p(r2.ctypes.data), len(r2), 1 if case["periodic"] else 0, ctypes.c_void_p(out.data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise sjcs.SjcsError(rc, nat.lib().sjcs_last_error().decode())
        return out
    ctx = _context()
    if case["call"] == "query":
        q = _query(ctx, s)
        q.count_many(s["index"])
        return _device_counts(ctx, q)
    index = [_build(ctx, s, p) for p in s["particles"]]
    q = _query(ctx, s)
    q.count_many(index)
    if case["call"] == "host":
        q.read_counts(s["out"])
    for i in index:
        i.destroy()
    return s["out"] if case["call"] == "host" else _device_counts(ctx, q)


def work(case):
    counts = case["halos"] * case["shells"] * (8 if case["call"] == "host" else 4)
    hits = _pairs(case)  # a lower bound for clustered data
    particles = 12 * case["files"] * case["particles"]
    if case["call"] == "query":  # the resident particles near the request's halos
        particles = min(particles, 12 * hits)
    # a pair inside R: three differences, three squares, two sums
    return {"bytes": particles + 12 * case["halos"] + counts, "flops": 8 * hits}
