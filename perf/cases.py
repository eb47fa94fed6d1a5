"""The Swendsen-Wang work whose speed matters, as cases: what a program has this package do, through
its public entry points, over the range of sizes, tiles, lcg widths and temperatures it is used with.

Every case is one of these kinds:

  cli    one 2D lattice swept call by call and measured every tenth sweep, as the Ising2D program
         does it (one update per call, energy and magnetisation on the host)
  chain  one 2D lattice over a stretch of its Markov chain: n sweeps in one call, measured every
         tenth, the sample series read at the end (a point of a temperature scan; a job on its own)
  bulk   the same without measurement: equilibration, or a caller that works on the device spins
  batch  many independent 2D lattices advanced together, measured every tenth sweep, their sample
         series read at the end
  io     the same lattices through host buffers: every round's spins come from and go to the host
  serve  simulation jobs (side, temperature, sweeps, seed) through the continuous-batching server
  cube   one 3D lattice: n sweeps, measured every tenth, series and final spins read
  lcg32  the random-number generator on its own

The state starts from a hot start per seed followed by a few sweeps, so that a pass meets clusters as
they are in a simulation and not those of a random start.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import computational_physics_b200 as cp
from computational_physics_b200 import autotune, rng_bench
from computational_physics_b200.batch import BatchedSW
from computational_physics_b200.lattice3 import SwendsenWang3D
from computational_physics_b200.serving import Job, Server, poisson_jobs

T_C = 2.2691853        # critical temperature of the 2D model
T_C3 = 4.5115          # of the 3D model
MIX_SIDES = (64, 96, 128, 192, 256, 384, 512)
L2_BYTES = 126e6       # a state below this stays on the chip from sweep to sweep
TILES = ((16, 8), (8, 8), (32, 4), (16, 16), (32, 8), (8, 16), (16, 4), (16, 6), (8, 5))
TILES3 = ((16, 4, 4), (8, 4, 4), (32, 2, 4), (16, 2, 8), (8, 8, 2))


def listed():
    return [
        # The reference's own default run: 128 x 128 at T_c from the Ising2D loop.  Ten sweeps and a
        # measurement per pass: nothing but latency.
        dict(name="cli_128", kind="cli", L0=128, L1=128, tx=16, ty=8, W=16, T=T_C, sweeps=10),
        # A small lattice's long chain in one call (a job of a scan, or one served on its own).
        dict(name="chain_256", kind="chain", L0=256, L1=256, tx=16, ty=8, W=16, T=2.3, sweeps=200, every=10),
        # The 1024 x 1024 run with 8 x 8 tiles.
        dict(name="chain_1024", kind="chain", L0=1024, L1=1024, tx=8, ty=8, W=16, T=T_C, sweeps=20, every=10),
        # Ragged: extents that are a multiple of neither tile nor block nor 16 bytes, the lcg width
        # of an AVX2 host, ordered phase (one cluster holds most sites).
        dict(name="chain_ragged_w8", kind="chain", L0=1500, L1=1102, tx=8, ty=8, W=8, T=2.0, sweeps=10, every=10),
        # Bandwidth sizes: 4096 x 4096 in the disordered phase (many small clusters) ...
        dict(name="bulk_4096", kind="bulk", L0=4096, L1=4096, tx=16, ty=8, W=16, T=3.0, sweeps=4),
        # ... and the largest lattice, 16384 x 16384 at T_c.
        dict(name="bulk_16384", kind="bulk", L0=16384, L1=16384, tx=16, ty=8, W=16, T=T_C, sweeps=2),
        # The mix of 512 lattices of 64 to 512 sites a side at T in [2.0, 2.6].
        dict(name="batch_512", kind="batch", count=512, low=0, high=6, rounds=500, every=10),
        # The same mix through host buffers (spins in and out every round).
        dict(name="io_512", kind="io", count=512, low=0, high=6, rounds=4),
        # A burst of served jobs: side log-uniform in [32, 1024], sweeps log-uniform.
        dict(name="serve_24", kind="serve", jobs=24, L_low=32, L_high=1024, S_low=1000, S_high=5000),
        # 3D at its critical temperature, default tile, whole blocks ...
        dict(name="cube_256", kind="cube", L0=256, L1=256, L2=256, tx=16, ty=4, tz=4, W=16, T=T_C3, sweeps=100,
             every=10),
        # ... and a small ragged one.
        dict(name="cube_ragged", kind="cube", L0=90, L1=76, L2=54, tx=16, ty=4, tz=4, W=16, T=T_C3, sweeps=50,
             every=10),
        # The generator alone (TestRNG): 2e9 numbers from 148 x 512 streams.
        dict(name="lcg32_2e9", kind="lcg32", streams=148 * 512, W=16, updates=1652),
    ]


# ---------------------------------------------------------------------------------------------
# one more case of the same ranges

def _log(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def _even(x):
    return max(2, 2 * round(x / 2))


def _sweeps(sites, budget, most):
    return int(max(1, min(most, budget // sites)))


def draw(rng):
    kind = rng.choice(("cli", "chain", "chain", "bulk", "bulk", "batch", "io", "serve", "cube", "cube", "lcg32"))
    tx, ty = rng.choice(TILES)
    W = rng.choice((8, 16, 16, 16, 32))
    T = round(rng.uniform(1.5, 3.5), 3)
    if kind in ("cli", "chain", "bulk"):
        top = {"cli": 1024, "chain": 4096, "bulk": 16384}[kind]
        L0, L1 = _even(_log(rng, 32, top)), _even(_log(rng, 32, top))
        if rng.random() < 0.5:  # sides that are multiples of the tile, as most programs choose them
            L0, L1 = max(32, L0 // 32 * 32), max(32, L1 // 32 * 32)
        n = L0 * L1
        c = dict(kind=kind, L0=L0, L1=L1, tx=tx, ty=ty, W=W, T=T)
        if kind == "cli":
            return dict(c, sweeps=10)
        if kind == "bulk":
            return dict(c, sweeps=_sweeps(n, 2 ** 29, 50))
        return dict(c, sweeps=10 * max(1, _sweeps(n, 2 ** 29, 500) // 10), every=10)
    if kind in ("batch", "io"):
        low = rng.randrange(0, 5)
        high = rng.randrange(low, 7)
        count = int(_log(rng, 4, 512))
        if kind == "io":
            return dict(kind=kind, count=count, low=low, high=high, rounds=2 * rng.randrange(1, 3))
        return dict(kind=kind, count=count, low=low, high=high, rounds=10 * rng.randrange(5, 40), every=10)
    if kind == "serve":
        return dict(kind=kind, jobs=rng.randrange(4, 24), L_low=32, L_high=rng.choice((256, 512, 1024)),
                    S_low=rng.randrange(200, 1000), S_high=rng.randrange(1001, 4000))
    if kind == "cube":
        t3 = rng.choice(TILES3)
        L0, L1, L2 = (_even(_log(rng, 16, 256)) for _ in range(3))
        if rng.random() < 0.5:
            L0, L1, L2 = max(32, L0 // 32 * 32), max(16, L1 // 16 * 16), max(16, L2 // 16 * 16)
        return dict(kind=kind, L0=L0, L1=L1, L2=L2, tx=t3[0], ty=t3[1], tz=t3[2], W=W,
                    T=round(rng.uniform(3.5, 6.0), 3), sweeps=10 * max(1, _sweeps(L0 * L1 * L2, 2 ** 29, 50) // 10),
                    every=10)
    streams = int(_log(rng, 500, 148 * 512))
    updates = 64 // W * int(_log(rng, 8, 9 + 2 ** 30 / (64 * streams)))  # up to 2^30 numbers
    return dict(kind=kind, streams=streams, W=W, updates=updates)


# ---------------------------------------------------------------------------------------------
# states

class _DeviceSpins:
    """A lattice's device spins as torch takes them (zero copy); a tensor made of it keeps it, and so
    the lattice that owns the buffer."""

    def __init__(self, sw, shape):
        self.owner = sw
        ptr = sw.device_buffers()[0]
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "|u1", "version": 3}


def _mix(case, seed):
    """(side, temperature, seed) per lattice: sides uniform in a range of MIX_SIDES."""
    rng = np.random.default_rng([case["count"], seed])
    sides = rng.choice(MIX_SIDES[case["low"]:case["high"] + 1], size=case["count"])
    temps = rng.uniform(2.0, 2.6, size=case["count"]).astype(np.float32)
    seeds = rng.integers(1, 2 ** 31 - 1, size=case["count"])
    return [(int(L), float(T), int(s)) for L, T, s in zip(sides, temps, seeds)]


def _same_sides(case):
    """The sides of the mix do not depend on the seed, so that a case is the same work each time."""
    return [L for L, _, _ in _mix(case, 0)]


def _add_mix(case, seed, every):
    table = autotune.load("nvidia_b200")
    b = BatchedSW(capacity=case["count"])
    ids = []
    for L, (_, T, s) in zip(_same_sides(case), _mix(case, seed)):
        tile, block = autotune.choice(L, table)
        lid = b.add(L, L, T, s, tile, block)
        b.hot_start(lid, s)
        if every:
            b.set_schedule(lid, measure_every=every)
        ids.append(lid)
    return b, ids


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("cli", "chain", "bulk"):
        sw = cp.SwendsenWang2D(case["L0"], case["L1"], (case["tx"], case["ty"]), case["W"], seed_base=seed + 1)
        if kind == "cli":
            sw.cold_start(1)
        else:
            sw.hot_start(seed + 1)
        sw.update(case["T"], 20)
        s["sw"] = sw
        s["spins"] = torch.as_tensor(_DeviceSpins(sw, (case["L1"], case["L0"])), device="cuda")
    elif kind == "batch":
        s["batch"], s["ids"] = _add_mix(case, seed, case["every"])
        s["batch"].sweep(10)
    elif kind == "io":
        s["batch"], s["ids"] = _add_mix(case, seed, 0)
        io = s["batch"].host_io(s["ids"])
        total = sum(v.size for v in io.inputs)
        # the lattices' buffers follow each other in one arena; the array over it keeps it allocated
        buf = (ctypes.c_uint8 * total).from_address(io.inputs[0].ctypes.data)
        buf.owner = io
        arena = np.frombuffer(buf, np.uint8)
        arena[:] = np.unpackbits(np.frombuffer(np.random.default_rng(seed).bytes(total // 8 + 1), np.uint8))[:total]
        s["batch"].update_host_io_rounds(io, 4)
        s["io"], s["arena"] = io, arena
    elif kind == "serve":
        jobs = poisson_jobs(100.0, case["jobs"], 7, (case["L_low"], case["L_high"]), (1.5, 3.5),
                            (case["S_low"], case["S_high"]))
        rng = np.random.default_rng([case["jobs"], seed])
        # the sizes and lengths are the same for every seed, the temperatures and streams are not
        s["jobs"] = [(j.L, float(np.float32(rng.uniform(1.5, 3.5))), j.sweeps, int(rng.integers(1, 2 ** 31 - 1)))
                     for j in jobs]
        s["server"] = Server(hbm_budget_bytes=8 << 30, capacity=256)
    elif kind == "cube":
        sw = SwendsenWang3D(case["L0"], case["L1"], case["L2"], (case["tx"], case["ty"], case["tz"]), case["W"], seed + 1)
        sw.hot_start(seed + 1)
        sw.update(case["T"], 20)
        s["sw"] = sw
    else:
        s["seed"] = seed + 1
    return s


# ---------------------------------------------------------------------------------------------
# one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "cli":
        sw = state["sw"]
        for _ in range(case["sweeps"]):
            sw.update(case["T"])
        return {"em": list(sw.energy_magnetization_sums()), "spins": state["spins"]}
    if kind == "chain":
        sw = state["sw"]
        sw.reset_accumulators()
        sw.update(case["T"], case["sweeps"], case["every"])
        return {"samples": sw.samples(), "spins": state["spins"]}
    if kind == "bulk":
        state["sw"].update(case["T"], case["sweeps"])
        return state["spins"]
    if kind == "batch":
        b = state["batch"]
        b.sweep(case["rounds"], measure=True)
        return np.concatenate([b.samples(i) for i in state["ids"]])
    if kind == "io":
        state["batch"].update_host_io_rounds(state["io"], case["rounds"])
        return state["arena"]
    if kind == "serve":
        jobs = [Job(i, L, T, n, sd) for i, (L, T, n, sd) in enumerate(state["jobs"])]
        state["server"].run(jobs, realtime=False)
        return {"series": np.concatenate([j.result["series"] for j in jobs]),
                "E": np.array([j.result["E"] for j in jobs])}
    if kind == "cube":
        sw = state["sw"]
        sw.update(case["T"], case["sweeps"], case["every"])
        return {"samples": sw.samples()[0], "spins": sw.get_spins()}
    r = rng_bench.generate(case["streams"], case["updates"], case["W"], state["seed"], case["streams"] // 2)
    return {"report": r["report"], "checksum": r["checksum"]}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    """bytes: spins and lcg32 streams in and out, once per pass while they fit the L2 and once per
    sweep beyond it; host spins in and out every round.  flops: two random numbers and two
    comparisons per site and sweep (three in 3D), one multiply and one add per number, and the flip;
    for the generator alone one multiply, one add and the conversion per number."""
    kind = case["kind"]

    def lattice(n, tiles, W, sweeps, numbers):
        state = 2 * (n + tiles * (5 * W + 4))
        return dict(bytes=state * (sweeps if state / 2 > L2_BYTES else 1), flops=n * sweeps * (3 * numbers + 1))

    if kind in ("cli", "chain", "bulk"):
        tiles = -(-case["L0"] // case["tx"]) * -(-case["L1"] // case["ty"])
        return lattice(case["L0"] * case["L1"], tiles, case["W"], case["sweeps"], 2)
    if kind == "cube":
        tiles = -(-case["L0"] // case["tx"]) * -(-case["L1"] // case["ty"]) * -(-case["L2"] // case["tz"])
        return lattice(case["L0"] * case["L1"] * case["L2"], tiles, case["W"], case["sweeps"], 3)
    if kind in ("batch", "io"):
        n = sum(L * L for L in _same_sides(case))
        w = lattice(n, n / 128, 16, case["rounds"], 2)
        return dict(w, bytes=2 * n * case["rounds"]) if kind == "io" else w
    if kind == "serve":
        jobs = poisson_jobs(100.0, case["jobs"], 7, (case["L_low"], case["L_high"]), (1.5, 3.5),
                            (case["S_low"], case["S_high"]))
        return dict(bytes=sum(2 * j.L * j.L * (1 + 84 / 128) for j in jobs), flops=7 * sum(j.site_updates for j in jobs))
    numbers = case["streams"] * case["W"] * case["updates"]
    return dict(bytes=256, flops=3 * numbers)


# ---------------------------------------------------------------------------------------------
# the generator's last 64 numbers in 64 bits

_A = np.array([1372383749, 2891336453, 2024337845, 32310901, 29943829], np.uint64)
_C = np.array([1289706101, 1640531513, 797082193, 626627237, 1013904223], np.uint64)


def exact(case, seed):
    """Spins, samples and sums are whole numbers.  The generator's report is u / 2^32 of the stream's
    last 64 draws u, followed here from POSIX drand48 and the lcg32 recurrence (random/src/lcg32.cpp:27-84)."""
    if case["kind"] != "lcg32" or case["updates"] > 200000:
        return None
    W = case["W"]
    x = ((seed + 1 + case["streams"] // 2) << 16 | 0x330E) & ((1 << 48) - 1)
    draws = []
    for _ in range(W + 1):
        x = (0x5DEECE66D * x + 0xB) & ((1 << 48) - 1)
        draws.append(x / 2.0 ** 48)
    sel = np.array([int(1000.0 * d) % 5 for d in draws[:W]])
    a, c = _A[sel], _C[sel]
    state = np.zeros(W, np.uint64)
    v = int(0xEFFFFFFF * draws[W]) + 1
    for i in range(W):
        v = (int(a[i]) * v + int(c[i])) & 0xFFFFFFFF
        state[i] = v
    lanes = np.arange(W)
    last = []
    for it in range(1, case["updates"] + 1):
        if it % 15 == 0:
            turn = (lanes + int(state[it % W]) + (0 if it % 2 else 1)) % W
            a, c = a[turn], c[turn]
        state = (a * state + c) & np.uint64(0xFFFFFFFF)
        if it > case["updates"] - 64 // W:
            last.append(state.astype(np.float64) / 2.0 ** 32)
    return {"report": np.concatenate(last), "checksum": None}
