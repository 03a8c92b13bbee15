"""Workloads that time the framework through its public entry points.

Each case is one thing a user's program does: sweeps of one lattice with or without measurements
and the lattice handed back, a temperature scan on one lattice, cluster updates, a batched
ensemble, a stream of jobs through the server.  Sizes and temperatures are those of the
repository's own configurations (bench.py, plan.py, validate.py) or ragged neighbours of them.
Every result is an integer: spins, packed words, exact (M, E).
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

import pyising_b200 as pb
from pyising_b200.ensemble import Ensemble, Job, Server

TC = {2: pb.TC_2D, 3: 1.0 / 0.221654626}

#: Site updates of the largest case of each kind (a drawn case stays below).
CAP = {"int8": 200 * 16384**2, "int8_3d": 200 * 256**3, "msc": 1000 * 16384**2}


def sim(name, variant, shape, algorithm, sweeps, every=0, t_rel=1.0):
    lz, ly, lx = ((1, *shape) if len(shape) == 2 else shape)
    return {"name": name, "kind": "sweeps", "variant": variant, "ndim": len(shape), "lz": lz,
            "ly": ly, "lx": lx, "algorithm": algorithm, "sweeps": sweeps, "every": every,
            "t_rel": t_rel}


def listed():
    return [
        # the smallest call: a few sweeps of a small lattice, then its energy (a user's loop body)
        sim("int8 64^2 call", "int8", (64, 64), "metropolis", 10),
        # the energy scan of the validation suite: one L = 128 lattice taken through temperatures
        {"name": "int8 128^2 scan", "kind": "scan", "variant": "int8", "ly": 128, "lx": 128,
         "algorithm": "heatbath", "temps": 5, "sweeps": 100, "every": 10},
        # the small benchmark job: 1024^2, 1000 sweeps at T_c
        sim("int8 1024^2", "int8", (1024, 1024), "metropolis", 1000),
        # an odd size with heat bath, measured as a Monte Carlo run is: rows padded on the device
        sim("int8 1500x2488 heat bath", "int8", (1500, 2488), "heatbath", 200, 10, 1.05),
        # a lattice beyond L2, many sweeps, then a checkpoint
        sim("int8 16384^2", "int8", (16384, 16384), "metropolis", 200),
        # the 3D benchmark job's measured heat bath (shortened)
        sim("int8 3D 256^3 heat bath", "int8", (256, 256, 256), "heatbath", 200, 10),
        # a small 3D lattice of uneven sides
        sim("int8 3D 70x90x120", "int8", (70, 90, 120), "metropolis", 200, 10, 0.95),
        # a packed lattice whose rows are neither a power of two nor whole 32-word strips
        sim("msc 1152^2", "msc", (1152, 1152), "metropolis", 200, 10),
        # the headline job: packed 16384^2, 1000 sweeps at T_c, measured every 100
        sim("msc 16384^2", "msc", (16384, 16384), "metropolis", 1000, 100),
        # equilibrated starts and Binder chains: Swendsen-Wang updates with (M, E) after each
        {"name": "cluster 1024^2", "kind": "cluster", "variant": "int8", "ndim": 2, "lz": 1,
         "ly": 1024, "lx": 1024, "sweeps": 20},
        # the temperature ensemble: power-of-two int8 lattices of uneven size in one batch
        {"name": "ensemble", "kind": "ensemble", "jobs": 32, "mix": 0, "l_min": 64, "l_max": 2048,
         "sweeps": 200, "every": 10},
        # the served mix: 2D int8, packed and 3D heat-bath jobs of uneven length through the server
        {"name": "server", "kind": "server", "jobs": 21, "mix": 2026, "l_min": 128, "l_max": 4096,
         "sweeps": 200, "every": 10},
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def even(x):
    return max(2, x // 2 * 2)


def mult(x, m):
    return max(m, x // m * m)


def draw(rng):
    what = rng.choice(["int8", "int8", "int8_3d", "int8_3d", "msc", "msc", "scan", "cluster",
                       "ensemble", "server"])
    every = rng.choice([0, 10, 10, 100])
    t_rel = round(rng.uniform(0.85, 1.15), 4)
    if what in ("int8", "int8_3d", "msc"):
        if what == "int8_3d":
            side = log_int(rng, 32, 256)
            shape = (even(side), even(int(side * rng.uniform(0.7, 1.0))),
                     mult(int(side * rng.uniform(0.7, 1.0)), 8))
        else:
            side = log_int(rng, 128 if what == "msc" else 64, 16384)
            if rng.random() < 0.3:
                side = 1 << int(math.log2(side))
                shape = (side, mult(side, 128 if what == "msc" else 8))
            else:
                shape = (even(int(side * rng.uniform(0.6, 1.0))),
                         mult(side, 128 if what == "msc" else 8))
        most = max(10, CAP[what] // math.prod(shape))
        sweeps = min(log_int(rng, 10, 1000), most)
        algorithm = "metropolis" if what == "msc" else rng.choice(["metropolis", "heatbath"])
        c = sim("", "msc" if what == "msc" else "int8", shape, algorithm, sweeps, every, t_rel)
    elif what == "scan":
        side = log_int(rng, 64, 512)
        c = {"kind": "scan", "variant": "int8", "ly": even(side), "lx": mult(side, 8),
             "algorithm": rng.choice(["metropolis", "heatbath"]), "temps": rng.randint(2, 6),
             "sweeps": log_int(rng, 50, 400), "every": 10}
    elif what == "cluster":
        side = log_int(rng, 128, 4096)
        c = {"kind": "cluster", "variant": "int8", "ndim": 2, "lz": 1, "ly": even(side),
             "lx": mult(side, 8), "sweeps": rng.randint(5, 20)}
    else:
        c = {"kind": what, "jobs": rng.randint(8, 21), "mix": rng.randrange(1 << 30),
             "l_min": 64 if what == "ensemble" else 128, "l_max": rng.choice([512, 1024, 2048]),
             "sweeps": log_int(rng, 50, 200), "every": 10}
    c.pop("name", None)
    return c


def make_sim(case, seed, beta):
    shape = (case["ly"], case["lx"])
    if case.get("ndim", 2) == 3:
        shape = (case["lz"], *shape)
    return pb.create("b200", case["variant"], shape=shape, beta=beta, seed=seed,
                     algorithm=case.get("algorithm", "metropolis"), init="philox")


def host_buffers(s):
    """Page-locked arrays for the two colours, kept by the program across checkpoints."""
    lh = s.lh // 64 if s.variant == "msc" else s.lh
    dtype = torch.int64 if s.variant == "msc" else torch.int8
    bufs = [torch.empty((s.rows, lh), dtype=dtype, pin_memory=True) for _ in range(2)]
    as_np = [b.numpy().view(np.uint64) if s.variant == "msc" else b.numpy() for b in bufs]
    return tuple(as_np), bufs


def job_list(case, seed):
    """The jobs of an ensemble or a served stream: their sizes, temperatures and lengths belong to
    the case, their seeds to the inputs."""
    r = random.Random(case["mix"])
    jobs = []
    lo, hi = case["l_min"], case["l_max"]
    for i in range(case["jobs"]):
        key = seed * 1000 + i
        if case["kind"] == "ensemble":
            side = 1 << r.randint(int(math.log2(lo)), int(math.log2(hi)))
            jobs.append(Job((side, side), 1.0 / r.uniform(2.0, 2.6), case["sweeps"], seed=key,
                            measure_every=case["every"], init="philox", keep_lattice=True))
            continue
        sweeps = log_int(r, case["sweeps"] // 2, case["sweeps"] * 2)
        if r.random() < 0.7:
            variant = r.choice(["int8", "msc"])
            side = mult(log_int(r, lo, hi), 128 if variant == "msc" else 8)
            beta = 1.0 / (TC[2] * r.uniform(0.85, 1.15))
            jobs.append(Job((side, side), beta, sweeps, seed=key, variant=variant,
                            measure_every=case["every"], init="philox", keep_lattice=True))
        else:
            side = mult(log_int(r, 32, max(64, hi // 16)), 8)
            beta = 1.0 / (TC[3] * r.uniform(0.85, 1.15))
            jobs.append(Job((side, side, side), beta, sweeps, seed=key, algorithm="heatbath",
                            measure_every=case["every"], init="philox", keep_lattice=True))
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("ensemble", "server"):
        pool = Ensemble() if kind == "ensemble" else Server()
        return {"case": case, "pool": pool, "jobs": job_list(case, seed)}
    if kind == "scan":
        betas = [1.0 / (TC[2] * (0.85 + 0.3 * (k + 0.5) / case["temps"]))
                 for k in range(case["temps"])]
        s = make_sim(case, seed, betas[0])
        return {"case": case, "sim": s, "betas": betas}
    ndim = case["ndim"]
    s = make_sim(case, seed, 1.0 / (TC[ndim] * case.get("t_rel", 1.0)))
    out, keep = host_buffers(s)
    return {"case": case, "sim": s, "out": out, "keep": keep}


def spins(state):
    """The lattice as the program checkpoints it: both colour arrays in its own host buffers."""
    a, b = state["sim"].colour_arrays(state["out"])
    return [a.view(np.int64), b.view(np.int64)] if a.dtype == np.uint64 else [a, b]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        pool = state["pool"]
        ids = [pool.add(j) for j in state["jobs"]]
        pool.run()
        return collect(pool, ids)
    if kind == "server":
        pool = state["pool"]
        ids = [pool.submit(j) for j in state["jobs"]]
        for i in ids:
            pool.wait(i)
        return collect(pool, ids)
    s = state["sim"]
    if kind == "scan":
        series = []
        for beta in state["betas"]:
            s.set_beta(beta)
            s.sweep(case["sweeps"] // 2)
            series.append(s.sweep_measured(case["sweeps"], case["every"]))
        return {"series": series, "lattice": s.get_lattice()}
    if kind == "cluster":
        series = s.cluster_sweep(case["sweeps"], measure=True)
        return {"series": series, "spins": spins(state)}
    if case["every"] > 0:
        series = s.sweep_measured(case["sweeps"], case["every"])
    else:
        s.sweep(case["sweeps"])
        series = list(s.observables_int())
    return {"series": series, "spins": spins(state)}


def collect(pool, ids):
    """Series and final lattices of the finished jobs (the lattices end to end: one array)."""
    results = [pool.result(i) for i in ids]
    for i in ids:
        pool.release(i)
    return {"series": np.concatenate([r.series for r in results]),
            "lattices": np.concatenate([r.lattice.reshape(-1) for r in results])}


# Integer operations of one Philox4x32-10 block: ten rounds of two multiplies and four XORs.
BLOCK_OPS = 60
MSC_BLOCKS_PER_WORD = 3.8  # blocks until every lane of a 64-spin word is decided, at T_c


def one_lattice(variant, sites, sweeps):
    """Bytes of the lattice in and out, and the random-number operations of its updates."""
    if variant == "msc":
        return 2 * sites / 8, sweeps * sites / 64 * MSC_BLOCKS_PER_WORD * BLOCK_OPS
    return 2 * sites, sweeps * sites / 4 * BLOCK_OPS


def work(case):
    kind = case["kind"]
    if kind in ("ensemble", "server"):
        parts = [one_lattice(j.variant, j.n_spins, j.sweeps) for j in job_list(case, 0)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    sites = case.get("lz", 1) * case["ly"] * case["lx"]
    if kind == "cluster":  # a block per colour-0 site for its bonds, a bit per cluster
        return {"bytes": 2 * sites, "flops": case["sweeps"] * sites / 2 * BLOCK_OPS}
    sweeps = case["sweeps"] * (1.5 * case["temps"] if kind == "scan" else 1)
    b, f = one_lattice(case["variant"], sites, sweeps)
    return {"bytes": b, "flops": f}
