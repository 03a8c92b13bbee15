"""Batches of several kernel classes at once (each on its own stream) and on both sides of the rules
that pick one chunk or word per thread: every job against the oracle, with jobs joining while
others run, in odd numbers of half-sweeps and in graph chunks."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

JOBS = [  # shape, variant, algorithm, sweeps, every
    ((16, 24), "int8", "metropolis", 41, 3),
    ((64, 64), "int8", "metropolis", 150, 10),
    ((300, 1032), "int8", "heatbath", 37, 5),
    ((8, 6, 40), "int8", "heatbath", 64, 4),
    ((20, 30, 32), "int8", "metropolis", 33, 7),
    ((2, 128), "msc", "metropolis", 55, 5),
    ((130, 1152), "msc", "metropolis", 140, 10),
    ((64, 4096), "msc", "metropolis", 20, 0),
]


def check(oracle_mod, job, result):
    cls = oracle_mod.OracleMultiSpin if job.variant == "msc" else oracle_mod.OracleInt8
    kw = {} if job.variant == "msc" else {"algorithm": job.algorithm}
    ref = cls(job.shape, job.beta, seed=job.seed, init=job.init, **kw)
    want = ref.sweep(job.sweeps, measure_every=job.measure_every)
    if job.measure_every:
        np.testing.assert_array_equal(result.series, want, err_msg=str(job.shape))
    np.testing.assert_array_equal(result.lattice, ref.get_lattice(), err_msg=str(job.shape))


def make(oracle_mod, specs, sweeps=None):
    from pyising_b200.ensemble import Job

    return [Job(shape, 0.43 if len(shape) == 2 else 0.22, sweeps or n, seed=2**33 + i,
                variant=variant, algorithm=alg, measure_every=every,
                init=oracle_mod.random_lattice(shape, i), keep_lattice=True)
            for i, (shape, variant, alg, n, every) in enumerate(specs)]


@pytest.mark.parametrize("chunk", [0, 8, 32])
def test_classes_side_by_side(oracle_mod, chunk):
    from pyising_b200.ensemble import Ensemble

    jobs = make(oracle_mod, JOBS)
    with Ensemble() as ens:
        ens.set_knob("graph_chunk", chunk)
        ids = [ens.add(j) for j in jobs[:5]]
        ens.run(7)                     # stops between the colours of a sweep
        ids += [ens.add(j) for j in jobs[5:]]
        ens.run(90)
        late = make(oracle_mod, JOBS[:2])
        late_ids = [ens.add(j) for j in late]
        ens.run()
        for j, i in zip(jobs + late, ids + late_ids, strict=True):
            check(oracle_mod, j, ens.result(i))


@pytest.mark.parametrize("spec,count", [
    (((1024, 1024), "int8", "metropolis", 6, 2), 20),   # bands
    (((160, 160, 160), "int8", "heatbath", 4, 2), 9),   # 3D bands
    (((4096, 4096), "msc", "metropolis", 4, 2), 8),     # word ranges
], ids=str)
def test_large_classes(oracle_mod, spec, count):
    from pyising_b200.ensemble import Ensemble

    jobs = make(oracle_mod, [spec] * count + [JOBS[0]])
    with Ensemble() as ens:
        ids = [ens.add(j) for j in jobs]
        ens.run()
        for k in (0, count - 1, count):
            check(oracle_mod, jobs[k], ens.result(ids[k]))
