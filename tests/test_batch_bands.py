"""Batches whose lattices need bands of different heights in one launch: rows of one chunk, of a few
and of many, big enough for the band kernel, against the lattices run alone."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [
    [(300000, 8), (150000, 32), (4096, 4096), (400, 8192)],
    [(600, 400, 24), (300, 300, 32), (64, 400, 64), (40, 200, 512)],
    [(250000, 24), (1000, 4104)],
], ids=str)
def test_bands_of_different_heights_in_one_batch(shapes):
    from pyising_b200.backend import B200Int8
    from pyising_b200.ensemble import Ensemble, Job

    beta = 0.44 if len(shapes[0]) == 2 else 0.22
    jobs = [Job(s, beta, 3, seed=5 + i, measure_every=2, init="philox", keep_lattice=True)
            for i, s in enumerate(shapes)]
    jobs += [Job(s, beta, 3, seed=50 + i, init="philox", keep_lattice=True)
             for i, s in enumerate(shapes * 2)]
    with Ensemble() as ens:
        ids = [ens.add(j) for j in jobs]
        ens.run()
        for i, job in zip(ids, jobs, strict=True):
            res = ens.result(i)
            sim = B200Int8(job.shape, beta, seed=job.seed, init="philox")
            series = sim.sweep_measured(3, 2) if job.measure_every else sim.sweep(3)
            if job.measure_every:
                np.testing.assert_array_equal(res.series, series)
            np.testing.assert_array_equal(res.lattice, sim.get_lattice())
