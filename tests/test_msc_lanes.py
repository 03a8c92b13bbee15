"""The packed lane walk against the oracle: one word per row, a few, a warp's, more; bands of two
rows and of four with a shorter last one; the last warp partly without a column; and just below
its range."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# words per row: 1 (37886 rows: below the range), 3, 5, 32, 33, 40; four-row bands with 3 and 65
@pytest.mark.parametrize("shape", [(37886, 128), (37890, 128), (12634, 384), (7700, 640),
                                   (1186, 4096), (1150, 4224), (970, 5120), (50522, 384),
                                   (2370, 8320)], ids=str)
@pytest.mark.parametrize("beta", [0.1, 0.44068679350977147, 1.5])
def test_msc_lanes(oracle_mod, shape, beta):
    from pyising_b200.backend import B200MultiSpin

    lat = oracle_mod.random_lattice(shape, 6)
    sim = B200MultiSpin(shape, beta, seed=2**37 + 5, init=lat)
    ref = oracle_mod.OracleMultiSpin(shape, beta, seed=2**37 + 5, init=lat)
    sim.set_schedule("launches")
    sim.t = ref.t = 2**32 - 2  # the sweep counter wraps on the way
    sim.sweep(3)
    ref.sweep(3)
    np.testing.assert_array_equal(sim.sweep_measured(3, 2), ref.sweep(3, measure_every=2))
    w0, w1 = sim.colour_arrays()
    np.testing.assert_array_equal(w0, ref.w[0])
    np.testing.assert_array_equal(w1, ref.w[1])
    assert sim.observables_int() == ref.observables_int()
