"""The packed lane walk with bands of four and six rows and a shorter last one against the oracle:
one, three and more words per row (the smallest sizes with such bands, from the share of the lanes
that makes them faster than word ranges)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA_C_2D = 0.44068679350977147


@pytest.mark.parametrize("shape", [(243006, 128), (82002, 384), (3742, 8320), (9242, 4224)],
                         ids=str)
def test_lane_bands_of_several_pairs_of_rows(oracle_mod, shape):
    from pyising_b200.backend import B200MultiSpin

    lat = oracle_mod.random_lattice(shape, 6)
    sim = B200MultiSpin(shape, BETA_C_2D, seed=2**37 + 5, init=lat)
    ref = oracle_mod.OracleMultiSpin(shape, BETA_C_2D, seed=2**37 + 5, init=lat)
    sim.set_schedule("launches")
    sim.sweep(2)
    ref.sweep(2)
    np.testing.assert_array_equal(sim.sweep_measured(1, 1), ref.sweep(1, measure_every=1))
    w0, w1 = sim.colour_arrays()
    np.testing.assert_array_equal(w0, ref.w[0])
    np.testing.assert_array_equal(w1, ref.w[1])
