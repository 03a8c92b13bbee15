"""Temporal tiles whose steps have more items than a CTA has threads, packed words on one lane each,
padded rows among them, and lattices much wider than high (few bands, tiles that wrap onto
themselves), against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA_C_2D = 0.44068679350977147


# 148 SMs: bands of 17, 2 and 2 rows; 693, 2048 and 3072 chunks in a step
@pytest.mark.parametrize("shape", [(2400, 1032), (6, 16384), (10, 16392)], ids=str)
@pytest.mark.parametrize("algorithm,beta", [("metropolis", BETA_C_2D), ("heatbath", 0.4),
                                            ("metropolis", 3.0)])
def test_int8_steps_of_several_passes(oracle_mod, shape, algorithm, beta):
    from pyising_b200.backend import B200Int8

    lat = oracle_mod.random_lattice(shape, 4)
    sim = B200Int8(shape, beta, seed=2**36 + 1, algorithm=algorithm, init=lat)
    ref = oracle_mod.OracleInt8(shape, beta, seed=2**36 + 1, algorithm=algorithm, init=lat)
    sim.set_schedule("temporal")
    sim.sweep(4)
    ref.sweep(4)
    np.testing.assert_array_equal(sim.sweep_measured(5, 2), ref.sweep(5, measure_every=2))
    np.testing.assert_array_equal(sim.get_lattice(), ref.get_lattice())


# 288 words in the first step (one lane per word), 600, and 2048 and more in rows of 512
@pytest.mark.parametrize("shape", [(600, 4096), (3000, 3200), (4, 65536), (20, 65536)], ids=str)
@pytest.mark.parametrize("beta", [0.1, BETA_C_2D, 1.5])
def test_msc_steps_of_several_passes(oracle_mod, shape, beta):
    from pyising_b200.backend import B200MultiSpin

    lat = oracle_mod.random_lattice(shape, 6)
    sim = B200MultiSpin(shape, beta, seed=2**37 + 5, init=lat)
    ref = oracle_mod.OracleMultiSpin(shape, beta, seed=2**37 + 5, init=lat)
    sim.set_schedule("temporal")
    sim.sweep(4)
    ref.sweep(4)
    np.testing.assert_array_equal(sim.sweep_measured(5, 2), ref.sweep(5, measure_every=2))
    w0, w1 = sim.colour_arrays()
    np.testing.assert_array_equal(w0, ref.w[0])
    np.testing.assert_array_equal(w1, ref.w[1])
