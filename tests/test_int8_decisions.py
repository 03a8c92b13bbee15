"""The int8 decision rules against the oracle where their tables change form: Metropolis tables
with a zero among the thresholds (low temperature: no uniform flips) take the general rule, all
others the one-comparison rule; heat bath takes any table.  Shapes cover one chunk per row, rows
padded to 16 bytes, and rows and planes that wrap onto themselves."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(2, 8), (6, 24), (34, 96), (40, 1032), (2, 2, 8), (8, 6, 24), (4, 10, 64)]


# 2D: exp(-8 beta) 2^32 < 1 above beta = 2.7726; 3D: exp(-12 beta) 2^32 < 1 above 1.8484
@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("algorithm", ["metropolis", "heatbath"])
@pytest.mark.parametrize("beta", [0.0, 0.44, 1.84, 1.86, 2.76, 2.78, 6.0])
def test_rules_at_their_limits(oracle_mod, shape, algorithm, beta):
    from pyising_b200.backend import B200Int8

    lat = oracle_mod.random_lattice(shape, 5)
    sim = B200Int8(shape, beta, seed=2**34 + 3, algorithm=algorithm, init=lat)
    ref = oracle_mod.OracleInt8(shape, beta, seed=2**34 + 3, algorithm=algorithm, init=lat)
    np.testing.assert_array_equal(sim.sweep_measured(6, 2), ref.sweep(6, measure_every=2))
    sim.sweep(9)
    ref.sweep(9)
    np.testing.assert_array_equal(sim.get_lattice(), ref.get_lattice())
    assert sim.observables_int() == ref.observables_int()


@pytest.mark.parametrize("shape", [(64, 96), (32, 48), (8, 6, 24)], ids=str)
@pytest.mark.parametrize("algorithm", ["metropolis", "heatbath"])
@pytest.mark.parametrize("low", [0, 1, 0xFFFFFFFF])
def test_tables_with_extreme_entries(oracle_mod, shape, algorithm, low):
    """Custom tables with an entry that never, hardly ever or (but for one uniform) always accepts,
    on every schedule and on bands of odd and even height."""
    from pyising_b200._lib import check, lib
    from pyising_b200.backend import B200Int8

    n = 2 * len(shape) + 1
    table = np.array([(0x9E3779B9 * (i + 5)) & 0xFFFFFFFF for i in range(n)], np.uint32)
    table[n - 1] = low
    table[n // 2 + 1] = max(int(table[n // 2 + 1]), 1)
    lat = oracle_mod.random_lattice(shape, 9)
    ref = oracle_mod.OracleInt8(shape, 0.4, seed=11, algorithm=algorithm, init=lat)
    ref.table = table.copy()
    ref.sweep(8)
    for band in (0, 1, 2, 3, 4):
        for schedule in ("auto", "launches", "temporal"):
            sim = B200Int8(shape, 0.4, seed=11, algorithm=algorithm, init=lat)
            check(lib().ising_set_knob(sim._h, 1, band), "set_knob")
            sim.table = table
            sim._upload_table()
            sim.set_schedule(schedule)
            sim.sweep(8)
            np.testing.assert_array_equal(sim.get_lattice(), ref.get_lattice(),
                                          err_msg=f"{schedule} band {band}")
