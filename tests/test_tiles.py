"""The temporal tiles against the oracle: lattices with fewer rows than a tile holds (a tile then
wraps onto itself), a shorter last band, padded rows, one-word and one-chunk items, each split of
a packed word over lanes, and every way a number of sweeps is cut into launches."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA_C_2D = 0.44068679350977147


def run(sim, ref, final):
    sim.set_schedule("temporal")
    for n in (1, 2, 3, 7, 70):
        sim.sweep(n)
        ref.sweep(n)
    np.testing.assert_array_equal(sim.sweep_measured(23, 5), ref.sweep(23, measure_every=5))
    np.testing.assert_array_equal(sim.sweep_measured(3, 1), ref.sweep(3, measure_every=1))
    final()
    assert sim.observables_int() == ref.observables_int()


@pytest.mark.parametrize("shape", [(2, 8), (4, 16), (6, 40), (62, 24), (300, 72), (298, 1032),
                                   (150, 2048), (1200, 520)], ids=str)
@pytest.mark.parametrize("algorithm,beta", [("metropolis", BETA_C_2D), ("heatbath", 0.4),
                                            ("metropolis", 3.0)])
def test_int8_tiles(oracle_mod, shape, algorithm, beta):
    from pyising_b200.backend import B200Int8

    lat = oracle_mod.random_lattice(shape, 4)
    sim = B200Int8(shape, beta, seed=2**36 + 1, algorithm=algorithm, init=lat)
    ref = oracle_mod.OracleInt8(shape, beta, seed=2**36 + 1, algorithm=algorithm, init=lat)
    sim.t = ref.t = 2**32 - 60  # the sweep counter wraps on the way
    run(sim, ref, lambda: np.testing.assert_array_equal(sim.get_lattice(), ref.get_lattice()))


# rows of 1, 3, 5, 16 and 32 words: four, two and one lane per word
@pytest.mark.parametrize("shape", [(2, 128), (6, 128), (302, 384), (500, 640), (296, 1152),
                                   (700, 2048), (450, 4096)], ids=str)
@pytest.mark.parametrize("beta", [0.1, BETA_C_2D, 1.5])
def test_msc_tiles(oracle_mod, shape, beta):
    from pyising_b200.backend import B200MultiSpin

    lat = oracle_mod.random_lattice(shape, 6)
    sim = B200MultiSpin(shape, beta, seed=2**37 + 5, init=lat)
    ref = oracle_mod.OracleMultiSpin(shape, beta, seed=2**37 + 5, init=lat)
    sim.t = ref.t = 2**32 - 60

    def final():
        w0, w1 = sim.colour_arrays()
        np.testing.assert_array_equal(w0, ref.w[0])
        np.testing.assert_array_equal(w1, ref.w[1])

    run(sim, ref, final)


def test_sweeps_into_a_captured_stream():
    """Sweeps issued into a stream under capture: without the tiles' second arrays (a capture cannot
    allocate them for later use) and, after a sweep outside it, with them."""
    import torch

    from pyising_b200.backend import B200MultiSpin

    for warm in (False, True):
        a = B200MultiSpin((64, 256), BETA_C_2D, seed=3, init="philox")
        b = B200MultiSpin((64, 256), BETA_C_2D, seed=3, init="philox")
        if warm:
            a.sweep(2)
            b.sweep(2)
        a.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            a.set_stream(torch.cuda.current_stream().cuda_stream)
            a.sweep(3)
        a.set_stream(None)
        graph.replay()
        torch.cuda.synchronize()
        b.sweep(3)
        for x, y in zip(a.colour_arrays(), b.colour_arrays(), strict=True):
            np.testing.assert_array_equal(x, y)
        a.sweep(5)
        b.sweep(5)
        assert a.observables_int() == b.observables_int()
