"""Host threads that drive lattices of different tile sizes at the same time: the shared-memory
limit of a kernel belongs to the function, so one thread's launch must not change another's."""

from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA_C_2D = 0.44068679350977147
CALLS, SWEEPS = 600, 20


def drive(sim, calls, errors):
    try:
        for _ in range(calls):
            sim.sweep(SWEEPS)
        sim.synchronize()
    except Exception as exc:  # noqa: BLE001 - reported by the test
        errors.append(exc)


def test_threads_with_tiles_of_different_sizes():
    from pyising_b200.backend import B200Int8

    # tiles of 69 and 39 KiB (on 148 SMs) of the same kernel
    shapes = [(600, 6400), (600, 3584)]
    sims = [B200Int8(shape, BETA_C_2D, seed=7, init="philox") for shape in shapes]
    alone = [B200Int8(shape, BETA_C_2D, seed=7, init="philox") for shape in shapes]
    for sim in sims + alone:
        sim.set_schedule("temporal")
    errors = []
    threads = [threading.Thread(target=drive, args=(sim, CALLS, errors)) for sim in sims]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for sim, ref in zip(sims, alone, strict=True):
        drive(ref, CALLS, errors)
        np.testing.assert_array_equal(sim.get_lattice(), ref.get_lattice())
    assert not errors
