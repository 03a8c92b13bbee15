"""Which lattices the automatic schedule runs on temporal tiles, told by the device memory that the
handle reports: tiles hold a second pair of colour arrays."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

BETA_C_2D = 0.44068679350977147


def second_pair(variant, shape, schedule="auto"):
    """Whether a swept lattice holds a second pair of colour arrays."""
    from pyising_b200.backend import B200Int8, B200MultiSpin

    cls = B200MultiSpin if variant == "msc" else B200Int8
    sim = cls(shape, BETA_C_2D, seed=3, init="cold")
    sim.set_schedule(schedule)
    before = sim.device_bytes()
    sim.sweep(3)
    more = sim.device_bytes() - before
    pair = sum(c.nbytes for c in sim.colour_arrays())
    if variant == "int8":  # rows are padded to 16 bytes on the device
        pair = pair // (shape[1] // 2) * -(-shape[1] // 32) * 16
    assert more in (0, pair)
    return more == pair


@pytest.mark.parametrize("variant,shape", [("int8", (64, 64)), ("int8", (62, 72)),
                                           ("msc", (64, 256))], ids=str)
def test_device_bytes_count_the_second_pair(variant, shape):
    assert second_pair(variant, shape, "temporal")
    assert not second_pair(variant, shape, "launches")
