"""Which lattices the automatic schedule runs on temporal tiles, told by the device memory that the
handle reports: tiles hold a second pair of colour arrays."""

from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

BETA_C_2D = 0.44068679350977147


def second_pair(variant, shape, schedule="auto", knobs=None):
    """Whether a swept lattice holds a second pair of colour arrays."""
    from pyising_b200 import autotune
    from pyising_b200.backend import B200Int8, B200MultiSpin

    cls = B200MultiSpin if variant == "msc" else B200Int8
    sim = cls(shape, BETA_C_2D, seed=3, init="cold")
    sim.set_schedule(schedule)
    if knobs:
        autotune.apply(sim, knobs)
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


# wide, low lattices: few bands of rows for the SMs, and most of a band's work is its halo
@pytest.mark.parametrize("variant,shape,tiles", [
    ("int8", (1024, 1024), True), ("int8", (1500, 2488), True), ("msc", (1152, 1152), True),
    ("msc", (4096, 4096), True), ("int8", (64, 16384), False), ("int8", (256, 8192), False),
    ("msc", (64, 65536), False), ("msc", (128, 32768), False), ("msc", (6000, 5248), False),
], ids=str)
def test_automatic_schedule_takes_tiles_where_they_are_faster(variant, shape, tiles):
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the choice depends on the number of SMs")
    assert second_pair(variant, shape) == tiles


def test_launch_knobs_set_by_hand_select_the_half_sweeps_they_belong_to():
    shape = (1600, 1600)  # above 512K sites per colour
    assert second_pair("int8", shape)
    for name, default, value in [("band", 0, 2), ("chunk_width", 16, 4)]:
        assert second_pair("int8", shape, knobs={name: default})
        assert not second_pair("int8", shape, knobs={name: value})
    for name, default, value in [("msc_kernel", 0, 1), ("msc_waves", 1, 2)]:
        assert second_pair("msc", (256, 1024), knobs={name: default})
        assert not second_pair("msc", (256, 1024), knobs={name: value})
