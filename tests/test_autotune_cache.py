"""Cache entries of the autotuner belong to the kernels they were measured with, and every 2D shape is
tried on the temporal tiles."""

from __future__ import annotations

import json

import pytest

from pyising_b200 import autotune


def test_entries_of_other_kernels_are_not_applied(tmp_path):
    path = tmp_path / "tune.json"
    cfg = {"msc_kernel": 2, "msc_waves": 2, "schedule": "launches"}
    # as an earlier version wrote it, and one of a later version
    path.write_text(json.dumps({"a": {"config": cfg, "flips_per_ns": 1.0},
                                "b": {"config": cfg, "schedules": autotune.SCHEDULES + 1}}))
    assert autotune.lookup("a", path) is None
    assert autotune.lookup("b", path) is None
    autotune.save_entry("a", {"config": cfg}, path)
    assert autotune.lookup("a", path) == cfg
    assert set(json.loads(path.read_text())) == {"a", "b"}


@pytest.mark.parametrize("variant,shape,tiles", [
    ("int8", (64, 64), True), ("int8", (62, 72), True), ("int8", (24, 1032), True),
    ("int8", (4096, 4096), True), ("msc", (128, 256), True), ("msc", (6144, 6144), True),
    ("int8", (16, 16, 32), False)], ids=str)
def test_every_2d_shape_is_tried_on_tiles(variant, shape, tiles):
    space = autotune.search_space(variant, shape)
    assert ("temporal" in space["schedule"]) == tiles
    assert space["schedule"][0] == "auto"


@pytest.mark.gpu
def test_a_stale_entry_leaves_a_new_simulation_at_its_defaults(tmp_path, monkeypatch):
    from pyising_b200.backend import B200MultiSpin

    path = tmp_path / "tune.json"
    monkeypatch.setenv("PYISING_B200_TUNE_CACHE", str(path))
    monkeypatch.delenv("PYISING_B200_AUTOTUNE", raising=False)
    key = autotune.key(autotune.device_name(0), "msc", "metropolis", (128, 256))
    path.write_text(json.dumps({key: {"config": {"msc_kernel": 1, "msc_waves": 4}}}))
    sim = B200MultiSpin((128, 256), 0.44, seed=1, init="cold")
    cur = autotune.current(sim)
    assert (cur["msc_kernel"], cur["msc_waves"]) == (0, 1)
