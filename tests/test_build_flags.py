"""Flags of the device build that the first call of a process depends on."""

from __future__ import annotations

from pyising_b200 import build


def test_device_code_is_not_compressed():
    # nvcc compresses large modules by itself; unpacking one held up the first launch from it
    assert "--no-compress" in build.NVCC_FLAGS
    assert "arch=compute_100a,code=sm_100a" in build.ARCH
