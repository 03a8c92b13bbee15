"""The host arithmetic of the temporal tiles (csrc/tile_plan.h), compiled for the CPU."""

from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pyising_b200" / "csrc"

SHIM = r"""
#include "tile_plan.h"
extern "C" void cuts(long long halves, int depth, long long* out)
{
    const ising::TileCuts c(halves, depth);
    out[0] = c.launches;
    out[1] = c.base;
    out[2] = c.longer;
    out[3] = c.launches ? c.depth(0) : 0;
    out[4] = c.launches ? c.depth(c.launches - 1) : 0;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    d = tmp_path_factory.mktemp("tile_plan")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CSRC), "shim.cpp",
                    "-o", "shim.so"], cwd=d, check=True)
    return ctypes.CDLL(str(d / "shim.so"))


# up to more sweeps than any counter of 32 bits holds
@pytest.mark.parametrize("sweeps", [0, 1, 2, 3, 7, 70, 1000, 2**31 + 3, 5 * 10**9, 2**40 + 1])
@pytest.mark.parametrize("depth", [1, 2, 3, 5, 16])
def test_cuts_cover_the_run(plan, sweeps, depth):
    out = (ctypes.c_longlong * 5)()
    plan.cuts(ctypes.c_longlong(2 * sweeps), depth, out)
    launches, base, longer, first, last = out
    assert launches % 2 == 0 and 0 <= longer <= launches
    assert launches * base + longer == 2 * sweeps
    assert (first, last) == ((base + (longer > 0), base) if launches else (0, 0))
    if sweeps:
        assert 1 <= last <= first <= depth
        assert launches - 2 < 2 * sweeps / depth  # no more launches than the depth asks for
