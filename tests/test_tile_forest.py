"""The bounded union-find walks of a cluster update's tiles (csrc/tile_forest.h), on the CPU: a cycle,
which no correct union-find makes, must end a root walk by its step budget."""

from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pyising_b200" / "csrc"

SHIM = r"""
#include "tile_forest.h"
extern "C" int limit() { return ising::kTileSteps; }
extern "C" int find(int* lab, int x, int* left)
{
    return ising::tile_find(lab, x, *left);
}
extern "C" int root(int* lab, int x, int* left)
{
    return ising::tile_root(lab, x, *left);
}
"""


@pytest.fixture(scope="module")
def walks(tmp_path_factory):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    d = tmp_path_factory.mktemp("tile_forest")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CSRC), "shim.cpp",
                    "-o", "shim.so"], cwd=d, check=True)
    return ctypes.CDLL(str(d / "shim.so"))


@pytest.mark.parametrize("walk", ["find", "root"])
def test_roots_of_a_forest(walks, walk):
    parents = [0, 0, 1, 2, 3, 5, 5, 6]
    for x, want in enumerate([0, 0, 0, 0, 0, 5, 5, 5]):
        lab = (ctypes.c_int * 8)(*parents)
        left = ctypes.c_int(walks.limit())
        assert getattr(walks, walk)(lab, x, ctypes.byref(left)) == want
        assert left.value > walks.limit() - 8


@pytest.mark.parametrize("walk", ["find", "root"])
def test_the_longest_chain_of_a_tile_fits_the_budget(walks, walk):
    n = 2 * 6144  # both colours of the largest tile, every node the child of the one before it
    lab = (ctypes.c_int * n)(*[max(i - 1, 0) for i in range(n)])
    left = ctypes.c_int(walks.limit())
    assert getattr(walks, walk)(lab, n - 1, ctypes.byref(left)) == 0
    assert left.value > walks.limit() // 2


def test_a_cycle_spends_the_budget(walks):
    # (the path halving of a find cuts a cycle itself; a root walk writes nothing)
    lab = (ctypes.c_int * 4)(1, 2, 3, 0)
    left = ctypes.c_int(walks.limit())
    walks.root(lab, 0, ctypes.byref(left))
    assert left.value < 0
