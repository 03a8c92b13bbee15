"""The host arithmetic of the temporal tiles (csrc/tile_plan.h) and of the packed lane walk
(csrc/lane_plan.h), and the bands of int8 half-sweeps (csrc/band_plan.h), compiled for the CPU."""

from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pyising_b200" / "csrc"

SHIM = r"""
#include "band_plan.h"
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
extern "C" long long lane_band(long long rows, long long nw, long long lanes, long long sms)
{
    return ising::lane_band(rows, nw, lanes, sms);
}
extern "C" int band(long long rows, int ly, int cpr, int sms)
{
    return ising::int8_default_band(rows, ly, cpr, sms);
}
extern "C" int limit(int ndim, int cpr) { return ising::int8_band_limit(ndim, cpr); }
extern "C" int plan(int msc, int ly, int units, int row_bytes, int sms, int every, int* shape,
                    double* us)
{
    const ising::TileRows r{msc != 0, ly, units, (size_t)row_bytes, sms};
    const ising::TileShape s = ising::tile_shape(r);
    shape[0] = s.band;
    shape[1] = s.depth;
    us[0] = s.depth > 0 ? ising::tile_half_us(r, s, s.depth) : 0.0;
    us[1] = ising::single_half_us(r);
    return ising::tiles_pay(r, every);
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


def choose(lib, variant, shape, sms=148, every=0):
    ly, lx = shape
    units = lx // 128 if variant == "msc" else -(-lx // 32)
    row_bytes = units * (8 if variant == "msc" else 16)
    out, us = (ctypes.c_int * 2)(), (ctypes.c_double * 2)()
    pays = lib.plan(int(variant == "msc"), ly, units, row_bytes, sms, every, out, us)
    band, depth = out
    assert band * sms >= ly and band >= 2
    assert 0 <= depth <= 16 and 2 * depth <= ly
    assert 2 * (band + 2 * depth) * row_bytes <= 200 * 1024 or depth == 0
    return bool(pays), tuple(us)


# the faster schedule as measured on a B200 (by more than a few percent), wide and low lattices
# among them: these have few bands, and a band's halo rows are recomputed
@pytest.mark.parametrize("variant,shape,tiles", [
    ("int8", (64, 64), True), ("int8", (1024, 1024), True), ("int8", (1500, 2488), True),
    ("int8", (3000, 3000), True), ("int8", (3500, 3584), True), ("int8", (64, 1024), True),
    ("int8", (128, 2048), True), ("int8", (512, 4096), True), ("int8", (65536, 64), True),
    ("int8", (8192, 1024), True), ("int8", (2, 32768), False), ("int8", (16, 4096), False),
    ("int8", (16, 32768), False), ("int8", (64, 4096), False), ("int8", (64, 16384), False),
    ("int8", (128, 16384), False), ("int8", (256, 8192), False), ("int8", (256, 32768), False),
    ("int8", (512, 8192), False), ("int8", (1024, 8192), False), ("int8", (2, 10**6), False),
    ("msc", (128, 128), True), ("msc", (1152, 1152), True), ("msc", (2048, 2048), True),
    ("msc", (3072, 3072), True), ("msc", (4096, 4096), True), ("msc", (4600, 4608), True),
    ("msc", (5000, 4992), True), ("msc", (16, 16384), True), ("msc", (64, 8192), True),
    ("msc", (128, 4096), True), ("msc", (2048, 8192), True), ("msc", (65536, 128), True),
    ("msc", (6000, 5248), False), ("msc", (2, 131072), False), ("msc", (16, 131072), False),
    ("msc", (64, 65536), False), ("msc", (128, 32768), False), ("msc", (256, 32768), False),
], ids=str)
def test_tiles_where_they_are_faster(plan, variant, shape, tiles):
    pays, us = choose(plan, variant, shape)
    assert pays == tiles, us
    if tiles:  # a graph per measurement costs single half-sweeps more
        for every in (1, 2, 10, 1000):
            assert choose(plan, variant, shape, every=every)[0]


@pytest.mark.parametrize("variant,shape,every,tiles", [
    ("int8", (256, 8192), 1, True), ("int8", (256, 8192), 10, False), ("int8", (64, 4096), 1, True),
    ("int8", (256, 8192), 10**9, False), ("int8", (16, 4096), 2, True), ("msc", (64, 65536), 2, False),
    ("msc", (128, 32768), 10, False), ("int8", (16, 32768), 1, False)], ids=str)
def test_measured_sweeps_take_tiles_where_they_are_faster(plan, variant, shape, every, tiles):
    assert choose(plan, variant, shape, every=every)[0] == tiles


LANES = 148 * 512


@pytest.mark.parametrize("nw", [1, 2, 3, 5, 31, 32, 49, 128, 1000, 40000, 80000])
@pytest.mark.parametrize("fill", [0.3, 0.51, 1.0, 1.9, 2.03, 3.0, 3.3, 3.99, 4.05, 5.9, 8.1, 14.2,
                                  19.99, 20.0, 40.0, 100.0])
def test_lane_bands_fit_the_resident_lanes(plan, nw, fill):
    plan.lane_band.restype = ctypes.c_longlong
    rows = max(2, int(fill * LANES / nw) // 2 * 2)
    args = [ctypes.c_longlong(x) for x in (rows, nw, LANES, 148)]
    band = plan.lane_band(*args)
    words = rows * nw
    if words < 256 * 148:
        assert band == 0
        return
    assert band % 2 == 0 and 0 <= band <= rows
    if nw <= 128 and not 2 < words / LANES <= 4:
        assert band > 0  # word ranges only where the walk would leave many lanes idle
    if band > 2:
        assert -(-rows // band) * nw <= LANES  # one wave: no block left over
        assert nw > 1 or band % 16
        assert words >= 0.4 * LANES * band  # and not mostly idle


@pytest.mark.parametrize("shape,band", [((505172, 384), 22), ((2402, 8192), 0), ((3552, 8192), 0), ((58726, 512), 4), ((302, 128000), 0),
                                        ((4616, 8192), 4), ((4794, 8192), 6), ((650, 8192), 2),
                                        ((4600, 4608), 0), ((6000, 5248), 4), ((16384, 16384), 28),
                                        ((1152, 1152), 0)], ids=str)
def test_lane_bands(plan, shape, band):
    plan.lane_band.restype = ctypes.c_longlong
    args = [ctypes.c_longlong(x) for x in (shape[0], shape[1] // 128, LANES, 148)]
    assert plan.lane_band(*args) == band


# the measured best heights (or, in brackets, those within a few percent of it)
@pytest.mark.parametrize("shape,best", [
    ((16384, 16384), [16]), ((12000, 12000), [8, 16]), ((9000, 9000), [4, 8]),
    ((8192, 8192), [4, 8]), ((7000, 7000), [4]), ((5000, 5000), [2]), ((4096, 4096), [2]),
    ((2000000, 32), [4]), ((256, 256, 256), [2]), ((300, 300, 304), [2]), ((400, 400, 416), [4]),
    ((448, 448, 448), [4]), ((512, 512, 512), [8, 16]), ((640, 640, 640), [16]),
    ((1000, 1000, 24), [2]), ((2000, 2000, 32), [2]), ((100, 1000, 1000), [4]), ((64, 64), [1]),
], ids=str)
def test_default_band(plan, shape, best):
    rows = 1
    for extent in shape[:-1]:
        rows *= extent
    got = plan.band(ctypes.c_longlong(rows), shape[-2], -(-shape[-1] // 32), 148)
    assert got in best


@pytest.mark.parametrize("ndim,cpr,most", [(2, 1, 4), (2, 2, 64), (2, 512, 64), (3, 1, 2), (3, 2, 4),
                                           (3, 15, 4), (3, 16, 64)])
def test_band_limit_of_batches(plan, ndim, cpr, most):
    assert plan.limit(ndim, cpr) == most
