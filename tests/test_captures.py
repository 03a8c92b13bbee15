"""Sweeps while CUDA graphs are captured: on another stream (a capture that has nothing to do with
the lattice), and on the lattice's own stream, cold and after a sweep outside the capture, with
more sweeps than a replayed chunk of the library's own graphs holds."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BETA_C_2D = 0.44068679350977147


def pair(variant, shape):
    from pyising_b200.backend import B200Int8, B200MultiSpin

    cls = B200MultiSpin if variant == "msc" else B200Int8
    return [cls(shape, BETA_C_2D, seed=3, init="philox") for _ in range(2)]


def assert_same(a, b):
    for x, y in zip(a.colour_arrays(), b.colour_arrays(), strict=True):
        np.testing.assert_array_equal(x, y)


# (the last one's tiles need more shared memory than a kernel has by default)
@pytest.mark.parametrize("variant,shape", [("msc", (64, 256)), ("int8", (62, 72)),
                                           ("int8", (64, 64)), ("int8", (1600, 2488))], ids=str)
def test_first_sweep_while_another_stream_is_captured(variant, shape):
    import torch

    a, b = pair(variant, shape)
    a.synchronize()
    x = torch.zeros(4, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # the global mode: no waiting for streams from this thread
        x += 1
        a.sweep(3)
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 4
    b.sweep(3)
    assert_same(a, b)


# 2D lattices with and without tiles (one is far wider than high) and 3D
@pytest.mark.parametrize("variant,shape", [("msc", (64, 256)), ("int8", (64, 64)),
                                           ("int8", (62, 72)), ("msc", (2, 65536)),
                                           ("int8", (8, 16, 24))], ids=str)
@pytest.mark.parametrize("sweeps", [1, 64, 70])
@pytest.mark.parametrize("warm", [False, True])
def test_sweeps_into_a_captured_stream(variant, shape, sweeps, warm):
    import torch

    a, b = pair(variant, shape)
    if warm:
        a.sweep(70)
        b.sweep(70)
    a.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        a.set_stream(torch.cuda.current_stream().cuda_stream)
        a.sweep(sweeps)
    a.set_stream(None)
    graph.replay()
    torch.cuda.synchronize()
    b.sweep(sweeps)
    assert_same(a, b)
    a.sweep(70)  # the handle's own graphs still work afterwards
    b.sweep(70)
    assert_same(a, b)
