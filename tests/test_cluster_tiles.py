"""Exact labels of cluster updates where tiles meet the lattice's own shape: rows that several lanes of
a warp share with other rows, tiles as wide or as high as the lattice (the bonds around it stay in
the tile), several full tiles with a ragged last one, and extents of two, where both vertical bonds
of a site join the same pair."""

from __future__ import annotations

import numpy as np
import pytest
from test_cluster import components_min, neighbours, set_cluster_tile

pytestmark = pytest.mark.gpu

SHAPES = [(2, 8), (4, 8), (30, 8), (520, 8), (34, 24), (18, 40), (2, 64), (20, 64), (70, 16), (40, 144),
          (34, 136), (2, 72), (2, 2, 8), (2, 6, 16), (4, 2, 24), (6, 20, 72), (2, 36, 64)]


@pytest.mark.parametrize("tile", [0, 32, 1000, 6144])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_labels_at_the_edges_of_tiles(oracle_mod, shape, tile):
    from pyising_b200.backend import B200Int8

    for beta in ((0.25, 0.44, 0.9) if len(shape) == 2 else (0.12, 0.25, 0.6)):
        sim = B200Int8(shape, beta, seed=77, init=oracle_mod.random_lattice(shape, 5))
        set_cluster_tile(sim, tile)
        sim.sweep(5)
        c0, c1 = sim.colour_arrays()
        labels, bonds = sim.cluster_labels(step=9)
        rows, lh = c0.shape
        flat, edges = c1.reshape(-1), []
        for r in range(rows):
            for j in range(lh):
                for k, m in enumerate(neighbours(shape, r, j)):
                    if bonds[r, j] >> k & 1:
                        assert c0[r, j] == flat[m]
                        edges.append((r * lh + j, rows * lh + m))
        want = components_min(2 * rows * lh, edges)
        np.testing.assert_array_equal(labels.reshape(-1), want)


@pytest.mark.parametrize("shape", [(520, 8), (36, 24), (40, 144), (4, 36, 72)], ids=str)
def test_updates_are_those_of_one_union_find(shape):
    """The flips too: tiles against the single union-find in global memory (tile knob 1)."""
    from pyising_b200.backend import B200Int8

    out = []
    for tile in (1, 0, 32, 6144):
        sim = B200Int8(shape, 0.44 if len(shape) == 2 else 0.22, seed=9, init="hot")
        set_cluster_tile(sim, tile)
        out.append((sim.cluster_sweep(6, measure=True), sim.get_lattice()))
    for series, lattice in out[1:]:
        np.testing.assert_array_equal(series, out[0][0])
        np.testing.assert_array_equal(lattice, out[0][1])


@pytest.mark.parametrize("shape", [(48, 48, 48), (4, 40, 1024)], ids=str)
def test_unions_of_several_planes_bonds_per_thread(shape):
    """Ordered 3D lattices of a size at which a thread takes four z bonds."""
    from pyising_b200.backend import B200Int8

    out = []
    for tile in (1, 0, 1000):
        sim = B200Int8(shape, 0.3, seed=9, init="hot")
        set_cluster_tile(sim, tile)
        out.append((sim.cluster_sweep(4, measure=True), sim.cluster_labels(step=2)))
    for series, (labels, bonds) in out[1:]:
        np.testing.assert_array_equal(series, out[0][0])
        np.testing.assert_array_equal(labels, out[0][1][0])
        np.testing.assert_array_equal(bonds, out[0][1][1])
