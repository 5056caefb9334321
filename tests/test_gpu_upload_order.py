"""The batched search's row masks are made on the device from units copied to it
just before: on fresh versions of graphs with many units every search sees all
rows, upload after upload."""

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", ["even", "skewed"])
def test_searches_on_fresh_versions_see_every_row(graph):
    g = W.gnm(6007, 900000, seed=2) if graph == "even" else W.rmat(17, seed=2)
    og = O.Graph.from_csr(g.id_space, g.offsets, g.targets)
    sources, caps = [0, 5, 77], [3, 4, 8]
    want, edges = O.bfs_depths(og, sources, caps)
    for _ in range(12):
        depth, traversed = W.bfs_batched(g.upload(), sources, caps)
        assert np.array_equal(depth, want) and np.array_equal(traversed, edges)
