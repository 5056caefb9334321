"""The 32-bit batched min-plus on graphs on either side of the line between
its two iteration kernels (the share of long rows' pieces, the number of
units, the pass's columns), against the oracle's search per source."""

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,weights", [(12, "int"), (17, "int"), (17, "none")])
@pytest.mark.parametrize("width", [31, 64, 100])
def test_minplus_rows_and_tiles(scale, weights, width):
    g = W.rmat(scale, seed=6)
    w = W.edge_weights(g, "int") if weights == "int" else None
    og = O.Graph.from_csr(g.id_space, g.offsets, g.targets, w)
    gv = W.GraphVersion(g.offsets, g.targets, w)
    rng = np.random.default_rng(width)
    src = rng.integers(0, g.id_space, width).astype(np.uint64)
    src[1] = src[0]
    hops = rng.integers(0, 17, width).astype(np.uint32)
    d, it = W.minplus_batched(gv, src, hops)
    some = np.unique(np.concatenate([[0, 1, width - 1], rng.integers(0, width, 5)]))
    do, ito = O.sssp_i64(og, src[some], hops[some])
    assert np.array_equal(d[some], do)
    assert np.array_equal(it[some], ito)
