"""PageRank on either side of the sizes between which it turns from the
row-split schedule to the lane-major copy, with long rows and without: ranks
and iterations against the oracle, the same bits from run to run (its sums are
added in a fixed order on both) and from wc_pagerank_noalloc."""

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph,weighted", [
    ("rmat 10", False), ("rmat 13", True), ("rmat 16", False), ("rmat 16", True),
    ("rmat 17", False), ("rmat 17", True), ("rmat 18", False),
    ("gnm 262000", False), ("gnm 262300", False), ("gnm 262300", True), ("gnm 7", False)])
def test_pagerank_on_either_side_of_the_line(graph, weighted):
    kind, size = graph.split()
    if kind == "rmat":
        g = W.rmat(int(size), seed=3)
    else:
        g = W.gnm(max(3, int(size) // 13), int(size), seed=3)
    w = W.edge_weights(g, "uniform") if weighted else None
    og = O.Graph.from_csr(g.id_space, g.offsets, g.targets, w)
    gv = W.GraphVersion(g.offsets, g.targets, w)
    seed = np.random.default_rng(2).random(g.id_space)
    for tomb, s in ((None, None), (O.tombstone_words(g.id_space, [0, 2]), seed)):
        ranks, its, _, _ = O.pagerank(og, 0.85, 1e-10, 100, tombstones=tomb, seed=s)
        opts = W.PageRank(0.85, 1e-10, 100, seed=s)
        first = W.pagerank(gv, tomb, opts)
        assert first.iterations == its
        assert np.abs(first.values - ranks).sum() / np.abs(ranks).sum() <= 1e-12
        for _ in range(3):
            again = W.pagerank(gv, tomb, opts)
            assert again.iterations == its and np.array_equal(again.values, first.values)
    first = W.pagerank(gv, None, W.PageRank(0.85, 1e-10, 100))
    again = W.pagerank_noalloc(gv, None, W.PageRank(0.85, 1e-10, 100))
    assert again.iterations == first.iterations and np.array_equal(again.values, first.values)
