"""The 32-column pull and the level search at the row lengths where they
change what they do: about a gather group, the rows emitted together, a tile
and a piece; about the entries a lane scans alone, a warp's batch of a push
and the long-row push."""

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W

pytestmark = pytest.mark.gpu

LENGTHS = [0, 0, 1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 127, 128, 129, 240, 255, 256, 257, 272, 511,
           512, 513, 700]


def graph(n, weighted, seed):
    """Both orientations' rows about LENGTHS: a random half of the rows have
    them, and the targets of the others are skewed to the same lengths."""
    rng = np.random.default_rng(seed)
    lengths = rng.poisson(3, n)
    lengths[rng.permutation(n)[:4 * len(LENGTHS)]] = LENGTHS * 4
    popular = np.repeat(rng.permutation(n)[:2 * len(LENGTHS)], np.array(LENGTHS * 2) // 3 + 1)
    pairs = [np.stack([np.full(k, i), rng.choice(n, k, replace=False)], 1)
             for i, k in enumerate(lengths)]
    pairs.append(np.stack([rng.integers(0, n, len(popular)), popular], 1))
    pairs = np.unique(np.concatenate(pairs), axis=0)
    pairs = pairs[pairs[:, 0] != pairs[:, 1]]
    offsets = np.searchsorted(pairs[:, 0], np.arange(n + 1)).astype(np.uint64)
    targets = pairs[:, 1].astype(np.uint32)
    return offsets, targets, rng.random(len(targets)) + 0.1 if weighted else None


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("sets", [1, 31, 40])
def test_batched_pagerank_at_row_edges(weighted, sets):
    offsets, targets, w = graph(1501, weighted, 2)
    n = len(offsets) - 1
    og, gv = O.Graph.from_csr(n, offsets, targets, w), W.GraphVersion(offsets, targets, w)
    rng = np.random.default_rng(4)
    nodes = [rng.choice(n, int(k), replace=False) for k in rng.integers(1, 20, sets)]
    ranks, its = W.ppr_batched(gv, nodes, W.PageRank(0.85, 1e-9, 60))
    for q in range(sets):
        seed = np.zeros(n)
        seed[nodes[q]] = 1.0
        want, it, _, _ = O.pagerank(og, 0.85, 1e-9, 60, seed=seed)
        assert its[q] == it
        assert np.abs(ranks[q] - want).sum() <= 1e-12 * want.sum()


@pytest.mark.parametrize("losses", [1, 33])
def test_adjoint_at_row_edges(losses):
    offsets, targets, w = graph(1501, True, 3)
    n = len(offsets) - 1
    og, gv = O.Graph.from_csr(n, offsets, targets, w), W.GraphVersion(offsets, targets, w)
    rng = np.random.default_rng(5)
    nodes = [rng.choice(n, 20, replace=False) for _ in range(losses)]
    grad, ranks, _ = W.pagerank_adjoint(gv, nodes, W.PageRank(0.85, None, 60), adjoint_tol=1e-14)
    want, ro, _ = O.pagerank_adjoint(og, nodes, 0.85, None, 60, 1e-14)
    # λ_j - S_i cancels: errors are relative to the largest gradient.
    assert np.abs(grad - want).max() <= 1e-11 * np.abs(want).max()
    assert np.abs(ranks - ro).sum() <= 1e-12 * ro.sum()


@pytest.mark.parametrize("direction", ["out", "in", "both"])
def test_bfs_at_row_edges(direction):
    offsets, targets, _ = graph(6001, False, 7)
    n = len(offsets) - 1
    og, gv = O.Graph.from_csr(n, offsets, targets), W.GraphVersion(offsets, targets)
    code = {"out": 0, "in": 1, "both": 2}[direction]
    longest = int(np.argmax(np.diff(offsets.astype(np.int64))))
    for start in (0, 17, longest):
        for depth in (None, 2):
            got = W.bfs(gv, [start], limits=W.Limits(depth, None), direction=direction)
            want, stats = O.bfs(og, [start], code, depth)
            assert [(v.node, v.depth, v.via) for v in got.result] == want
            assert got.stats.edges_traversed == stats["edges_traversed"]
            reach = W.reachable_set(gv, [start], depth, direction)
            nodes, rstats = O.reachable_set(og, [start], code, depth)
            assert reach.result == nodes
            assert reach.stats.edges_traversed == rstats["edges_traversed"]
