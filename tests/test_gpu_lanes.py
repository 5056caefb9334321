"""The products over the lane-major copy at the edges of its layout: rows
about a slice's length, about a row of eight lanes, about a piece and about a
unit's pieces, empty rows, nodes gathered often enough for a slot, in both
orientations, against the oracle's fold."""

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 3, 4, 5, 31, 32, 33, 39, 40, 41, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511,
           512, 513, 2047, 2048, 2049, 2305, 4100]


def edge_graph(n, weights, hubs, seed):
    """Rows of the LENGTHS (then of about 8 entries), some over 50 hubs."""
    rng = np.random.default_rng(seed)
    lengths = rng.poisson(8, n)
    lengths[rng.permutation(n)[:3 * len(LENGTHS)]] = LENGTHS * 3
    rows = []
    for length in lengths:
        t = rng.choice(n, length, replace=False)
        if hubs and length > 1:
            t = np.unique(np.concatenate([t[: length // 2], rng.choice(50, min(length // 2, 40))]))
        rows.append(np.sort(t))
    offsets = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    targets = np.concatenate(rows).astype(np.uint32)
    w = {"none": None, "int": rng.integers(1, 50, len(targets)).astype(np.float64),
         "float": rng.random(len(targets)) + 0.5}[weights]
    return offsets, targets, w


def check(og, gv, semiring, code, x, transpose, lengths):
    y = np.zeros_like(x)
    W.spmv(gv, W.Product(semiring, transpose=transpose), x, y)
    want = np.zeros_like(x)
    assert O.product(og, code, x, want, transpose=transpose) == 0
    if x.dtype == np.float64 and semiring == "plus_times":
        # Positive terms: a reassociated sum is within (terms) ulps of the
        # fold's; rows of at most 256 entries fold in order.
        assert np.allclose(y, want, rtol=4200 * 2.3e-16, atol=0)
        assert np.array_equal(y[lengths <= 256], want[lengths <= 256])
    else:
        assert np.array_equal(y, want)


@pytest.mark.parametrize("weights", ["none", "int", "float"])
@pytest.mark.parametrize("hubs", [False, True])
def test_products_at_the_layouts_edges(weights, hubs):
    offsets, targets, w = edge_graph(6007, weights, hubs, 3)
    n = len(offsets) - 1
    og = O.Graph.from_csr(n, offsets, targets, w)
    gv = W.GraphVersion(offsets, targets, w)
    rng = np.random.default_rng(5)
    out = np.diff(offsets).astype(np.int64)
    into = np.bincount(targets, minlength=n)
    if hubs:
        assert (into >= 296).sum() >= 50
    for transpose, lengths in ((False, out), (True, into)):
        check(og, gv, "plus_times", 0, rng.random(n), transpose, lengths)
        x = rng.integers(0, 1000, n)
        x[rng.random(n) < 0.5] = np.iinfo(np.int64).max
        check(og, gv, "min_plus", 1, x, transpose, lengths)
        check(og, gv, "plus_times", 0, rng.integers(-9, 9, n), transpose, lengths)
        check(og, gv, "lor_land", 5, (rng.random(n) < 0.1).astype(np.uint8), transpose, lengths)


def test_products_over_longer_slices():
    # Enough entries for slices of more than 32 steps (lanes.cu), lengths
    # about the 64 they may then have.
    g = W.gnm(300000, 300000 * 60, seed=4)
    og = O.Graph.from_csr(g.id_space, g.offsets, g.targets)
    gv = g.upload()
    rng = np.random.default_rng(6)
    lengths = np.bincount(g.targets, minlength=g.id_space)
    assert lengths.min() < 64 < lengths.max()
    check(og, gv, "plus_times", 0, rng.random(g.id_space), True, lengths)
    check(og, gv, "min_plus", 1, rng.integers(0, 1000, g.id_space), True, lengths)


def test_pagerank_is_the_same_from_run_to_run():
    # Its two sums are added in a fixed order, whichever warp finishes a row.
    offsets, targets, w = edge_graph(6007, "float", True, 9)
    gv = W.GraphVersion(offsets, targets, w)
    first = W.pagerank(gv, None, W.PageRank(0.85, 1e-10, 100))
    for _ in range(5):
        again = W.pagerank(gv, None, W.PageRank(0.85, 1e-10, 100))
        assert again.iterations == first.iterations
        assert np.array_equal(again.values, first.values)
