"""The products on either side of the sizes between which they turn from the
row-split schedule to the lane-major copy, over even and skewed graphs with rows
at the edges of the copy's layout (about a slice's length, a row of eight lanes,
a piece, a unit's pieces, empty), in both orientations, against the oracle's
fold; a row of at most 256 entries bit for bit."""

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W

pytestmark = pytest.mark.gpu

SHORT = [0, 1, 3, 4, 5, 31, 32, 33, 39, 40, 41, 63, 64, 65, 127, 128, 129, 255, 256]
LONG = [257, 511, 512, 513, 2047, 2048, 2049, 2305, 4100]


def edge_graph(entries, mean, skewed, seed):
    """About `entries` entries in rows of Poisson(mean), some of the edge
    lengths; every row a run of distinct targets, into all nodes alike or, in
    half of a skewed graph's rows, also into one of 64 hubs."""
    rng = np.random.default_rng(seed)
    n = entries // mean
    lengths = rng.poisson(mean, n)
    edges = (SHORT + LONG if skewed else SHORT) * 3
    lengths[rng.permutation(n)[:len(edges)]] = edges
    src = np.repeat(np.arange(n), lengths)
    k = np.arange(len(src)) - np.repeat(np.cumsum(lengths) - lengths, lengths)
    start = rng.integers(0, n, n)
    dst = (start[src] + k * 7) % n
    if skewed:
        to_hub = (k == 0) & (src % 2 == 0) & (lengths[src] > 1)
        dst[to_hub] = rng.integers(0, 64, to_hub.sum())
    key = np.unique(src * n + dst)
    src, dst = key // n, key % n
    offsets = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint64)
    return n, offsets, dst.astype(np.uint32)


def check(og, gv, semiring, code, x, transpose, lengths):
    y = np.zeros_like(x)
    W.spmv(gv, W.Product(semiring, transpose=transpose), x, y)
    want = np.zeros_like(x)
    assert O.product(og, code, x, want, transpose=transpose) == 0
    if x.dtype.kind == "f" and semiring == "plus_times":
        # Positive terms: a reassociated sum is within (terms) ulps of the
        # fold's; rows of at most 256 entries fold in order.
        assert np.allclose(y, want, rtol=float(lengths.max()) * np.finfo(x.dtype).eps, atol=0)
        assert np.array_equal(y[lengths <= 256], want[lengths <= 256])
    else:
        assert np.array_equal(y, want)


LINE = 1 << 17  # the lines in units of this


@pytest.mark.parametrize("skewed,weights,mean,entries", [
    (False, "float", 11, 3 * LINE - 40000), (False, "float", 11, 3 * LINE + 40000),
    (False, "none", 11, 6 * LINE - 40000), (False, "none", 11, 6 * LINE + 40000),
    (False, "int", 11, 6 * LINE + 40000),
    (True, "float", 14, 7 * LINE - 60000), (True, "float", 14, 7 * LINE + 60000),
    (True, "float", 6, 8 * LINE - 60000), (True, "float", 6, 8 * LINE + 60000),
    (True, "none", 7, 12 * LINE - 60000), (True, "none", 7, 12 * LINE + 60000),
    (True, "int", 15, 18 * LINE - 60000), (True, "int", 15, 18 * LINE + 60000),
    (True, "none", 15, 24 * LINE - 90000), (True, "none", 15, 24 * LINE + 90000)])
def test_products_on_either_side_of_the_lines(skewed, weights, mean, entries):
    n, offsets, targets = edge_graph(entries, mean, skewed, 3)
    rng = np.random.default_rng(5)
    m = len(targets)
    w = {"none": None, "int": rng.integers(1, 50, m).astype(np.float64),
         "float": rng.random(m) + 0.5}[weights]
    og = O.Graph.from_csr(n, offsets, targets, w)
    gv = W.GraphVersion(offsets, targets, w)
    out = np.diff(offsets).astype(np.int64)
    into = np.bincount(targets, minlength=n)
    assert (into.max() > 256) == skewed and (out.max() > 256) == skewed
    for transpose, lengths in ((False, out), (True, into)):
        check(og, gv, "plus_times", 0, rng.random(n), transpose, lengths)
        check(og, gv, "plus_times", 0, rng.random(n).astype(np.float32), transpose, lengths)
        x = rng.integers(0, 1000, n)
        x[rng.random(n) < 0.5] = np.iinfo(np.int64).max
        check(og, gv, "min_plus", 1, x, transpose, lengths)
        check(og, gv, "plus_times", 0, rng.integers(-9, 9, n), transpose, lengths)
        check(og, gv, "lor_land", 5, (rng.random(n) < 0.1).astype(np.uint8), transpose, lengths)
