"""The multi-column product on either side of the lines between its two kernels
(by element type, semiring, columns, skew and entries), against the oracle's
fold: values are halves, so every sum is exact whatever its grouping."""

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W

pytestmark = pytest.mark.gpu

CODES = {"plus_times": 0, "min_plus": 1, "lor_land": 5}


@pytest.fixture(scope="module")
def graphs():
    kept = {}

    def get(name, weights):
        if (name, weights) not in kept:
            kind, size = name.split()
            g = W.gnm(int(size) // 12, int(size), seed=3) if kind == "even" else W.rmat(int(size), seed=3)
            rng = np.random.default_rng(1)
            m = len(g.targets)
            w = {"none": None, "int": rng.integers(1, 9, m).astype(np.float64),
                 "half": rng.integers(1, 9, m) / 2}[weights]
            kept[name, weights] = (g, O.Graph.from_csr(g.id_space, g.offsets, g.targets, w),
                                   W.GraphVersion(g.offsets, g.targets, w))
        return kept[name, weights]

    return get


@pytest.mark.parametrize("graph,weights,semiring,dtype,widths", [
    ("even 60000", "half", "plus_times", np.float64, (2, 4, 6, 8, 16, 17, 32, 34, 64)),
    ("even 60000", "none", "plus_times", np.float64, (2, 8, 32, 40)),
    ("even 60000", "none", "plus_times", np.float32, (4, 8, 12, 16, 32, 44)),
    ("even 60000", "int", "min_plus", np.int64, (2, 4, 6, 16, 33, 36)),
    ("even 60000", "none", "min_plus", np.int64, (4, 8, 32)),
    ("even 60000", "none", "lor_land", np.uint8, (8, 16, 17, 32, 48)),
    ("even 1300000", "half", "min_plus", np.float64, (4, 8, 10, 32)),
    ("even 1300000", "none", "lor_land", np.uint8, (20,)),
    ("skew 15", "half", "plus_times", np.float64, (8, 32)),
    ("skew 16", "half", "plus_times", np.float64, (4, 6, 16, 24, 32)),
    ("skew 16", "half", "plus_times", np.float32, (2, 3, 4, 16, 21, 32)),
    ("skew 17", "none", "plus_times", np.float32, (16, 20, 32)),
    ("skew 17", "int", "min_plus", np.int64, (16, 18, 32)),
    ("skew 17", "none", "lor_land", np.uint8, (16, 17, 32)),
    ("skew 18", "half", "min_plus", np.float64, (8, 16, 32))])
def test_either_side_of_the_kernels_lines(graphs, graph, weights, semiring, dtype, widths):
    g, og, gv = graphs(graph, weights)
    n = g.id_space
    for width in widths:
        rng = np.random.default_rng(width)
        if dtype == np.uint8:
            x = (rng.random((n, width)) < 0.2).astype(np.uint8)
        elif dtype == np.int64:
            x = rng.integers(0, 1000, (n, width))
        else:
            x = (rng.integers(-8, 9, (n, width)) / 2).astype(dtype)
        mask = (rng.random(n) < 0.5).astype(np.uint8)
        for transpose in (False, True):
            y = np.full((n, width), 3, dtype)
            want = y.copy()
            assert O.product(og, CODES[semiring], x, want, transpose=transpose) == 0
            W.spmm(gv, W.Product(semiring, transpose=transpose), x, y)
            assert np.array_equal(y, want)
        y = np.full((n, width), 3, dtype)
        want = y.copy()
        assert O.product(og, CODES[semiring], x, want, mask=mask, mask_dtype=3) == 0
        W.spmm(gv, W.Product(semiring, mask=mask), x, y)
        assert np.array_equal(y, want)
