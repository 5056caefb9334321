"""The multi-column product at its widths' edges: each block of columns (2, 4,
8, 16 and 32, and what is left of one), rows that start on 16-byte boundaries
and rows that do not, rows about a batch, a tile and a piece, masks and
accumulators, against the oracle's fold."""

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W

pytestmark = pytest.mark.gpu

LENGTHS = [0, 0, 1, 7, 8, 9, 16, 17, 31, 63, 64, 65, 255, 256, 257, 513, 2100]
SEMIRINGS = {"plus_times": 0, "min_plus": 1, "lor_land": 5}


@pytest.fixture(scope="module")
def graph():
    rng = np.random.default_rng(8)
    n = 2501
    lengths = rng.poisson(5, n)
    lengths[rng.permutation(n)[:2 * len(LENGTHS)]] = LENGTHS * 2
    rows = [np.sort(rng.choice(n, k, replace=False)) for k in lengths]
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    targets = np.concatenate(rows).astype(np.uint32)
    w = rng.integers(1, 50, len(targets)).astype(np.float64)
    return n, lengths, O.Graph.from_csr(n, offsets, targets, w), W.GraphVersion(offsets, targets, w)


def operand(rng, dtype, shape):
    if dtype == np.uint8:
        return (rng.random(shape) < 0.3).astype(np.uint8)
    if dtype == np.int64:
        return rng.integers(0, 1000, shape)
    return (rng.random(shape) + 0.5).astype(dtype)


def same(got, want, dtype, semiring, lengths, transpose):
    if semiring != "plus_times" or dtype in (np.int64, np.uint8):
        assert np.array_equal(got, want)
        return
    # Positive terms, at most 2,100 a row: a reassociated sum is within that
    # many ulps of the fold's; forward rows of at most 256 fold in order.
    assert np.allclose(got, want, rtol=2100 * np.finfo(dtype).eps, atol=0)
    if not transpose:
        assert np.array_equal(got[lengths <= 256], want[lengths <= 256])


@pytest.mark.parametrize("width", [2, 3, 4, 5, 8, 9, 16, 17, 24, 31, 32, 33, 50, 64])
@pytest.mark.parametrize("semiring,dtype", [("plus_times", np.float64), ("plus_times", np.float32),
                                            ("min_plus", np.int64), ("plus_times", np.int64),
                                            ("lor_land", np.uint8)])
def test_every_column_of_every_width(graph, width, semiring, dtype):
    n, lengths, og, gv = graph
    rng = np.random.default_rng(width)
    for transpose in (False, True):
        x, y = operand(rng, dtype, (n, width)), operand(rng, dtype, (n, width))
        want = y.copy()
        assert O.product(og, SEMIRINGS[semiring], x, want, transpose=transpose) == 0
        W.spmm(gv, W.Product(semiring, transpose=transpose), x, y)
        same(y, want, dtype, semiring, lengths, transpose)


@pytest.mark.parametrize("width", [4, 8])
def test_rows_off_their_boundary(graph, width):
    # x and y one element past a 16-byte boundary: the element-wise variant.
    torch = pytest.importorskip("torch")
    n, lengths, og, gv = graph
    rng = np.random.default_rng(2)
    x = operand(rng, np.float32, (n, width))
    want = np.zeros_like(x)
    assert O.product(og, 0, x, want) == 0
    for shift in (0, 1):
        xd = torch.zeros(n * width + 1, dtype=torch.float32, device="cuda")[shift:shift + n * width]
        yd = torch.zeros_like(torch.zeros(n * width + 1, dtype=torch.float32, device="cuda"))
        yd = yd[shift:shift + n * width].view(n, width)
        xd.copy_(torch.as_tensor(x.reshape(-1)))
        torch.cuda.synchronize()
        W.spmm(gv, W.Product("plus_times"), xd.view(n, width), yd)
        same(yd.cpu().numpy(), want, np.float32, "plus_times", lengths, False)


@pytest.mark.parametrize("accumulate", [None, "plus", "min"])
@pytest.mark.parametrize("replace", [False, True])
def test_masks_and_accumulators(graph, accumulate, replace):
    n, lengths, og, gv = graph
    rng = np.random.default_rng(3)
    x, y = operand(rng, np.int64, (n, 20)), operand(rng, np.int64, (n, 20))
    mask = (rng.random(n) < 0.5).astype(np.float64)
    want = y.copy()
    code = -1 if accumulate is None else W.api.A.BINARY_OPS.index(accumulate)
    assert O.product(og, 1, x, want, mask=mask, mask_dtype=1, replace=replace, accumulate=code) == 0
    W.spmm(gv, W.Product("min_plus", mask=mask, replace=replace, accumulate=accumulate), x, y)
    assert np.array_equal(y, want)
