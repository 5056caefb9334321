"""A version's lane-major copies make room for what a budget could hold without
them: a second upload and a search's scratch are served, the version that gave
its copies back answers as before, and one whose walk a caller has captured in
a graph of its own keeps them."""

import numpy as np
import pytest

import pg_warren_b200 as W

pytestmark = pytest.mark.gpu


def upload(g, budget):
    rev = W.api.host_reverse(g.offsets, g.targets)
    return W.GraphVersion(g.offsets, g.targets, reverse=rev, budget=budget)


def products(gv):
    x = np.random.default_rng(1).random(gv.id_space)
    out = []
    for transpose in (False, True):
        y = np.zeros_like(x)
        W.spmv(gv, W.Product("plus_times", transpose=transpose), x, y)
        out.append(y)
    return out


def graph():
    return W.gnm(300007, 3000000, seed=2)  # enough entries for its products to walk the copies


def copies(g):
    """The least that the copies of a version take: three of its targets."""
    return 12 * g.edges


def test_a_second_upload_takes_the_room_of_the_first_ones_copies():
    g = graph()
    budget = W.Budget()
    a = upload(g, budget)
    one = budget.peak
    want = products(a)
    # Two versions without their copies fit, two with them do not.
    tight = W.Budget(2 * one - 2 * copies(g) + (1 << 16) + 16 * g.id_space)
    first = upload(g, tight)
    held = first.info().device_bytes
    second = upload(g, tight)
    assert first.info().device_bytes <= held - copies(g)
    for gv in (first, second):
        for y, w in zip(products(gv), want):
            assert np.array_equal(y, w)


def test_a_search_takes_the_room_of_its_versions_copies():
    g = graph()
    budget = W.Budget()
    gv = upload(g, budget)
    want = W.bfs_batched(gv, [0, 5, 9], [4, 4, 4])
    ranks = W.pagerank(gv, None, W.PageRank(0.85, 1e-10, 100))
    probe = W.Budget()
    upload(g, probe)
    tight = W.Budget(probe.peak)
    gv = upload(g, tight)
    held = gv.info().device_bytes
    got = W.bfs_batched(gv, [0, 5, 9], [4, 4, 4])
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert gv.info().device_bytes <= held - copies(g)
    again = W.pagerank(gv, None, W.PageRank(0.85, 1e-10, 100))
    assert again.iterations == ranks.iterations
    assert np.abs(again.values - ranks.values).sum() <= 1e-12


def test_a_captured_walk_keeps_its_versions_copies():
    torch = pytest.importorskip("torch")
    g = graph()
    probe = W.Budget()
    upload(g, probe)
    tight = W.Budget(2 * probe.peak - 2 * copies(g))
    gv = upload(g, tight)
    x = torch.rand(g.id_space, dtype=torch.float64, device="cuda")
    y, z = torch.zeros_like(x), torch.zeros_like(x)
    product = W.Product("plus_times", transpose=True)
    W.spmv(gv, product, x, z)
    stream = torch.cuda.Stream()
    captured = torch.cuda.CUDAGraph()
    with torch.cuda.graph(captured, stream=stream):
        W.spmv(gv, product, x, y, stream=stream, asynchronous=True)
    held = gv.info().device_bytes
    with pytest.raises(W.MemoryLimit):
        upload(g, tight)
    assert gv.info().device_bytes == held
    captured.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, z)
