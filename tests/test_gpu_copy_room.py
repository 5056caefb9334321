"""What a version holds only to make calls faster (the lane-major copies, the
batched search's order of units) is left out where its budget has no room for
it: the upload is accepted as soon as the arrays that every call needs fit,
and each call that gets its scratch answers as on a version that has it all."""

import numpy as np
import pytest

import pg_warren_b200 as W

pytestmark = pytest.mark.gpu


def version(g, weights, limit=1 << 62):
    budget = W.Budget(limit)
    rev = W.api.host_reverse(g.offsets, g.targets, weights)
    return budget, W.GraphVersion(g.offsets, g.targets, weights, reverse=rev, budget=budget)


def accepted(g, weights, limit):
    try:
        version(g, weights, limit)
        return True
    except W.MemoryLimit as e:
        d = e.detail
        assert d.limit == limit and d.requested > limit - d.in_use
        return False


def calls(g, gv, weights):
    """name -> a call's outputs, or None where its scratch was refused."""
    torch = pytest.importorskip("torch")
    n = g.id_space
    x = torch.from_numpy(np.random.default_rng(4).random(n)).cuda()
    opts = W.PageRank(0.85, 1e-10, 100)

    def product(transpose):
        y = torch.zeros_like(x)
        W.spmv(gv, W.Product("plus_times", transpose=transpose), x, y)
        return [y.cpu().numpy()]

    def ranks(call):
        r = call(gv, None, opts)
        return [np.uint32(r.iterations), r.values]

    # The smallest scratch first.
    todo = [("noalloc", lambda: ranks(W.pagerank_noalloc)),
            ("product", lambda: product(False)), ("transposed", lambda: product(True)),
            ("batched", lambda: list(W.bfs_batched(gv, [0, 5], [3, 3]))),
            ("bfs", lambda: list(W.bfs_depths(gv, [3])[:2])),
            ("pagerank", lambda: ranks(W.pagerank))]
    if weights is not None:
        todo.append(("minplus", lambda: list(W.minplus_batched(gv, [0, 7], [4, 4]))))
    out = {}
    for name, call in todo:
        try:
            out[name] = [np.array(o) for o in call()]
        except W.MemoryLimit:
            out[name] = None
    return out


@pytest.mark.parametrize("nodes,edges,weighted", [(60007, 900000, False),
                                                  (60007, 900000, True), (9, 0, False)])
def test_an_upload_is_accepted_without_room_for_the_fast_copies(nodes, edges, weighted):
    g = W.gnm(nodes, edges, seed=2)
    w = W.edge_weights(g, "int") if weighted else None
    budget, gv = version(g, w)
    full, m = budget.peak, g.edges
    held = gv.info().device_bytes
    want = calls(g, gv, w)
    assert all(v is not None for v in want.values())
    lo, hi = 0, full  # refused, accepted
    while hi - lo > 256:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if accepted(g, w, mid) else (mid, hi)
    # Both orientations' targets and one renumbered, at the least, and their
    # weights in 64 and 32 bits.
    assert full - hi >= 12 * m + (24 * m if weighted else 0)
    served = set()
    room = full - hi
    for extra in sorted({0, room // 16, room // 8, room // 4, room // 2, 3 * room // 4, room}):
        _, tight = version(g, w, hi + extra)
        got = calls(g, tight, w)
        for name, outputs in got.items():
            if outputs is None:
                continue
            if tight.info().device_bytes < held:
                served.add(name)
            for a, b in zip(outputs, want[name]):
                if name in ("noalloc", "pagerank") and a.ndim:
                    assert np.abs(a - b).sum() <= 1e-12 * np.abs(b).sum()
                else:
                    assert np.array_equal(a, b)
        if got["pagerank"] is not None:
            assert np.array_equal(got["pagerank"][1], got["noalloc"][1])
    if m > 12 * nodes:  # the copies are larger than any of the calls' scratch
        assert served == set(want)  # each of them without some copy


def test_the_renumbered_copy_holds_no_integer_weights():
    # Its readers (the ranks) take 64-bit weights.  What 64-bit weights add: 8
    # bytes an entry of three row-major copies and a place of the two
    # lane-major ones; what integer ones add to that: 4 an entry of two and a
    # place of two.
    g = W.gnm(60007, 900000, seed=6)
    bytes_of = {k: version(g, w)[1].info().device_bytes for k, w in {
        "none": None, "float": W.edge_weights(g, "uniform"), "int": W.edge_weights(g, "int")}.items()}
    places = (bytes_of["float"] - bytes_of["none"] - 24 * g.edges) // 8
    assert places >= 2 * g.edges
    rounding = 4 * 256  # buffers come in multiples of 256 bytes
    assert bytes_of["int"] - bytes_of["float"] <= 8 * g.edges + 4 * places + rounding


@pytest.mark.parametrize("graph,copies", [("rmat 12", 0), ("rmat 16", 0), ("gnm 30000", 2),
                                          ("gnm 900000", 3)])
def test_a_copy_that_no_call_would_walk_is_not_built(graph, copies):
    # Small skewed graphs' calls walk the row-split schedule; PageRank on small
    # even ones the reverse copy, renumbered; products on larger ones both.
    kind, size = graph.split()
    g = W.rmat(int(size), seed=2) if kind == "rmat" else W.gnm(int(size) // 12, int(size), seed=2)
    n, m = g.id_space, g.edges
    held = version(g, None)[1].info().device_bytes
    rows = 12 * m + 20 * n  # three row-major copies and the renumbering
    # Beside them a version holds schedules (28 bytes a unit or less, of at most
    # 32 rows or 256 entries, and 76 a long row's piece) and buffers' roundings.
    schedules = 3 * (n // 16 + m // 128 + 64) * 104
    assert rows + 4 * copies * m <= held <= rows + 4 * copies * m + schedules + (copies and 16 * n)
