"""What a plain search charges to its call's budget for the list of long rows:
four bytes for every 2,048 entries of the rows it searches; and searches whose
frontier has more long rows than that list holds, against the oracle."""

import ctypes as C

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W
from pg_warren_b200 import _abi as A

pytestmark = pytest.mark.gpu


def charged(edges, direction):
    g = W.gnm(5000, edges, seed=1)
    gv = g.upload()
    budget = W.Budget()
    call, detail = W.api._call(None, None, 0, budget)
    starts = np.zeros(1, np.uint64)
    depth, via = np.zeros(g.id_space, np.uint32), np.zeros(g.id_space, np.uint64)
    limits, stats = W.api._limits(W.Limits(4, None)), A.TraversalStats()
    status = A.load().wc_bfs(gv.handle, C.byref(call), {"out": 0, "both": 2}[direction],
                             starts.ctypes.data, 1, C.byref(limits), None, depth.ctypes.data,
                             via.ctypes.data, C.byref(stats))
    assert status == 0
    return g.edges, budget.peak


@pytest.mark.parametrize("direction", ["out", "both"])
def test_the_long_row_list_takes_four_bytes_for_2048_entries(direction):
    rows = 2 if direction == "both" else 1
    (m0, b0), (m1, b1) = charged(20000, direction), charged(900000, direction)
    assert b1 - b0 == 4 * rows * (m1 // 2048 - m0 // 2048)


@pytest.mark.parametrize("direction", ["out", "in", "both"])
@pytest.mark.parametrize("nodes,degree", [(3000, 700), (2000, 900), (5000, 650)])
def test_more_long_rows_than_the_list_holds(nodes, degree, direction):
    g = W.gnm(nodes, nodes * degree, seed=4)
    assert (np.diff(g.offsets.astype(np.int64)) > 512).sum() > g.edges // 2048
    og = O.Graph.from_csr(g.id_space, g.offsets, g.targets)
    gv = g.upload()
    starts = list(range(0, nodes, 7))  # many long rows in the first frontier
    got = W.bfs(gv, starts, limits=W.Limits(3, None), direction=direction)
    want, stats = O.bfs(og, starts, {"out": 0, "in": 1, "both": 2}[direction], 3)
    assert [(v.node, v.depth, v.via) for v in got.result] == want
    assert got.stats.edges_traversed == stats["edges_traversed"]
