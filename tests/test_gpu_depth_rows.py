"""The batched search's depth rows stored into a buffer that starts anywhere:
node counts of every remainder by four, whole tiles and a last one, the bytes
before and behind the rows left as they were."""

import numpy as np
import pytest

import oracle as O
import pg_warren_b200 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 5, 15])
@pytest.mark.parametrize("nodes", [640, 1001, 1002, 1003, 1024])
def test_depth_rows_off_a_word_boundary(nodes, offset):
    torch = pytest.importorskip("torch")
    g = W.gnm(nodes, 5 * nodes, seed=7)
    og = O.Graph.from_csr(g.id_space, g.offsets, g.targets)
    gv = g.upload()
    n = g.id_space
    sources = np.arange(0, 37, dtype=np.uint64) * 3
    caps = np.full(37, 5, np.uint32)
    want, _ = O.bfs_depths(og, sources, caps)
    buffer = torch.full((37 * n + 64,), 77, dtype=torch.uint8, device="cuda")
    rows = buffer[offset:offset + 37 * n].view(37, n)
    W.bfs_batched(gv, sources, caps, depth_out=rows)
    assert np.array_equal(rows.cpu().numpy(), want)
    assert bool((buffer[:offset] == 77).all()) and bool((buffer[offset + 37 * n:] == 77).all())
