"""A target outside the id space is what an upload is refused for, also under a
budget that does not hold the arrays, with the first such target reported."""

import numpy as np
import pytest

import pg_warren_b200 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [1 << 30, 1 << 20, 1000, 0])
def test_a_target_outside_the_id_space_comes_before_a_memory_refusal(limit):
    n, m = 100, 200000
    offsets = np.full(n + 1, m, np.uint64)
    offsets[0] = 0
    targets = np.arange(m, dtype=np.uint32) % n
    targets[1234] = 107
    targets[150000] = 100
    with pytest.raises(W.api.NodeOutsideIdSpace) as e:
        W.GraphVersion(offsets, targets, budget=W.Budget(limit))
    assert e.value.detail.node == 107
