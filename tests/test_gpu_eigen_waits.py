"""Lanczos reads its products' results on the host only once they are there: the
symmetry test of a large matrix that is not symmetric, on fresh versions (whose
buffers hold nothing of an earlier call's), and the vectors that a call returns,
each a unit vector, call after call."""

import numpy as np
import pytest

import pg_warren_b200 as W

pytestmark = pytest.mark.gpu


def test_a_large_matrix_that_is_not_symmetric_is_refused_each_time():
    g = W.rmat(19, seed=5)
    for _ in range(4):
        gv = g.upload()
        for _ in range(3):
            with pytest.raises(W.api.NotSymmetric):
                W.eigen(gv, W.EigenOptions(2, which="largest", operator="adjacency",
                                           symmetrize=False, tol=1e-8, max_iter=200))


@pytest.mark.parametrize("operator,which", [("random_walk", "largest"),
                                            ("normalized_laplacian", "smallest")])
def test_the_vectors_returned_are_unit_vectors(operator, which):
    g = W.rmat(17, seed=5)
    gv = g.upload()
    for _ in range(3):
        e = W.eigen(gv, W.EigenOptions(3, which=which, operator=operator, symmetrize=True,
                                       tol=1e-6, max_iter=200))
        norms = np.linalg.norm(np.asarray(e.vectors), axis=1)
        # A sum of n squares of about 1 / n each: n ulps at the most.
        assert np.abs(norms - 1.0).max() <= g.id_space * 2.3e-16
