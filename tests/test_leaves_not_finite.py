"""Leaves whose crosses overflow (the reference's stopping rule does not end in time where
distances are of 1e-100) are not finite; none of them is dropped as a block of rank 0."""
import numpy as np
import pytest

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("scale", [1e-100, 1e-140])
def test_overflowed_leaves_show(scale, cplx):
    n = 700
    g = np.random.default_rng(3).standard_normal((n, 3))
    P = g / np.linalg.norm(g, axis=1, keepdims=True) * scale
    H = A.HMatrix(P, "bbx", bmin=6, eta=0.8)
    h = A.mean_nn(P)
    H.helmholtz_assemble(1.0 / scale, h, 1e-6) if cplx else H.matgenGeH_omp(h, 1e-6)
    ranks = H.helm_ranks() if cplx else H.ranks()
    assert (ranks > 0).any()
    # every entry is far from 0: a leaf of rank 0 is wrong
    assert not (ranks == 0).any()
    H.close()
