"""FP64 product with one right-hand side over the block layout (AHX_F1_MIN=1 lays it out
at once) against the kernel that takes a leaf per CTA: A and A^T, odd sizes, clusters of a
few points and of more than a tile's rows, a symmetric tree, values that are not finite."""
import numpy as np
import pytest

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bmin,sym", [(61, 4, False), (700, 5, False), (2111, 32, False), (2111, 20, True),
                                        (5000, 64, False)])
def test_matches_the_leaf_kernel(n, bmin, sym, monkeypatch):
    g = np.random.default_rng(n).standard_normal((n, 3))
    pts = g / np.linalg.norm(g, axis=1, keepdims=True)
    H = A.HMatrix(pts, "bbx", bmin=bmin, eta=0.8, symmetric=sym).matgenGeH_omp(A.mean_nn(pts), 1e-6)
    rng = np.random.default_rng(2)
    x = rng.standard_normal(n)
    y0 = rng.standard_normal(n)
    for op in ("mltaGeHVec", "mltaGeHhVec"):
        for d in (1.0, -0.75):
            monkeypatch.setenv("AHX_F1_MIN", str(10**18))
            want = getattr(H, op)(d, x, y0.copy())
            monkeypatch.setenv("AHX_F1_MIN", "1")
            got = getattr(H, op)(d, x, y0.copy())
            # the same FP64 sums in another order: sqrt(n) roundings of 2^-53 of the result's
            # norm, a few times over (V^T x, then the rows)
            assert np.linalg.norm(got - want) <= 2.0**-53 * 4 * np.sqrt(n) * np.linalg.norm(want), (op, d)
    x[n // 2] = np.inf
    got = H.mltaGeHVec(1.0, x, y0.copy())
    assert not np.isfinite(got).all()
    H.close()
