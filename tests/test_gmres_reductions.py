"""Gram-Schmidt sums (groups of 8, 4, 2 and 1 basis vectors, tiles of 64, a ragged last
chunk) and the triangular solve (blocks of 32 unknowns): one cycle of m steps reaches the
least residual over the Krylov space, found on the CPU from the same matrix."""
import numpy as np
import pytest

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 15, 32, 33, 75])
@pytest.mark.parametrize("p", [1, 3])
def test_a_cycle_minimises_the_residual(m, p):
    n = 1500  # a full chunk of 1,024 and a ragged one
    pts = A.geometry.sphere_surface(n, 3)
    H = A.HMatrix(pts, "bbx")
    H.matgenGeH_omp(A.mean_nn(pts), 1e-6)  # indefinite: no cycle here converges
    D = np.zeros((n, n))
    H.mltaGeHGeM(1.0, n, np.eye(n), n, D, n)
    D = D.T.copy()  # row j of the output is A e_j
    B = np.random.default_rng(m).standard_normal((p, n))
    X = np.zeros_like(B)
    b, x = (B[0], X[0]) if p == 1 else (B, X)
    ret, res, its = H.GMRes(b, x, 1e-13, m, m)
    assert ret == 1 and (its == m).all()
    for r in range(p):
        V = np.zeros((n, m + 1))
        V[:, 0] = B[r] / np.linalg.norm(B[r])
        for k in range(m):
            w = D @ V[:, k]
            for _ in range(2):
                w -= V[:, :k + 1] @ (V[:, :k + 1].T @ w)
            V[:, k + 1] = w / np.linalg.norm(w)
        y = np.linalg.lstsq(D @ V[:, :m], B[r], rcond=None)[0]
        best = np.linalg.norm(B[r] - D @ (V[:, :m] @ y))
        got = np.linalg.norm(B[r] - D @ X[r])
        # both are minima over the same space up to rounding (1e-16 times at most 80 steps
        # times the condition of the projected matrix, below 1e5)
        assert abs(got - best) <= 1e-8 * best
    H.close()
