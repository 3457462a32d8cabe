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


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_solves_share_a_handles_scratch(precision):
    """Solves of other sizes in turn, from zero and from a given x, equal those of a handle
    of their own."""
    n = 2111
    pts = A.geometry.sphere_surface(n, 4)
    g = np.random.default_rng(0)

    def handle():
        H = A.HMatrix(pts, "bbx")
        H.matgenGeH_omp(A.min_nn(pts) / 2, 1e-6)  # positive definite, condition below 10
        return H

    kept = handle()
    for p, m, steps, zero in ((1, 30, 60, True), (3, 5, 40, False), (1, 50, 50, False), (2, 30, 60, True), (1, 2, 3, True)):
        B = g.standard_normal((p, n))
        X = np.zeros((p, n)) if zero else g.standard_normal((p, n))
        Y = X.copy()
        own = handle()
        s1 = kept.GMRes(B, X, 1e-8, m, steps, precision)
        s2 = own.GMRes(B, Y, 1e-8, m, steps, precision)
        own.close()
        assert s1[0] == s2[0] and (s1[2] == s2[2]).all()
        # products add with atomics, in another order each time: rounding (FP32-class products
        # 1e-6 of the result) times the condition
        assert np.linalg.norm(X - Y) <= (1e-9 if precision == "fp64" else 1e-5) * np.linalg.norm(Y)
    kept.close()
