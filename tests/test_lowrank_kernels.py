"""ACA + recompression kernels over their branches: ranks up to 16 and 32 (shared-memory
squares) and beyond (workspace), the Cholesky and the Householder QR, clusters of a few points (ranks up to the block's sides), the symmetric cross,
factors that outgrow the arena's estimate, and a workspace that holds one team at a time."""
import numpy as np
import pytest

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu


def _points(n, seed):
    g = np.random.default_rng(seed).standard_normal((n, 3))
    return g / np.linalg.norm(g, axis=1, keepdims=True)


def _dense(P, h, k=None):
    r = np.linalg.norm(P[:, None] - P[None], axis=2)
    r[np.arange(len(P)), np.arange(len(P))] = h
    return 1.0 / (4 * np.pi * r) if k is None else np.exp(1j * k * r) / (4 * np.pi * r)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n,bmin,eps,sym,budget", [
    (700, 4, 1e-3, False, None),     # clusters of a few points
    (1500, 32, 1e-6, True, None),
    (2111, 24, 1e-9, False, None),   # ranks beyond 16
    (2111, 24, 1e-9, False, 1 << 16),
    (3000, 60, 1e-12, False, None),  # Householder, ranks beyond 32
    (900, 6, 1e-12, True, None),
])
def test_every_leaf_approximates_its_block(n, bmin, eps, sym, budget, cplx, monkeypatch):
    if budget:
        monkeypatch.setenv("AHX_ACA_WS_BYTES", str(budget))
    pts = _points(n, n)
    H = A.HMatrix(pts, "bbx", bmin=bmin, eta=0.8, symmetric=sym)
    h = A.mean_nn(pts)
    if cplx:
        H.helmholtz_assemble(6.0, h, eps)
        ranks, data = H.helm_ranks(), H.helm_leaf_data
    else:
        H.matgenGeH_omp(h, eps)
        ranks, data = H.ranks(), H.leaf_data
    M = _dense(pts[H.perm()[0]], h, 6.0 if cplx else None)
    lv = H.leaves()
    assert (ranks > 0).any()
    # the reference's stopping rule estimates the error by the last cross: within 20 eps of
    # the block here and in the other assembly tests; 1e-13 is the rounding of k <= 60 crosses
    tol = 20 * eps + 1e-13 * 60
    for l in np.nonzero(ranks >= 0)[0]:
        b1, n1, b2, n2 = (int(v) for v in lv[l, :4])
        k = int(ranks[l])
        d = data(int(l))
        assert d.size == k * (n1 + n2)
        B = M[b1:b1 + n1, b2:b2 + n2]
        U, V = d[:n1 * k].reshape(k, n1).T, d[n1 * k:].reshape(k, n2).T
        assert np.linalg.norm(U @ V.conj().T - B) <= tol * np.linalg.norm(B), (l, n1, n2, k)
        # truncated to the SVD: columns of U orthogonal, of V orthonormal, to the
        # tolerance's accuracy (the smallest kept direction is known to eps_mach / eps)
        G = V.conj().T @ V
        assert np.abs(G - np.eye(k)).max() <= 1e-14 * n2 / eps + 1e-9
    H.close()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("eps", [1e-6, 1e-12])
def test_a_cta_per_leaf(eps, cplx):
    """Few large leaves: the blocks above 512 rows and columns go to CTAs."""
    n = 20011
    pts = _points(n, 5)
    H = A.HMatrix(pts, "bbx", bmin=600, eta=1.5)
    lv = H.leaves()
    big = np.nonzero((lv[:, 4] == 1) & (lv[:, 1] + lv[:, 3] > 512))[0]
    assert len(big)
    h = A.mean_nn(pts)
    if cplx:
        H.helmholtz_assemble(3.0, h, eps)
        ranks, data = H.helm_ranks(), H.helm_leaf_data
    else:
        H.matgenGeH_omp(h, eps)
        ranks, data = H.ranks(), H.leaf_data
    assert (ranks[big] > 0).all()
    Q = pts[H.perm()[0]]
    for l in big[:: max(1, len(big) // 12)]:
        b1, n1, b2, n2 = (int(v) for v in lv[l, :4])
        r = np.linalg.norm(Q[b1:b1 + n1, None] - Q[None, b2:b2 + n2], axis=2)
        B = (np.exp(3j * r) if cplx else 1.0) / (4 * np.pi * r)
        k = int(ranks[l])
        d = data(int(l))
        U, V = d[:n1 * k].reshape(k, n1).T, d[n1 * k:].reshape(k, n2).T
        assert np.linalg.norm(U @ V.conj().T - B) <= (20 * eps + 6e-12) * np.linalg.norm(B), (l, n1, n2, k)
    H.close()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n,bmin,eta,eps", [(2500, 8, 0.8, 1e-3), (2500, 40, 0.8, 1e-6), (6007, 200, 2.0, 1e-9)])
def test_columns_of_u_are_orthogonal(n, bmin, eta, eps, cplx):
    """The triangular form and the last Jacobi sweep: ranks of 1 to more than 32, rows that
    the threshold empties, columns of very different lengths."""
    pts = _points(n, n + 1)
    H = A.HMatrix(pts, "bbx", bmin=bmin, eta=eta)
    h = A.mean_nn(pts)
    if cplx:
        H.helmholtz_assemble(9.0, h, eps)
        ranks, data = H.helm_ranks(), H.helm_leaf_data
    else:
        H.matgenGeH_omp(h, eps)
        ranks, data = H.ranks(), H.leaf_data
    lv = H.leaves()
    low = np.nonzero(ranks > 1)[0]
    assert len(low)
    for l in low:
        n1, k = int(lv[l, 1]), int(ranks[l])
        U = data(int(l))[:n1 * k].reshape(k, n1).T
        s = np.linalg.norm(U, axis=0)
        assert (s[1:] <= s[:-1] * (1 + 1e-6)).all()
        # Q1 = U R1^-1 is orthonormal to k u cond(R1)^2: column pivots above 1e-6 of their
        # columns' squares keep that below 1e-6; a sweep too few leaves 1e-5 to 1
        G = np.abs(U.conj().T @ U) / np.outer(s, s) - np.eye(k)
        assert np.abs(G).max() <= 1e-6, (l, n1, k)
    H.close()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("budget,batches", [(1 << 22, 2), (1 << 26, 1), (1 << 33, 1)])
def test_workspace_budgets(budget, batches, cplx, monkeypatch):
    """The largest leaves in a launch of their own (4 MB hold slots for few of them), leaves
    moved from warps to CTAs for want of slots, and neither."""
    import ctypes

    from ahmed_gb300._capi import lib
    monkeypatch.setenv("AHX_ACA_WS_BYTES", str(budget))
    n = 9001
    pts = _points(n, 11)
    H = A.HMatrix(pts, "bbx", bmin=16)
    h = A.mean_nn(pts)
    if cplx:
        H.helmholtz_assemble(3.0, h, 1e-6)
        ranks, data = H.helm_ranks(), H.helm_leaf_data
    else:
        H.matgenGeH_omp(h, 1e-6)
        ranks, data = H.ranks(), H.leaf_data
    stats = (ctypes.c_uint64 * 3)()
    lib().ahx_hmat_assembly_stats(H._h, stats)
    assert stats[0] <= budget and stats[2] == batches and stats[1] == 0
    Q = pts[H.perm()[0]]
    lv = H.leaves()
    low = np.nonzero(lv[:, 4] == 1)[0]
    assert (ranks[low] > 0).all()
    size = lv[low, 1] + lv[low, 3]
    for l in np.concatenate([low[np.argsort(size)[-6:]], low[:: len(low) // 40]]):
        b1, n1, b2, n2 = (int(v) for v in lv[l, :4])
        r = np.linalg.norm(Q[b1:b1 + n1, None] - Q[None, b2:b2 + n2], axis=2)
        B = (np.exp(3j * r) if cplx else 1.0) / (4 * np.pi * r)
        k, d = int(ranks[l]), data(int(l))
        U, V = d[:n1 * k].reshape(k, n1).T, d[n1 * k:].reshape(k, n2).T
        assert np.linalg.norm(U @ V.conj().T - B) <= 20 * 1e-6 * np.linalg.norm(B)
    H.close()
