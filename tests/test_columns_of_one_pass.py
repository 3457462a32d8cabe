"""FP64 and complex128 products whose right-hand sides meet columns of A of very different
size: each column of the result as exact as alone, whatever stands beside it."""
import numpy as np
import pytest

import ahmed_gb300 as A
import mbls_format as mbls

pytestmark = pytest.mark.gpu


def _scaled(n, cplx, side, s, tmp_path, bmin=8):
    """An H-matrix A diag(s) (side "col") or diag(s) A ("row")."""
    P = A.geometry.sphere_surface(n, 5)
    M = A.HMatrix(P, "bbx", bmin=bmin, eta=0.8)
    M.helmholtz_assemble(4.0, 0.05, 1e-6) if cplx else M.matgenGeH_omp(0.05, 1e-6)
    ranks = M.helm_ranks() if cplx else M.ranks()
    L, data, offs = M.leaves(), [], [0]
    assert (ranks > 0).any()
    for l in range(M.nleaves):
        b1, n1, b2, n2 = (int(v) for v in L[l][:4])
        k, d = int(ranks[l]), (M.helm_leaf_data(l) if cplx else M.leaf_data(l)).copy()
        if k < 0:
            D = d.reshape(n2, n1)
            D *= s[b2:b2 + n2, None] if side == "col" else s[None, b1:b1 + n1]
        else:
            U, V = d[:k * n1].reshape(k, n1), d[k * n1:].reshape(k, n2)
            if side == "col":
                V *= s[None, b2:b2 + n2]
            else:
                U *= s[None, b1:b1 + n1]
        data.append(d)
        offs.append(offs[-1] + d.size)
    data = np.concatenate(data)
    if cplx:
        path = str(tmp_path / "leaves")
        mbls.write(path, 0.8, bmin, L, ranks, data.view(np.float64), 2 * np.array(offs))
        M.helm_load(path)
    else:
        M.set_leaves(ranks, data, np.array(offs, np.uint64))
    return M


@pytest.mark.parametrize("ratio", [1e-5, 1e-12, 1e-40])
@pytest.mark.parametrize("cplx,op", [(False, "n"), (False, "t"), (True, "n"), (True, "h"), (True, "t")])
@pytest.mark.parametrize("p", [2, 7, 18])
def test_small_columns_beside_large_ones(cplx, op, p, ratio, tmp_path, monkeypatch):
    monkeypatch.setenv("AHX_DG_MIN", "0")
    n = 700
    rng = np.random.default_rng(p)
    s = np.where(rng.random(n) < 0.5, 1.0, ratio) * rng.uniform(0.5, 1.0, n)
    M = _scaled(n, cplx, "col" if op == "n" else "row", s, tmp_path)
    large, small = np.flatnonzero(s > 0.4), np.flatnonzero(s < 0.4)
    X = np.zeros((p, n), np.complex128 if cplx else np.float64)
    for r in range(p):  # vectors over the large and over the small columns, by turns
        at = rng.permutation(small if r & 1 else large)[:1 + 40 * (r // 2)]
        X[r, at] = rng.standard_normal(len(at))
        if cplx:
            X[r, at] += 1j * rng.standard_normal(len(at))
    f = {"n": M.mltaGeHVec, "t": M.mltaGeHtVec, "h": M.mltaGeHhVec}[op]
    Y, Y1 = np.zeros_like(X), np.zeros_like(X)
    f(1.0, X, Y)
    for r in range(p):
        f(1.0, X[r], Y1[r])
    # both forms round each right-hand side to a few 1e-16 of its norm
    for r in range(p):
        assert np.linalg.norm(Y[r] - Y1[r]) <= 4e-15 * np.linalg.norm(Y1[r]), r
    M.close()
