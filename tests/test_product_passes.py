"""FP64 and complex128 products with more right-hand sides than one pass of the digit-sliced
product takes (16, complex 8): columns that do not fit the digits are left to the plain
kernel, the other passes' columns are added once.  Compared with the plain kernel, one
right-hand side at a time."""
import numpy as np
import pytest

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.fixture
def sliced(monkeypatch):
    monkeypatch.setenv("AHX_DG_MIN", "0")


def _check(f, X, Y0, skip=()):
    p, n = X.shape
    Y, Y1 = Y0.copy(), Y0.copy()
    f(-0.5, p, X, n, Y, n)
    for r in range(p):
        f(-0.5, 1, X[r:], n, Y1[r:], n)
    for r in range(p):
        if r in skip:
            assert np.array_equal(np.isnan(Y[r]), np.isnan(Y1[r])) and np.array_equal(np.isinf(Y[r]), np.isinf(Y1[r])), r
            continue
        # both forms round each right-hand side to a few 1e-16 of its norm
        assert np.linalg.norm(Y[r] - Y1[r]) <= 4e-15 * np.linalg.norm(Y1[r]), r


def _vectors(p, n, cplx, seed):
    rng = np.random.default_rng(seed)
    X, Y0 = rng.standard_normal((p, n)), rng.standard_normal((p, n))
    if cplx:
        X, Y0 = X + 1j * rng.standard_normal((p, n)), Y0 + 1j * rng.standard_normal((p, n))
    return X, Y0


# columns of the pass that does not fit: the last one, a ragged last one, one in the middle
@pytest.mark.parametrize("cplx,p,c0,c1", [(False, 17, 16, 17), (False, 20, 16, 20), (False, 33, 32, 33),
                                          (False, 40, 16, 32), (True, 9, 8, 9), (True, 11, 8, 11), (True, 17, 8, 16)])
@pytest.mark.parametrize("bad", ["spread", "subnormal", "inf", "none"])
def test_one_pass_does_not_fit(sliced, cplx, p, c0, c1, bad):
    n = 700
    M = A.HMatrix(A.geometry.sphere_surface(n, 5), "bbx", bmin=8, eta=0.8, symmetric=(p == 40))
    M.helmholtz_assemble(4.0, 0.01, 1e-6) if cplx else M.matgenGeH_omp(0.01, 1e-6)
    X, Y0 = _vectors(p, n, cplx, p)
    skip = ()
    if bad == "spread":
        X[c0:c1, 13] = 1e-250
    elif bad == "subnormal":
        X[c0:c1] *= 1e-310
    elif bad == "inf":
        X[c1 - 1, 13] = np.inf
        skip = (c1 - 1,)
    forms = [M.mltaGeHGeM, M.mltaGeHhGeM, M.mltaGeHtGeM] if cplx else [M.mltaGeHGeM, M.mltaGeHtGeM]
    if not cplx and p == 20:
        forms.append(lambda d, q, x, lx, y, ly: M.mltaGeHGeM(d, q, x, lx, y, ly, precision="df64" if q > 1 else "fp64"))
    for f in forms:
        _check(f, X, Y0, skip)
    M.close()


@pytest.mark.parametrize("p", [17, 33])
def test_inner_products_of_the_last_pass_do_not_fit(sliced, p):
    """V^T X below 2^-200 of X for the last right-hand sides, zero for the others."""
    n = 700
    M = A.HMatrix(A.geometry.sphere_surface(n, 5), "bbx", bmin=8, eta=0.8)
    M.matgenGeH_omp(0.01, 1e-6)
    ranks, L, data, offs = M.ranks(), M.leaves(), [], [0]
    low = int(np.argmax(ranks > 0))
    assert ranks[low] > 0
    for l in range(M.nleaves):
        d = M.leaf_data(l)
        if l == low:
            nu = int(ranks[l]) * int(L[l, 1])
            d[:nu] *= 1e90
            d[nu:] *= 1e-90
        data.append(d)
        offs.append(offs[-1] + d.size)
    M.set_leaves(ranks, np.concatenate(data), np.array(offs, np.uint64))
    b2, n2 = int(L[low, 2]), int(L[low, 3])
    X, Y0 = _vectors(p, n, False, p)
    X[:p - 1, b2:b2 + n2] = 0.0
    _check(M.mltaGeHGeM, X, Y0)
    M.close()
