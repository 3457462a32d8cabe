"""Complex64 products on the tensor cores (AHX_ZT_MIN=1): right-hand sides and leaves whose
parts cannot be split (infinities, NaN, the ends of FP32's range) give what the plain kernel
gives, beside others that can."""
import numpy as np
import pytest

import ahmed_gb300 as A
import mbls_format as mbls

pytestmark = pytest.mark.gpu


def _matrix(n=700):
    P = A.geometry.sphere_surface(n, 5)
    return A.HMatrix(P, "bbx", bmin=8, eta=0.8).helmholtz_assemble(4.0, 0.05, 1e-6)


def _both(f, X, monkeypatch, Y0=None):
    Y0 = np.zeros_like(X) if Y0 is None else Y0
    monkeypatch.setenv("AHX_ZT_MIN", "1")
    got = f(0.5, X, Y0.copy(), precision="fp32")
    monkeypatch.setenv("AHX_ZT_MIN", str(10**18))
    want = f(0.5, X, Y0.copy(), precision="fp32")
    return got, want


def _same(got, want):
    for a, b in ((got.real, want.real), (got.imag, want.imag)):
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b))
    for r in range(len(got)):
        if np.isfinite(want[r]).all():
            # complex64 operands and sums on both sides: a few 2^-24
            assert np.linalg.norm(got[r] - want[r]) <= 1e-6 * np.linalg.norm(want[r]), r


BAD = [np.inf, -np.inf, np.nan, complex(1.0, np.nan), complex(np.inf, 1.0), complex(0.0, -np.inf), 3.4e38, 3.40282e38,
       1e300, 1e30j]


@pytest.mark.parametrize("bad", BAD, ids=str)
@pytest.mark.parametrize("op", ["mltaGeHVec", "mltaGeHhVec", "mltaGeHtVec"])
@pytest.mark.parametrize("p", [3, 5, 16, 20])
def test_entries_of_x(bad, op, p, monkeypatch):
    M = _matrix()
    rng = np.random.default_rng(p)
    X = rng.standard_normal((p, M.n)) + 1j * rng.standard_normal((p, M.n))
    X[p - 1, 13] = bad
    _same(*_both(getattr(M, op), X, monkeypatch))
    M.close()


@pytest.mark.parametrize("scale", [1e-36, 1e-33, 1e-20, 1e20, 1e33])
def test_sizes_of_x(scale, monkeypatch):
    M = _matrix()
    rng = np.random.default_rng(3)
    X = rng.standard_normal((18, M.n)) + 1j * rng.standard_normal((18, M.n))
    X[::3] *= scale
    X[4] = 0.0
    _same(*_both(M.mltaGeHVec, X, monkeypatch))
    M.close()


@pytest.mark.parametrize("kind,value", [("one", np.inf), ("one", np.nan), ("one", 3.4e38), ("one", 1e300), ("all", 1e-35),
                                        ("all", 1e30), ("col", 1e-30), ("factors", 1e18), ("factors", 1e30)])
def test_leaves(kind, value, tmp_path, monkeypatch):
    M = _matrix()
    ranks, L, data, offs = M.helm_ranks(), M.leaves(), [], [0]
    low = int(np.argmax(ranks > 0))
    for l in range(M.nleaves):
        n1, b2, n2 = int(L[l][1]), int(L[l][2]), int(L[l][3])
        k, d = int(ranks[l]), M.helm_leaf_data(l).copy()
        if kind == "one" and l in (0, low):
            d[1] = value
        elif kind == "all":
            d *= value if k < 0 else np.sqrt(value)
        elif kind == "col" and b2 <= 13 < b2 + n2:
            D = d.reshape(n2, n1) if k < 0 else d[k * n1:].reshape(k, n2).T
            D[13 - b2] *= value
        elif kind == "factors" and k > 0:  # the same blocks
            d[:k * n1] *= value
            d[k * n1:] /= value
        data.append(d)
        offs.append(offs[-1] + d.size)
    path = str(tmp_path / "leaves")
    mbls.write(path, 0.8, 8, L, ranks, np.concatenate(data).view(np.float64), 2 * np.array(offs))
    M.helm_load(path)
    rng = np.random.default_rng(4)
    X = rng.standard_normal((6, M.n)) + 1j * rng.standard_normal((6, M.n))
    X[2] = 0.0
    X[2, 13] = 1.0
    for op in ("mltaGeHVec", "mltaGeHhVec"):
        _same(*_both(getattr(M, op), X, monkeypatch))
    M.close()
