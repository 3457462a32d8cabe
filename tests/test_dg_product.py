"""The digit-sliced FP64 / complex128 product (several right-hand sides): its layout
on the host against a direct evaluation of the leaves for every way a leaf acts, and
on the GPU against the plain FP64 kernel (one right-hand side at a time)."""
import ctypes as C
import os

import numpy as np
import pytest

import ahmed_gb300 as A
from ahmed_gb300 import _capi

N, T, H = 0, 1, 2


def _leaf_set(rng, n, cplx):
    """A random nested partition of an n x n matrix into dense and low-rank leaves."""
    out, parts, off = [], [], 0

    def val(m):
        v = rng.standard_normal(m)
        return v + 1j * rng.standard_normal(m) if cplx else v

    def split(b1, n1, b2, n2, depth):
        nonlocal off
        if depth == 0 or min(n1, n2) < 8 or rng.random() < 0.2:
            k = -1 if rng.random() < 0.5 else int(rng.integers(0, min(n1, n2, 20)))
            d = val(n1 * n2 if k < 0 else k * (n1 + n2))
            out.append((b1, n1, b2, n2, k, off))
            parts.append(d)
            off += d.size
            return
        h1, h2 = n1 // 2 + 1, n2 // 2
        for a, m in ((b1, h1), (b1 + h1, n1 - h1)):
            for b, w in ((b2, h2), (b2 + h2, n2 - h2)):
                split(a, m, b, w, depth - 1)

    split(0, n, 0, n, 4)
    return out, np.concatenate(parts)


def _apply(leaves, arena, X, mode):
    Y = np.zeros_like(X)
    for b1, n1, b2, n2, k, off in leaves:
        if k == 0:
            continue
        if k < 0:
            M = arena[off:off + n1 * n2].reshape(n2, n1).T
        else:
            U = arena[off:off + n1 * k].reshape(k, n1).T
            V = arena[off + n1 * k:off + (n1 + n2) * k].reshape(k, n2).T
            M = U @ V.conj().T
        if mode == N:
            Y[:, b1:b1 + n1] += X[:, b2:b2 + n2] @ M.T
        else:
            Y[:, b2:b2 + n2] += X[:, b1:b1 + n1] @ (M if mode == T else M.conj())
    return Y


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("mode", [N, T, H])
@pytest.mark.parametrize("n,ctas", [(1, 1), (7, 1), (49, 4), (300, 1), (1500, 4000), (2600, 1)])
def test_layout_applies_every_leaf(n, ctas, mode, cplx):
    rng = np.random.default_rng(n + mode)
    leaves, arena = _leaf_set(rng, n, cplx)
    X = rng.standard_normal((2, n)) + (1j * rng.standard_normal((2, n)) if cplx else 0)
    words = np.array([[b1, n1, b2, n2, np.uint32(np.int64(k) & 0xffffffff), mode] for b1, n1, b2, n2, k, _ in leaves],
                     dtype=np.uint32)
    offs = np.array([q[5] for q in leaves], dtype=np.uint64)
    Y = np.zeros_like(X)
    info = np.zeros(4, np.uint64)
    f = _capi.lib().ahx_dg_host_product
    f.restype = C.c_int
    f.argtypes = [C.c_uint32, C.c_uint32, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_uint32, C.c_void_p,
                  C.c_void_p, C.c_void_p, C.c_uint32]
    assert f(n, len(words), words.ctypes.data, offs.ctypes.data, arena.ctypes.data, int(cplx), 2, X.ctypes.data,
             Y.ctypes.data, info.ctypes.data, ctas) == 0
    ref = _apply(leaves, arena, X, mode)
    assert np.linalg.norm(Y - ref) <= 1e-12 * max(np.linalg.norm(ref), 1e-300)
    assert info[3] <= 48


@pytest.fixture
def sliced(monkeypatch):
    """Every product of two or more right-hand sides takes the sliced path."""
    monkeypatch.setenv("AHX_DG_MIN", "0")


def _matrix(n, kind="bbx", sym=False, bmin=32):
    P = A.geometry.sphere_surface(n, 5)
    return A.HMatrix(P, kind, bmin=bmin, eta=0.8, symmetric=sym)


def _close(Y, Y1, tol=4e-15):
    # both forms round each right-hand side to a few 1e-16 of its norm
    for r in range(len(Y)):
        assert np.linalg.norm(Y[r] - Y1[r]) <= tol * np.linalg.norm(Y1[r]), r


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind,sym", [(1, "bbx", False), (33, "bbx", False), (500, "pca", False),
                                        (2100, "bbx", True), (4097, "bbx", False)])
@pytest.mark.parametrize("p", [2, 8, 9, 17])
def test_real_products(sliced, n, kind, sym, p):
    M = _matrix(n, kind, sym)
    M.matgenGeH_omp(0.01, 1e-6)
    rng = np.random.default_rng(n + p)
    ld = n + 3
    # right-hand sides of very different sizes, one of them zero, one sparse
    X = rng.standard_normal((p, ld)) * 10.0 ** rng.uniform(-30, 30, (p, 1))
    X[p - 1] = 0.0
    X[0, rng.integers(0, n, n // 2)] = 0.0
    Y0 = rng.standard_normal((p, ld)) * np.abs(X).max(axis=1, keepdims=True)
    for f in (M.mltaGeHGeM, M.mltaGeHtGeM):
        Y, Y1 = Y0.copy(), Y0.copy()
        f(-0.75, p, X, ld, Y, ld)
        for r in range(p):
            f(-0.75, 1, X[r:], ld, Y1[r:], ld)
        assert np.array_equal(Y[:, n:], Y0[:, n:])
        assert np.array_equal(Y[p - 1], Y0[p - 1])
        _close(Y[:p - 1, :n], Y1[:p - 1, :n])


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind,sym", [(1, "bbx", False), (200, "pca", False), (1100, "bbx", True), (1501, "bbx", False)])
@pytest.mark.parametrize("p", [2, 5, 9])
def test_complex_products(sliced, n, kind, sym, p):
    M = _matrix(n, kind, sym)
    M.helmholtz_assemble(6.0, 0.02, 1e-6)
    rng = np.random.default_rng(n + p)
    X = (rng.standard_normal((p, n)) + 1j * rng.standard_normal((p, n))) * 10.0 ** rng.uniform(-20, 20, (p, 1))
    for f in (M.mltaGeHGeM, M.mltaGeHhGeM, M.mltaGeHtGeM):
        Y, Y1 = np.zeros_like(X), np.zeros_like(X)
        f(0.5 - 2.0j, p, X, n, Y, n)
        for r in range(p):
            f(0.5 - 2.0j, 1, X[r:], n, Y1[r:], n)
        _close(Y, Y1)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.inf, np.nan, 5e-324, 1e-250])
def test_vectors_that_do_not_fit_take_the_plain_kernel(sliced, bad):
    """Infinite and NaN entries, and entries spread over more than 2^200, give the plain product."""
    n = 700
    M = _matrix(n)
    M.matgenGeH_omp(0.01, 1e-6)
    X = np.random.default_rng(0).standard_normal((3, n))
    X[1, 13] = bad
    Y, Y1 = np.zeros_like(X), np.zeros_like(X)
    M.mltaGeHVec(1.0, X, Y)
    for r in range(3):
        M.mltaGeHVec(1.0, X[r], Y1[r])
    assert np.array_equal(np.isnan(Y), np.isnan(Y1)) and np.array_equal(np.isinf(Y), np.isinf(Y1))
    ok = [r for r in range(3) if np.isfinite(Y1[r]).all()]
    _close(Y[ok], Y1[ok])
    # and the next product with ordinary vectors is sliced again
    X[1, 13] = 1.0
    Y, Y1 = np.zeros_like(X), np.zeros_like(X)
    M.mltaGeHVec(1.0, X, Y)
    for r in range(3):
        M.mltaGeHVec(1.0, X[r], Y1[r])
    _close(Y, Y1)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0.0, 1e-200, 1e200, np.inf])
def test_leaves_of_extreme_sizes(sliced, scale):
    """Leaves with zeros, and with elements that are left to the plain kernel."""
    n = 300
    M = _matrix(n)
    M.matgenGeH_omp(0.01, 1e-6)
    ranks, data, offs = M.ranks(), [], [0]
    for l in range(M.nleaves):
        d = M.leaf_data(l)
        d[: d.size // 3] *= scale
        data.append(np.nan_to_num(d, nan=np.inf, posinf=np.inf, neginf=-np.inf))
        offs.append(offs[-1] + d.size)
    M.set_leaves(ranks, np.concatenate(data), np.array(offs, np.uint64))
    X = np.random.default_rng(1).standard_normal((4, n))
    Y, Y1 = np.zeros_like(X), np.zeros_like(X)
    M.mltaGeHVec(1.0, X, Y)
    for r in range(4):
        M.mltaGeHVec(1.0, X[r], Y1[r])
    if np.isfinite(Y1).all():
        _close(Y, Y1, 1e-14)
    else:
        assert np.array_equal(np.isnan(Y), np.isnan(Y1))


@pytest.mark.gpu
def test_gmres_and_new_leaves_use_the_present_matrix(sliced):
    """Captured GMRES steps on several right-hand sides; a second assembly drops the layout."""
    n = 900
    P = A.geometry.sphere_surface(n, 5)
    M = A.HMatrix(P, "bbx", bmin=32, eta=0.8)
    for h in (0.5 * A.min_nn(P), 0.25 * A.min_nn(P)):
        M.matgenGeH_omp(h, 1e-6)
        B = np.random.default_rng(2).standard_normal((5, n))
        X = np.zeros_like(B)
        M.GMRes(B, X, 1e-10, 30, 300)
        R = B.copy()
        for r in range(5):
            M.mltaGeHVec(-1.0, X[r], R[r])
        assert np.max(np.linalg.norm(R, axis=1) / np.linalg.norm(B, axis=1)) <= 2e-10
