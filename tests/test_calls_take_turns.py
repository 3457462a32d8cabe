"""One handle used from several threads at once, products beside solves, host vectors beside
device ones, different numbers of right-hand sides; and products that the caller captures
into a graph, replayed after the handle's work buffers have grown."""
import threading

import numpy as np
import pytest
import torch

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu


def _run(jobs):
    err = []

    def go(f):
        try:
            f()
        except Exception as e:  # noqa: BLE001 (reported below)
            err.append(e)

    ts = [threading.Thread(target=go, args=(f,)) for f in jobs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not err, err


def _handle(n, stream=None):
    pts = A.geometry.sphere_surface(n, 4)
    H = A.HMatrix(pts, "bbx", stream=stream.cuda_stream if stream else None)
    return H.matgenGeH_omp(A.min_nn(pts) / 2, 1e-6)


def _reference(H, X):
    """Products of right-hand sides X (p x n, host) by the plain kernel, one at a time."""
    Y = np.zeros_like(X)
    for r in range(len(X)):
        H.mltaGeHGeM(1.0, 1, X[r:], X.shape[1], Y[r:], X.shape[1])
    return Y


def _close(Y, want, tol=1e-13):
    # FP64 sums of 2,111 terms in another order
    assert np.linalg.norm(Y - want, axis=1).max() <= tol * np.linalg.norm(want, axis=1).max()


@pytest.mark.parametrize("device", [True, False])
def test_products_beside_solves(device, monkeypatch):
    monkeypatch.setenv("AHX_DG_MIN", "0")
    n = 2111
    s = torch.cuda.Stream()  # (one that can capture: the solves run graphs)
    H = _handle(n, s if device else None)
    rng = np.random.default_rng(2)
    give = (lambda a: torch.from_numpy(a).cuda()) if device else (lambda a: a.copy())
    take = (lambda a: a.cpu().numpy()) if device else (lambda a: a)
    sizes = (3, 16, 20, 1)
    X = [rng.standard_normal((p, n)) for p in sizes]
    B = [rng.standard_normal((5, n)), rng.standard_normal((2, n))]
    want = [_reference(H, x) for x in X]
    dX, dB = [give(x) for x in X], [give(b) for b in B]
    outs = [[give(np.zeros((p, n))) for _ in range(30)] for p in sizes]
    sols = [[give(np.zeros(b.shape)) for _ in range(6)] for b in B]
    torch.cuda.synchronize()

    def multiply(q):
        def f():
            for y in outs[q]:
                H.mltaGeHGeM(1.0, sizes[q], dX[q], n, y, n)
        return f

    def solve(q):
        def f():
            for x in sols[q]:
                status, res, _ = H.GMRes(dB[q], x, 1e-10, 30, 120, precision="fp32" if q else "fp64")
                assert status == 0 and res.max() < 1e-10
        return f

    _run([multiply(q) for q in range(len(sizes))] + [solve(q) for q in range(len(B))])
    torch.cuda.synchronize()
    for q in range(len(sizes)):
        for y in outs[q]:
            _close(take(y), want[q])
    for q, b in enumerate(B):
        for x in sols[q]:
            _close(_reference(H, np.ascontiguousarray(take(x))), b, 1e-9)
    H.close()


@pytest.mark.parametrize("kind,p,op", [("real", 1, "n"), ("real", 5, "n"), ("real", 5, "t"), ("c128", 3, "n"),
                                       ("c128", 3, "h"), ("c64", 6, "n")])
def test_captured_products(kind, p, op, monkeypatch):
    for v in ("AHX_DG_MIN", "AHX_ZT_MIN", "AHX_F1_MIN"):
        monkeypatch.setenv(v, "1")
    n = 2111
    s = torch.cuda.Stream()
    H = _handle(n, s)
    cplx = kind != "real"
    if cplx:
        H.helmholtz_assemble(4.0, 0.02, 1e-6)
    prec = "fp32" if kind == "c64" else "fp64"
    t = torch.complex128 if cplx else torch.float64
    f = {"n": H.mltaGeHVec, "t": H.mltaGeHtVec, "h": H.mltaGeHhVec}[op]
    big = torch.randn(40, n, dtype=t, device="cuda")
    X = torch.randn(p, n, dtype=t, device="cuda")
    X = X[0] if p == 1 else X
    want, Y, Z = torch.zeros_like(X), torch.zeros_like(X), torch.zeros_like(big)
    torch.cuda.synchronize()
    f(1.0, X, want, precision=prec)  # (layout and buffers are there)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        f(1.0, X, Y, precision=prec)
    f(1.0, big, Z, precision=prec)  # more right-hand sides: the work buffer grows
    torch.cuda.synchronize()
    junk = torch.full((64 << 20,), float("nan"), device="cuda")  # (what has been freed is reused)
    with torch.cuda.stream(s):
        for _ in range(3):
            Y.zero_()
            g.replay()
    torch.cuda.synchronize()
    tol = 1e-6 if kind == "c64" else 1e-13
    assert float((Y - want).norm() / want.norm()) <= tol
    del junk
    H.close()
