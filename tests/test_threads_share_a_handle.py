"""Products and solves of one handle from several threads: their work buffers are the
handle's, their kernels must not interleave."""
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


@pytest.mark.parametrize("cplx,p", [(False, 1), (False, 5), (True, 3)])
def test_products(cplx, p):
    n = 4001
    pts = A.geometry.sphere_surface(n, 6)
    H = A.HMatrix(pts, "bbx")
    if cplx:
        H.helmholtz_assemble(4.0, A.mean_nn(pts), 1e-6)
    else:
        H.matgenGeH_omp(A.mean_nn(pts), 1e-6)
    t = torch.complex128 if cplx else torch.float64
    g = torch.Generator().manual_seed(1)
    X = [torch.randn(p, n, dtype=t, generator=g).cuda() for _ in range(4)]
    ref = []
    for x in X:
        for _ in range(6):  # (beyond the products after which the block layout is there)
            y = torch.zeros_like(x)
            H.mltaGeHGeM(1.0, p, x, n, y, n)
        ref.append(y)
    out = [[] for _ in X]

    def job(q):
        def f():
            for _ in range(40):
                y = torch.zeros_like(X[q])
                H.mltaGeHGeM(1.0, p, X[q], n, y, n)
                out[q].append(y)
        return f

    _run([job(q) for q in range(4)])
    torch.cuda.synchronize()
    for q in range(4):
        for y in out[q]:
            # atomics add in another order: FP64 rounding of sums of 4,001 terms
            assert float((y - ref[q]).norm() / ref[q].norm()) <= 1e-13
    H.close()


def test_solves():
    n = 2111
    pts = A.geometry.sphere_surface(n, 4)
    H = A.HMatrix(pts, "bbx")
    H.matgenGeH_omp(A.min_nn(pts) / 2, 1e-6)
    B = np.random.default_rng(2).standard_normal((4, n))
    ref = np.zeros((4, n))
    for q in range(4):
        H.GMRes(torch.from_numpy(B[q]).cuda(), x := torch.zeros(n, dtype=torch.float64, device="cuda"), 1e-10, 30, 90)
        ref[q] = x.cpu().numpy()
    out = np.zeros((4, n))

    def job(q):
        def f():
            b = torch.from_numpy(B[q]).cuda()
            for _ in range(5):
                x = torch.zeros(n, dtype=torch.float64, device="cuda")
                status, res, _ = H.GMRes(b, x, 1e-10, 30, 90)
                assert status == 0 and res[0] < 1e-10
            out[q] = x.cpu().numpy()
        return f

    _run([job(q) for q in range(4)])
    # both solved to 1e-10, condition below 10
    assert np.linalg.norm(out - ref) <= 1e-8 * np.linalg.norm(ref)
    H.close()
