"""Products and `prepare` when device memory has no room for the block layout or its work
buffer: the plain kernels run, as they do where there is no layout."""
import numpy as np
import pytest
import torch

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu

SWITCHES = ("AHX_DG_MIN", "AHX_ZT_MIN", "AHX_F1_MIN")


def _fill():
    """Tensors that leave less than 4 MB of the device."""
    torch.cuda.empty_cache()
    held = []
    for size in (8 << 30, 1 << 30, 64 << 20, 2 << 20):
        while torch.cuda.mem_get_info()[0] >= size + (2 << 20):
            try:
                held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                break
    return held


@pytest.mark.parametrize("kind,p,op", [("real", 1, "n"), ("real", 1, "t"), ("real", 4, "n"), ("real", 4, "t"),
                                       ("c128", 3, "n"), ("c128", 3, "h"), ("c64", 6, "n")])
def test_product(kind, p, op, monkeypatch):
    n = 6007
    pts = A.geometry.sphere_surface(n, 5)
    cplx = kind != "real"
    prec = "fp32" if kind == "c64" else "fp64"
    rng = np.random.default_rng(1)
    X = rng.standard_normal((p, n)) + (1j * rng.standard_normal((p, n)) if cplx else 0)
    X = torch.from_numpy(X[0] if p == 1 else X).cuda()
    Y = torch.zeros_like(X)

    def handle():
        H = A.HMatrix(pts, "bbx")
        H.helmholtz_assemble(4.0, 0.02, 1e-6) if cplx else H.matgenGeH_omp(0.02, 1e-6)
        return H, {"n": H.mltaGeHVec, "t": H.mltaGeHtVec, "h": H.mltaGeHhVec}[op]

    def use(least):
        for v in SWITCHES:
            monkeypatch.setenv(v, least)

    K, g = handle()
    use("1")
    g(1.0, X, Y, precision=prec)  # (every kernel is loaded)
    H, f = handle()
    use(str(10**18))
    want = torch.zeros_like(X)
    f(1.0, X, want, precision=prec)
    torch.cuda.synchronize()
    use("1")
    held = _fill()
    if kind == "real" and op == "n":
        H.prepare("fp64")
    Y.zero_()
    f(1.0, X, Y, precision=prec)
    torch.cuda.synchronize()
    del held
    torch.cuda.empty_cache()
    Z = torch.zeros_like(X)
    f(1.0, X, Z, precision=prec)  # laid out, now that there is room
    # the same sums in another order (complex64: other roundings)
    tol = 1e-6 if kind == "c64" else 1e-13
    for y in (Y, Z):
        assert float((y - want).norm() / want.norm()) <= tol
    K.close()
    H.close()
