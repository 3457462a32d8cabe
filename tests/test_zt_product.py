"""Complex64 product on the tensor cores (AHX_ZT_MIN=1 lays it out at once) against the
complex128 product: every operation, right-hand side counts around the column tiles and
the block of 16, odd sizes, a symmetric tree, d other than 1, padded leading dimensions."""
import numpy as np
import pytest

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu


def _matrix(n, bmin, sym, seed):
    g = np.random.default_rng(seed).standard_normal((n, 3))
    pts = g / np.linalg.norm(g, axis=1, keepdims=True)
    H = A.HMatrix(pts, "bbx", bmin=bmin, eta=0.8, symmetric=sym)
    return H.helmholtz_assemble(5.0, A.mean_nn(pts), 1e-6)


@pytest.mark.parametrize("n,bmin,sym", [(300, 8, False), (1501, 32, False), (1501, 20, True), (2600, 64, False)])
def test_matches_complex128(n, bmin, sym, monkeypatch):
    monkeypatch.setenv("AHX_ZT_MIN", "1")
    H = _matrix(n, bmin, sym, n)
    rng = np.random.default_rng(1)
    for p in (1, 2, 4, 5, 8, 9, 16, 17, 35):
        x = rng.standard_normal((p, n)) + 1j * rng.standard_normal((p, n))
        y0 = rng.standard_normal((p, n)) + 1j * rng.standard_normal((p, n))
        for op in ("mltaGeHVec", "mltaGeHhVec", "mltaGeHtVec"):
            f = getattr(H, op)
            for d in (1.0, -0.5 + 2j):
                got = f(d, x, y0.copy(), precision="fp32") - y0
                want = f(d, x, y0.copy(), precision="fp64") - y0
                # complex64 leaves and X (2^-24 each), sums in FP32: a few 2^-24 of each
                # right-hand side's result; 1e-6 is 16 of them
                err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
                assert err.max() < 1e-6, (op, p, d)
    H.close()
