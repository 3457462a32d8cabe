"""GMRES on systems whose reductions go through groups of items (more than 262,144 points), alone
and beside a small system in a batch."""
import numpy as np
import pytest
import torch

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu


def _matrix(n, seed):
    g = np.random.default_rng(seed).standard_normal((n, 3))
    P = g / np.linalg.norm(g, axis=1, keepdims=True)
    return A.HMatrix(P, "bbx", bmin=64, eta=0.8).matgenGeH_omp(0.5 * A.min_nn(P), 1e-6)


@pytest.mark.parametrize("n,p,precision", [(262145, 1, "fp64"), (300007, 3, "fp32")])
def test_one_matrix(n, p, precision):
    H = _matrix(n, 1)
    B = torch.randn(p, n, dtype=torch.float64, device="cuda")
    X = torch.zeros_like(B)
    status, res, iters = H.GMRes(B, X, 1e-10, 20, 200, precision=precision)
    assert status == 0 and res.max() < 1e-10 and iters.min() > 1
    R = B.clone()
    H.mltaGeHGeM(-1.0, p, X, n, R, n)
    # the solver's own residual is within FP64 rounding of this one
    assert float((R.norm(dim=1) / B.norm(dim=1)).max()) <= 2e-10
    H.close()


def test_batch():
    mats = [_matrix(2048, 2), _matrix(270001, 3), _matrix(65, 4)]
    bt = A.HBatch(mats, "fp64")
    b = torch.randn(int(bt.n), dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    status, res, iters = bt.gmres(b, x, 1e-10, 20, 200)
    assert status == 0 and res.max() < 1e-10
    for H, i, j in zip(mats, bt.offsets, bt.offsets[1:]):
        r = b[i:j].clone()
        H.mltaGeHVec(-1.0, x[i:j].clone(), r)
        assert float(r.norm() / b[i:j].norm()) <= 2e-10
    bt.close()
    for H in mats:
        H.close()
