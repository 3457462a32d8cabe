"""The Helmholtz diagonal exp(i k h) / (4 pi h) of a single point, an admissible leaf of its own,
at sizes of h whose square is not a number."""
import cmath
import math

import numpy as np
import pytest

import ahmed_gb300 as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,k", [(0.3, 2.0), (1e-155, 2.0), (1e-155, 1e155), (1e155, 1e-155), (3e154, 0.0)])
def test_one_point(h, k):
    H = A.HMatrix(np.zeros((1, 3)), "bbx").helmholtz_assemble(k, h, 1e-6)
    y = np.zeros(1, np.complex128)
    H.mltaGeHVec(1.0, np.ones(1, np.complex128), y)
    want = cmath.exp(1j * k * h) / (4.0 * math.pi * h)
    # an entry of a few roundings, split into two factors
    assert abs(y[0] - want) <= 2e-15 * abs(want)
    H.close()
