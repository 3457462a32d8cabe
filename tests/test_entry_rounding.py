"""Entries of dense leaves, 1 / (4 pi r), are the host's bit for bit at the distances where a
reciprocal or a square root lies closest to the middle of two doubles: t = 4 pi r = T 2^e with
T M = 2^106 + c (M odd of 54 bits, c small), r^2 = X 2^e with M^2 = X 2^q + c."""
import math

import numpy as np
import pytest

import ahmed_gb300 as A

FOUR_PI = 4.0 * math.pi
# c, T
HARD_T = [(-1, 9007199254740991), (-2, 5276938686109394), (-2, 5359079149933474), (-2, 5852518495683566),
          (-2, 4797136447748302), (-2, 8480179861092514), (-2, 6583997076838894), (-2, 8716460134775102),
          (-2, 5017593869129758), (-2, 7440678027627698), (-2, 4543885306550786), (-4, 5440503800133692),
          (-4, 9002296740580796), (-4, 4691463364816860), (-9, 9007199254740989), (-16, 7111558598256016),
          (-16, 5497283260653072), (-20, 4713086531278084), (-25, 9007199254740987)]


def _next(x, k):
    for _ in range(abs(k)):
        x = math.nextafter(x, math.inf if k > 0 else 0.0)
    return x


def _roots(c, q):
    """M mod 2^q with M^2 = c (mod 2^q), for c = 1 (mod 8)."""
    r = {x for x in range(8) if (x * x - c) % 8 == 0}
    for k in range(4, q + 1):
        h = 1 << (k - 1)
        r = {x % h + j * h for x in r for j in (0, 1) if ((x % h + j * h) ** 2 - c) % (2 * h) == 0}
    return r


def squared_distances():
    """Values of r^2."""
    out = set()
    for c, T in HARD_T:
        assert (2**106 + c) % T == 0
        for e in (-50, -49, -48, -47):
            t = math.ldexp(float(T), e)
            for k in range(-3, 4):
                r = _next(t / FOUR_PI, k)
                if FOUR_PI * r == t:
                    out |= {x for x in (_next(r * r, j) for j in range(-6, 7)) if math.sqrt(x) == r}
    for q in (54, 55):
        for c in range(-95, 96, 8):
            for s in _roots(c, q):
                for M in range(s, 2**54, 2**q):
                    X = (M * M - c) >> q
                    if M >= 2**53 and 2**52 <= X < 2**53:
                        out |= {math.ldexp(float(X), q - 108), math.ldexp(float(X), q - 106)}
    return sorted(out)


def _pair(x, rng):
    """dx, dy with fl(fl(dx dx) + fl(dy dy)) = x."""
    for _ in range(10000):
        dx = math.sqrt(x) * rng.uniform(0.3, 0.95)
        dy = math.sqrt(x - dx * dx)
        if dx * dx + dy * dy == x:
            return dx, dy
    raise AssertionError(x)


def test_the_hard_distances_exist():
    x = squared_distances()
    assert len(x) > 100
    rng = np.random.default_rng(0)
    for v in x[::7]:
        _pair(v, rng)


@pytest.mark.gpu
@pytest.mark.parametrize("cplx", [False, True])
def test_entries_equal_the_host(cplx):
    rng = np.random.default_rng(1)
    X = squared_distances() + [float(v) for v in rng.uniform(0.01, 4.0, 200)]
    bad = []
    for x in X:
        dx, dy = _pair(x, rng)
        H = A.HMatrix(np.array([[0.0, 0.0, 0.0], [dx, dy, 0.0]]), "bbx", bmin=8)
        assert H.nleaves == 1
        if cplx:  # wave number 0: cos = 1, sin = 0
            d = H.helmholtz_assemble(0.0, 1.0, 1e-6).helm_leaf_data(0).real
        else:
            H.matgenGeH_omp(1.0, 1e-6)
            d = H.leaf_data(0)
        want = 1.0 / (FOUR_PI * math.sqrt(x))
        if not (d[1] == want and d[2] == want):
            bad.append((x.hex(), float(d[1]).hex(), want.hex()))
        H.close()
    assert not bad, bad
