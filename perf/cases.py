"""The work that users of this framework have it do, as cases that can be timed and compared.

Kinds of cases (each through the package's public entry points):
  product    y = A x (or A^T x) with an assembled Laplace H-matrix kept by the program, for one to
             64 vectors, in each storage that products take; single-precision storages hand
             their result on in single precision, as the mblock<float> products do
  zproduct   the same for the complex Helmholtz H-matrix, A x and A^H x
  assemble   ACA assembly of every leaf of a cluster tree, then one product
  zassemble  the same for the Helmholtz kernel
  gmres      a restarted GMRES solve of many right-hand sides with one H-matrix
  batch      one GMRES solve of many uneven H-matrices together
  predictor  training of the ACA-rank network from (feature, rank) pairs, then its predictions

Vectors are in the cluster ordering of the bounding-box tree.
"""
import math

import numpy as np
import torch

import ahmed_gb300 as A
from ahmed_gb300.rank_predictor import RankPredictor

ETA = 0.8
EPS = 1e-6
FOUR_PI = 4.0 * math.pi


# -- the cases -------------------------------------------------------------

def listed():
    return [
        # the smallest call in earnest: one vector, 4096 sphere points, plain form; an iterative
        # solver of the user's own calls this once per step, so launches and latency count
        dict(name="product-fp64-4096-p1", kind="product", precision="fp64", op="n", shape="sphere", n=4096, leaf=32, p=1),
        # the plain form at the ordinary size: 65,536 sphere points, 16 vectors
        dict(name="product-fp64-65536-p16", kind="product", precision="fp64", op="n", shape="sphere", n=65536, leaf=32, p=16),
        # the adjoint of the plain form, odd number of points and vectors (normal equations, BiCG)
        dict(name="adjoint-fp64-20011-p5", kind="product", precision="fp64", op="t", shape="ellipsoid", n=20011, leaf=32, p=5),
        # the single-precision form at the ordinary size
        dict(name="product-fp32-65536-p16", kind="product", precision="fp32", op="n", shape="sphere", n=65536, leaf=32, p=16),
        # the large product: cube surface, leaf 64, a full block of 64 vectors
        dict(name="product-fp32-131072-p64", kind="product", precision="fp32", op="n", shape="cube", n=131072, leaf=64, p=64),
        # Helmholtz, single-precision leaves, 16 vectors: the inner product of a scattering solve
        dict(name="zproduct-c64-16384-p16", kind="zproduct", precision="fp32", op="n", shape="sphere", n=16384, leaf=32, p=16, k=10.0),
        # Helmholtz adjoint in the plain form, odd sizes, few vectors
        dict(name="zadjoint-c128-6007-p3", kind="zproduct", precision="fp64", op="h", shape="sphere", n=6007, leaf=32, p=3, k=5.0),
        # set-up of the ordinary H-matrix: every program starts with it
        dict(name="assemble-65536", kind="assemble", shape="sphere", n=65536, leaf=32, p=1),
        # set-up of a Helmholtz H-matrix, once per wave number
        dict(name="zassemble-12289", kind="zassemble", shape="sphere", n=12289, leaf=32, p=1, k=8.0),
        # GMRES(50) with single-precision inner solves and FP64 refinement, 16 systems at once
        dict(name="gmres-fp32-32768-p16", kind="gmres", precision="fp32", shape="cube", n=32768, leaf=64, p=16),
        # many uneven systems solved together, one right-hand side each (GMRES(30))
        dict(name="batch-gmres-fp32-16", kind="batch", precision="fp32", count=16, nmin=2048, nmax=16384, leaf=32),
        # the rank network of a run's first matrices: training, then predictions for the next one
        dict(name="predictor-16384", kind="predictor", n=16384, epochs=2, batch=1024, npredict=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product"] * 5 + ["zproduct"] * 2 + ["assemble", "zassemble", "gmres", "batch", "predictor"])
    shape = rng.choice(["sphere", "ellipsoid", "cube"])
    leaf = rng.choice([32, 32, 64])
    if kind == "product":
        precision, op = rng.choice([("fp64", "n"), ("fp64", "t"), ("fp32", "n"), ("fp32", "n"), ("bf16", "n")])
        plain = precision == "fp64"
        return dict(kind=kind, precision=precision, op=op, shape=shape, leaf=leaf,
                    n=_log_int(rng, 1024, 65536 if plain else 100000),
                    p=rng.choice([1, 2, 3, 4, 5, 8, 11, 16] + ([] if plain else [17, 32, 33, 64])))
    if kind == "zproduct":
        return dict(kind=kind, precision=rng.choice(["fp32", "fp64"]), op=rng.choice(["n", "n", "h"]), shape=shape,
                    leaf=leaf, n=_log_int(rng, 1024, 16384), p=rng.choice([1, 2, 3, 4, 5, 8, 16]),
                    k=round(rng.uniform(1.0, 12.0), 3))
    if kind == "assemble":
        return dict(kind=kind, shape=shape, leaf=leaf, n=_log_int(rng, 2048, 65536), p=1)
    if kind == "zassemble":
        return dict(kind=kind, shape=shape, leaf=leaf, n=_log_int(rng, 1024, 12289), p=1, k=round(rng.uniform(1.0, 8.0), 3))
    if kind == "gmres":
        return dict(kind=kind, precision=rng.choice(["fp32", "fp64"]), shape=shape, leaf=leaf,
                    n=_log_int(rng, 2048, 32768), p=rng.choice([1, 2, 4, 7, 16]))
    if kind == "batch":
        return dict(kind=kind, precision=rng.choice(["fp32", "fp64"]), count=rng.randint(4, 15), nmin=rng.randint(1024, 3000),
                    nmax=rng.randint(6000, 16384), leaf=32)
    n = _log_int(rng, 2048, 60000)
    return dict(kind="predictor", n=n, epochs=2 if n <= 20000 else 1, batch=rng.choice([512, 1024]), npredict=_log_int(rng, 2000, 100000))


# -- inputs ----------------------------------------------------------------

def _points(shape, n, rng):
    """n random points on a closed surface."""
    if shape == "cube":
        face, uv = rng.integers(0, 6, n), rng.random((n, 2))
        p = np.empty((n, 3))
        for a in range(3):
            sel = face // 2 == a
            others = [b for b in range(3) if b != a]
            p[sel, a] = face[sel] % 2
            p[np.ix_(sel, others)] = uv[sel]
        return p
    g = rng.standard_normal((n, 3))
    g /= np.linalg.norm(g, axis=1, keepdims=True)
    return g * np.array([1.0, 0.5, 0.25]) if shape == "ellipsoid" else g


def _vectors(rng, p, n, device, cplx=False):
    """p right-hand sides as rows (column-major n x p)."""
    v = rng.standard_normal((p, n))
    if cplx:
        v = v + 1j * rng.standard_normal((p, n))
    return torch.from_numpy(v[0] if p == 1 else v).to(device)


def _sizes(case):
    rng = np.random.default_rng(2)
    return [int(round(math.exp(u))) for u in rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["count"])]


def _features(n, rng):
    """Geometric features of admissible leaves and their ranks, spread as on surface meshes."""
    level = rng.integers(2, 9, n)
    f = np.empty((n, 8), np.float32)
    f[:, 0] = -0.35 * level + rng.normal(0.0, 0.1, n)
    f[:, 1] = f[:, 0] + rng.normal(0.0, 0.15, n)
    f[:, 2] = f[:, 0] + rng.uniform(0.2, 1.6, n)
    f[:, 3] = np.exp(np.minimum(f[:, 0], f[:, 1]) - f[:, 2])
    f[:, 4] = math.log(16384) - 0.69 * level + rng.normal(0.0, 0.2, n)
    f[:, 5] = f[:, 4] + rng.normal(0.0, 0.2, n)
    f[:, 6] = rng.choice([1.0, 5.0, 12.0], n) * np.exp(np.maximum(f[:, 0], f[:, 1]))
    f[:, 7] = 6.0
    r = np.round(3.0 + 6.0 * f[:, 3] + 0.6 * f[:, 6] + 0.4 * f[:, 4] + rng.normal(0.0, 0.5, n))
    return f, np.maximum(r, 1.0).astype(np.float32)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, dev = case["kind"], torch.device("cuda:0")
    s = dict(case)
    if kind == "predictor":
        s["F"], s["ranks"] = _features(case["n"], rng)
        s["Fnew"], _ = _features(case["npredict"], rng)
        s["seed"] = seed
        return s
    if kind == "batch":
        mats = []
        for q, n in enumerate(_sizes(case)):
            P = _points(("sphere", "ellipsoid", "cube")[q % 3], n, rng)
            mats.append(A.HMatrix(P, "bbx", bmin=case["leaf"], eta=ETA).matgenGeH_omp(0.5 * A.min_nn(P), EPS))
        s["mats"] = mats
        s["B"] = A.HBatch(mats, case["precision"])
        s["b"] = _vectors(rng, 1, int(s["B"].n), dev)
        s["x"] = torch.zeros_like(s["b"])
        return s
    n, p = case["n"], case["p"]
    P = _points(case["shape"], n, rng)
    H = A.HMatrix(P, "bbx", bmin=case["leaf"], eta=ETA)
    s["H"] = H
    # solves: the diagonal of half the smallest distance makes the matrix positive definite
    s["h"] = 0.5 * A.min_nn(P) if kind == "gmres" else A.mean_nn(P)
    s["X"] = _vectors(rng, p, n, dev, kind in ("zproduct", "zassemble"))
    s["Y"] = torch.zeros_like(s["X"])
    if kind in ("product", "gmres"):
        H.matgenGeH_omp(s["h"], EPS)
        H.prepare(case["precision"])
    elif kind == "zproduct":
        H.helmholtz_assemble(case["k"], s["h"], EPS)
    return s


# -- one pass --------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "predictor":
        net = RankPredictor(seed=s["seed"])
        losses = net.fit(s["F"], s["ranks"], epochs=s["epochs"], batch=s["batch"], seed=s["seed"])
        out = dict(losses=losses, params=net.params, log_ranks=net.predict_log(s["Fnew"]))
        net.close()
        return out
    if kind == "batch":
        s["x"].zero_()
        s["B"].gmres(s["b"], s["x"], 1e-10, 30, 300)
        return s["x"]
    H, X, Y = s["H"], s["X"], s["Y"]
    Y.zero_()
    if kind == "gmres":
        H.GMRes(X, Y, 1e-10, 50, 500, precision=s["precision"])
        return Y
    if kind == "assemble":
        H.matgenGeH_omp(s["h"], EPS)
        return H.mltaGeHVec(1.0, X, Y)
    if kind == "zassemble":
        H.helmholtz_assemble(s["k"], s["h"], EPS)
        return H.mltaGeHVec(1.0, X, Y)
    if s["op"] == "n":
        H.mltaGeHVec(1.0, X, Y, precision=s["precision"])
    else:
        H.mltaGeHhVec(1.0, X, Y, precision=s["precision"])
    if s["precision"] == "fp64":
        return Y
    return Y.to(torch.complex64 if kind == "zproduct" else torch.float32)


# -- what a pass cannot do without -----------------------------------------

def _leaf_values(case, n):
    """Values that the leaves of an H-matrix of n surface points hold, about (eps 1e-6, eta 0.8)."""
    per_point = 480.0 * math.log2(n) - 2400.0 if case["leaf"] == 64 else 452.0 * math.log2(n) - 3260.0
    per_point *= {"sphere": 1.0, "cube": 1.04, "ellipsoid": 0.98}[case.get("shape", "sphere")]
    if "k" in case:
        per_point *= 1.0 + 0.018 * case["k"]
    return n * min(per_point, float(n))


def work(case):
    kind = case["kind"]
    if kind == "predictor":
        passes = case["n"] * case["epochs"]
        weights = 8 * 64 + 64 * 64 + 64
        return {"bytes": 36 * case["n"] + 36 * case["npredict"], "flops": 2 * weights * (4 * passes + case["npredict"])}
    if kind == "batch":
        mean = (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        values = case["count"] * _leaf_values(case, mean)
        steps = 20
        return {"bytes": steps * 4 * values + 16 * case["count"] * mean, "flops": 2 * steps * values}
    n, p = case["n"], case["p"]
    values = _leaf_values(case, n)
    if kind == "gmres":
        size = 8 if case["precision"] == "fp64" else 4
        steps = 14
        return {"bytes": steps * size * values + 16 * n * p, "flops": 2 * steps * values * p}
    if kind in ("assemble", "zassemble"):
        z = kind == "zassemble"
        # the leaves written once; an evaluation (about 12 operations) and one update per value
        return {"bytes": (16 if z else 8) * values, "flops": (60 if z else 30) * values}
    z = kind == "zproduct"
    size = {"fp64": 8, "fp32": 4, "bf16": 2}[case["precision"]] * (2 if z else 1)
    wide = (8 if case["precision"] == "fp64" else 4) * (2 if z else 1)
    return {"bytes": size * values + ((16 if z else 8) + wide) * n * p, "flops": (8 if z else 2) * values * p}


# -- 64-bit results of the dense matrices ----------------------------------

def _cluster_order(P, bmin):
    """Positions of the points in the bounding-box cluster tree's ordering: bisection of the
    longest side (the first one where it is within 0.8 of it) at its middle, down to bmin points;
    points past the middle are exchanged with the last ones not yet looked at."""
    order = np.arange(len(P))
    todo = [(0, len(P))]
    while todo:
        b, e = todo.pop()
        o = order[b:e]
        C = P[o]
        lo, hi = C.min(axis=0), C.max(axis=0)
        side = hi - lo
        d = 0 if side[0] > 0.8 * side.max() else int(side.argmax())
        low = C[:, d] < 0.5 * (lo[d] + hi[d])
        nl, n = int(low.sum()), e - b
        new = o.copy()
        holes = np.flatnonzero(~low[:nl])
        tail = np.arange(n - 1, nl - 1, -1)       # looked at from the end
        tlow = low[tail]
        new[holes] = o[tail[tlow]]
        before = np.cumsum(tlow) - tlow           # low points met before this one
        high = tail[~tlow]
        key = 2.0 * before[~tlow] + 1.0
        key[high == nl] = 2.0 * len(holes)        # the last hole, if it is none of the tail's low points
        seq = np.concatenate([holes, high])
        key = np.concatenate([2.0 * np.arange(len(holes)), key])
        new[n - 1:nl - 1 if nl else None:-1] = o[seq[np.argsort(key, kind="stable")]]
        order[b:e] = new
        if nl > bmin and n - nl > bmin:
            todo += [(b, b + nl), (b + nl, e)]
    return order


def _nn(P):
    """Distance of every point to its nearest neighbour."""
    d = torch.empty(len(P), dtype=torch.float64, device=P.device)
    for i in range(0, len(P), 2048):
        r2 = ((P[i:i + 2048, None, :] - P[None, :, :]) ** 2).sum(-1)
        r2[torch.arange(len(r2)), torch.arange(i, i + len(r2))] = math.inf
        d[i:i + 2048] = r2.min(dim=1).values.sqrt()
    return d


def _rows(P, i, j, h, k=None):
    """Rows i to j of the collocation matrix exp(ikr) / (4 pi r)."""
    r = torch.zeros(j - i, len(P), dtype=torch.float64, device=P.device)
    for c in range(3):
        r += (P[i:j, c, None] - P[None, :, c]) ** 2
    r = r.sqrt_()
    r[torch.arange(j - i), torch.arange(i, j)] = h
    return 1.0 / (FOUR_PI * r) if k is None else torch.polar(1.0 / (FOUR_PI * r), k * r)


def _solve(P, h, B):
    """The positive definite system's solution by conjugate gradients in 64 bits, per column of B (n x p)."""
    n = len(P)
    M = torch.empty(n, n, dtype=torch.float64, device=P.device)
    for i in range(0, n, 2048):
        M[i:i + 2048] = _rows(P, i, min(n, i + 2048), h)
    x, r = torch.zeros_like(B), B.clone()
    q, rr = r.clone(), (r * r).sum(0)
    stop = 1e-28 * rr
    for _ in range(500):
        if bool((rr <= stop).all()):
            break
        Mq = M @ q
        a = rr / (q * Mq).sum(0)
        x += a * q
        r -= a * Mq
        new = (r * r).sum(0)
        q = r + (new / rr) * q
        rr = new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "predictor":
        return None  # the order of the samples is the library's own
    rng = np.random.default_rng(seed)
    dev = torch.device("cuda:0")
    if kind == "batch":
        clouds = []
        for q, n in enumerate(_sizes(case)):
            P = _points(("sphere", "ellipsoid", "cube")[q % 3], n, rng)
            clouds.append(torch.from_numpy(P[_cluster_order(P, case["leaf"])]).to(dev))
        b = _vectors(rng, 1, sum(len(P) for P in clouds), dev)
        parts = b.split([len(P) for P in clouds])
        return torch.cat([_solve(P, 0.5 * float(_nn(P).min()), v[:, None])[:, 0] for P, v in zip(clouds, parts)])
    n, p = case["n"], case["p"]
    P = _points(case["shape"], n, rng)
    P = torch.from_numpy(P[_cluster_order(P, case["leaf"])]).to(dev)
    X = _vectors(rng, p, n, dev, kind in ("zproduct", "zassemble"))
    XT = (X[None] if p == 1 else X).T.contiguous()
    d = _nn(P)
    if kind == "gmres":
        Y = _solve(P, 0.5 * float(d.min()), XT).T
        return Y[0] if p == 1 else Y
    Y, h = torch.empty_like(XT), float(d.mean())
    for i in range(0, n, 1024):
        j = min(n, i + 1024)
        M = _rows(P, i, j, h, case.get("k"))
        Y[i:j] = (M.conj() if case.get("op") == "h" else M) @ XT
    Y = Y.T.contiguous()
    return Y[0] if p == 1 else Y
