"""The table-driven j - log1p(j) and the corotational law through the polar
rotation, compiled for the host, against higher precision.

j over the table's rows, their boundaries, both sides of its end and of zero;
F near rest, far from it, turned by up to 180 degrees about each axis (every
branch of the quaternion), with singular values on both sides of the ratio up to
which the rotation is used, scaled, inverted and singular."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

mp = pytest.importorskip("mpmath")
HERE = os.path.dirname(os.path.abspath(__file__))
EPS = 2.0 ** -53
PV = np.array([1.5, 0.7])  # lambda, mu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fp64") / "laws.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "fp64_laws_harness.cpp"),
                    "-o", so], check=True)
    return C.CDLL(so)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def test_j_minus_log1p(lib):
    rng = np.random.default_rng(0)
    k = np.arange(-44, 45) / 64
    edges = np.concatenate([k, k + 1 / 128, np.nextafter(k + 1 / 128, 1), k - 1 / 128])
    j = np.concatenate([edges, [0.6875, -0.6875, np.nextafter(0.6875, 0), np.nextafter(-0.6875, 0), 0.0, 5.0, -0.99, 1e9],
                        rng.uniform(-0.95, 3, 500), 10.0 ** rng.uniform(-12, 0, 300), -(10.0 ** rng.uniform(-12, -0.1, 300))])
    out = np.empty_like(j)
    lib.jlog(len(j), _p(j), _p(out))
    with mp.workdps(60):
        ref = np.array([float(mp.mpf(float(x)) - mp.log(1 + mp.mpf(float(x)))) for x in j])
    # beyond the table j - log1p(j) >= 0.16, of terms up to |j| and |log1p(j)|; within it the three parts are at most
    # a few times the result, each with a few roundings
    assert (np.abs(out - ref) <= 16 * EPS * np.maximum(np.abs(ref), np.where(np.abs(j) < 0.6875, 0, np.abs(j)))).all()
    for bad in (np.nan, -1.5, -np.inf):
        x = np.array([bad])
        lib.jlog(1, _p(x), _p(out))
        assert np.isnan(out[0])


def _rot(rng, n, lo=0.0, hi=np.pi, axis=None):
    v = rng.standard_normal((n, 3)) if axis is None else np.eye(3)[axis] + 0.05 * rng.standard_normal((n, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    t = rng.uniform(lo, hi, n)[:, None, None]
    K = np.zeros((n, 3, 3))
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -v[:, 2], v[:, 1], -v[:, 0]
    K -= K.transpose(0, 2, 1)
    return np.eye(3) + np.sin(t) * K + (1 - np.cos(t)) * (K @ K)


def _samples(kind, rng, n=60):
    Q, V = _rot(rng, n), _rot(rng, n)
    s = rng.uniform(0.6, 1.6, (n, 3))
    if kind == "rest":
        return np.eye(3) + 10.0 ** rng.uniform(-9, -3, (n, 1, 1)) * rng.uniform(-1, 1, (n, 3, 3))
    if kind.startswith("turn"):
        Q = _rot(rng, n, 2.6, np.pi, int(kind[4])) @ V
    elif kind == "ratio":
        s[:, 0], s[:, 2] = 1.0, rng.uniform(0.09, 0.13, n)
    elif kind == "equal":
        s[:] = rng.uniform(0.5, 2, (n, 1))
    elif kind == "scaled":
        s *= 10.0 ** rng.uniform(-5, 5, (n, 1))
    elif kind == "inverted":
        s[:, 2] *= -1
    elif kind == "flat":
        s[:, 2] = rng.uniform(0, 1e-3, n)
    return (Q * s[:, None, :]) @ V.transpose(0, 2, 1)


@pytest.mark.parametrize("kind,used", [("rest", 1), ("any", 1), ("turn0", 1), ("turn1", 1), ("turn2", 1), ("ratio", None),
                                       ("equal", 1), ("scaled", 1), ("inverted", 0), ("flat", 0)])
def test_corotational(lib, kind, used):
    M = _samples(kind, np.random.default_rng(5))
    n = len(M)
    F = np.ascontiguousarray(M.transpose(0, 2, 1)).reshape(n, 9)
    psi, P, polar = np.empty(n), np.empty((n, 9)), np.empty(n, np.int32)
    lib.corot(n, _p(F), _p(PV), _p(psi), _p(P), _p(polar))
    if used is not None:
        assert (polar == used).all()
    elif kind == "ratio":
        assert polar.any() and not polar.all()
    for i in range(n):
        if kind in ("inverted", "flat"):
            U, S, Vt = np.linalg.svd(M[i])
            sg = np.linalg.det(U) * np.linalg.det(Vt)
            S2 = S * np.array([1, 1, np.sign(sg)])
            e = PV[1] * ((S2 - 1) ** 2).sum() + 0.5 * PV[0] * (S2.sum() - 3) ** 2
            assert abs(psi[i] - e) <= 1e-11 * abs(e)
            continue
        with mp.workdps(40):
            Fm = mp.matrix(M[i].tolist())
            R = Fm / mp.cbrt(mp.det(Fm))  # the iteration converges quadratically from order one
            for _ in range(12):
                R = (R + (R ** -1).T) / 2
            E = Fm - R
            tr = sum(R[a, b] * E[a, b] for a in range(3) for b in range(3))
            e2 = sum(E[a, b] ** 2 for a in range(3) for b in range(3))
            ref = float(mp.mpf(PV[1]) * e2 + mp.mpf(PV[0]) * tr * tr / 2)
            Pm = 2 * mp.mpf(PV[1]) * E + mp.mpf(PV[0]) * tr * R
            Pr = np.array([[float(Pm[a, b]) for b in range(3)] for a in range(3)])
            tr, e2 = float(tr), float(e2)
        s0 = max(np.abs(M[i]).max(), 1.0)
        # R and F - R to a few roundings of their entries (10 EPS s0 each); tr gathers nine of them
        d = 10 * EPS * s0
        # an error in R turns into P through (2 mu + lambda |tr|) d, in tr through 9 d
        tol = (2 * PV[1] + PV[0] * (9 + abs(tr))) * d * 4
        assert np.abs(P[i].reshape(3, 3).T - Pr).max() <= tol
        tol = (2 * PV[1] * np.sqrt(e2) * 3 + 9 * PV[0] * abs(tr)) * d + (9 * PV[1] + 41 * PV[0]) * d * d + 8 * EPS * ref
        # the rotation used is off by up to 1e-10, in which the energy is second order
        assert abs(psi[i] - ref) <= tol + 1e-20 * (PV[0] + PV[1]) * s0 * s0
