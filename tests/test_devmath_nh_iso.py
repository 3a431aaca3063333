"""The isochoric Neo-Hookean energy at small and at large volume ratios, compiled for
the host, against 60 digits: ln J has to be as good as log1p gives it where J - 1 is
far above it, not the difference of two numbers of the size of J."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

mp = pytest.importorskip("mpmath")
HERE = os.path.dirname(os.path.abspath(__file__))
EPS = 2.0 ** -53
PV = np.array([1.3, 0.0])  # the shear part; the volume's is (J - 1)^2


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("iso") / "iso.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "nh_iso_harness.cpp"), "-o", so],
                   check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("stretch", [1.001, 1.3, 1.7, 30.0, 1e4, 1e9, 1e12])
def test_energy(lib, stretch):
    rng = np.random.default_rng(1)
    n = 40
    H = np.zeros((n, 3, 3))
    H[:, 0, 0] = stretch * rng.uniform(1, 1.4, n) - 1  # one direction stretched, the others nearly kept
    H[:, 1, 1], H[:, 2, 2] = rng.uniform(-0.05, 0.05, (2, n))
    H[:, 0, 1] = rng.uniform(-0.1, 0.1, n)
    flat = np.ascontiguousarray(H.transpose(0, 2, 1)).reshape(n, 9)
    psi = np.empty(n)
    lib.nh_iso(n, *[a.ctypes.data_as(C.c_void_p) for a in (flat, PV, psi)])
    for i in range(n):
        with mp.workdps(60):
            Hm = mp.matrix(H[i].tolist())
            F = Hm + mp.eye(3)
            J = mp.det(F)
            I1 = sum(F[a, b] ** 2 for a in range(3) for b in range(3))
            ref = float(PV[0] * (J ** (mp.mpf(-2) / 3) * I1 - 3))
            y = -2 * mp.log(J) / 3
            e, j = mp.expm1(y), J - 1
            tr, n2 = Hm[0, 0] + Hm[1, 1] + Hm[2, 2], sum(Hm[a, b] ** 2 for a in range(3) for b in range(3))
            # the formula's terms: 3 (e - y), 2 (j - ln J), 2 (q2 + det) = 2 (j - tr H), |H|^2, e (2 tr H + |H|^2)
            terms = 3 * abs(e - y) + 2 * abs(j - mp.log(J)) + 2 * abs(j - tr) + n2 + abs(e) * (2 * abs(tr) + n2)
            # ln J through J: a few roundings of J - 1's parts, carried into J^-2/3 I1
            dj = float((abs(tr) + abs(j - tr)) / J)
            tol = EPS * PV[0] * (16 * float(terms) + 8 * (dj + float(abs(y)) + 1) * float(abs(1 + e) * I1))
        assert abs(psi[i] - ref) <= tol, (psi[i], ref, tol)
