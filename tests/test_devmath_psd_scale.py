"""The PSD projection at the ends of the float range. An element whose matrix is tiny
against the tolerance, down to the smallest floats, has every eigenvalue become the
tolerance, whatever power of two the eigen-solver scales by; and a huge one is
projected as its multiple of ordinary size."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("psd") / "psd.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "psd_scale_harness.cpp"),
                    "-o", so], check=True)
    return C.CDLL(so)


def _element(lib, scale, tol):
    rng = np.random.default_rng(4)
    F = (np.eye(3) + 0.4 * rng.uniform(-1, 1, (3, 3))).astype(np.float32).T.ravel().copy()
    pv = np.array([1.0, 0.7]).astype(np.float32) * np.float32(scale)
    dphi = rng.uniform(-1, 1, 9).astype(np.float32)
    K, Q = np.zeros(45, np.float32), np.zeros(12, np.float32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    lib.psd_nodes(p(F), p(pv), p(dphi), C.c_float(tol), p(K), p(Q))
    assert np.isfinite(K).all()
    return K, Q


@pytest.mark.parametrize("exponent", [60, 96, 110, 122])
def test_a_huge_matrix(lib, exponent):
    one, big = _element(lib, 1.0, 1e-3)[0], _element(lib, 2.0 ** exponent, 1e-3 * 2.0 ** exponent)[0]
    assert np.abs(np.ldexp(big.astype(np.float64), -exponent) - one).max() <= 4e-7 * np.abs(one).max()


@pytest.mark.parametrize("scale", [0.0, 1e-8, 1e-20, 1e-37, 1e-39, 1e-42, 1.5e-45])
@pytest.mark.parametrize("tol", [1e-6, 1e-3, 1.0, 1e3, 1e6])
def test_a_tiny_matrix_becomes_the_tolerance(lib, scale, tol):
    if scale > 1e-6 * tol:
        pytest.skip("not tiny")
    K, Q = _element(lib, scale, tol)
    full = np.zeros((9, 9))
    full[np.tril_indices(9)] = K
    full = full + np.tril(full, -1).T
    q = Q.reshape(4, 3)[1:].astype(np.float64)
    ref = tol * np.kron(q @ q.T, np.eye(3))
    # nine products of three roundings each, of entries up to the tolerance
    assert np.abs(full - ref).max() <= 9 * 3 * 6e-8 * tol + 1e-6 * tol
