"""The 9x9 eigen-solver of the PSD projection, compiled for the host, against numpy.

Matrices with entries of order one: random, diagonal, zero, decoupled into
blocks, with repeated eigenvalues, with off-diagonals around the negligibility
threshold and far below it, and rank one."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("eig9") / "eig9.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "eig9_harness.cpp"), "-o", so],
                   check=True)
    return C.CDLL(so)


def _matrices(kind, rng):
    n = 200
    Q = np.linalg.qr(rng.standard_normal((n, 9, 9)))[0]
    A = rng.uniform(-1, 1, (n, 9, 9))
    A = 0.5 * (A + A.transpose(0, 2, 1))
    if kind == "diagonal":
        A = A * np.eye(9)
    elif kind == "zero":
        A = np.zeros((1, 9, 9))
    elif kind == "blocks":
        A[:, :4, 4:] = A[:, 4:, :4] = 0.0
        A[:, 4:6, 6:] = A[:, 6:, 4:6] = 0.0
    elif kind == "repeated":
        L = rng.choice([-0.5, 0.0, 1.0], (n, 9))
        A = (Q * L[:, None, :]) @ Q.transpose(0, 2, 1)
    elif kind == "tiny":
        s = 10.0 ** rng.uniform(-22, -6, (n, 1, 1))
        A = A * np.eye(9) + A * s
    elif kind == "rank1":
        A = Q[:, :, :1] * Q[:, None, :, 0]
    return 0.5 * (A + A.transpose(0, 2, 1))


@pytest.mark.parametrize("kind", ["random", "diagonal", "zero", "blocks", "repeated", "tiny", "rank1"])
@pytest.mark.parametrize("dtype,fn,tol", [(np.float32, "eig9_f32", 9 * 1.2e-7 * 4), (np.float64, "eig9_f64", 1e-13)])
def test_eigen_decomposition(lib, kind, dtype, fn, tol):
    A = np.ascontiguousarray(_matrices(kind, np.random.default_rng(3)), dtype)
    n = len(A)
    d, Z = np.zeros((n, 9), dtype), np.zeros((n, 9, 9), dtype)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    getattr(lib, fn)(n, p(A), p(d), p(Z))
    W = Z.astype(np.float64).transpose(0, 2, 1)  # eigenvectors in columns
    R = (W * d.astype(np.float64)[:, None, :]) @ W.transpose(0, 2, 1) - A
    assert np.abs(R).max() <= tol
    assert np.abs(W.transpose(0, 2, 1) @ W - np.eye(9)).max() <= tol
    assert np.abs(np.sort(d, 1) - np.linalg.eigvalsh(A.astype(np.float64))).max() <= tol
