"""The rule for the Hessian assembly's launch: a plan's tuning decides the CTA shape at
every size, and the number of lanes (hence the order of the sums) never depends on it."""
import ctypes as C
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SMS = 152


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("shape") / "shape.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "hess_shape_harness.cpp"),
                    "-o", so], check=True)
    lib = C.CDLL(so)

    def call(vertices, cheap, tuned):
        out = (C.c_int * 2)()
        lib.shape(C.c_longlong(vertices), C.c_longlong(-(-vertices // 128)), C.c_longlong(SMS), cheap, tuned, out)
        return tuple(out)
    return call


SIZES = [1, 1000, 128 * SMS, 128 * SMS + 1, 190 * SMS, 190 * SMS + 1, 42875, 3 * 128 * SMS, 3 * 128 * SMS + 1, 912673]


@pytest.mark.parametrize("vertices", SIZES)
@pytest.mark.parametrize("cheap", [0, 1])
def test_the_tuning_decides_the_shape_only(shape, vertices, cheap):
    _, lanes = shape(vertices, cheap, 0)
    for tuned in (64, 128):
        assert shape(vertices, cheap, tuned) == (tuned, lanes)


def test_untuned(shape):
    assert [shape(v, 1, 0) for v in SIZES] == [(64, 4)] * 3 + [(64, 2)] * 2 + [(128, 1)] * 3 + [(64, 2)] * 2
    assert all(shape(v, 0, 0) == (64, 4 if v <= 128 * SMS else 2) for v in SIZES)
