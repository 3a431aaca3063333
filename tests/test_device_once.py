"""Kernel attributes are set once per device, not once per process: a context on a
second device needs its own, and a flag that the first one set would leave its
launches without their shared memory."""
import ctypes as C
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "bartels_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("once") / "once.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread",
                    os.path.join(HERE, "device_once_harness.cpp"), "-o", so], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("done,device,pending", [([], 0, 1), ([0], 0, 0), ([0], 1, 1), ([1], 0, 1), ([0, 7], 7, 0),
                                                 ([63], 63, 0), ([64], 64, 1), ([63], 64, 1)])
def test_each_device_has_its_own_flag(lib, done, device, pending):
    arr = (C.c_int * max(len(done), 1))(*done)
    assert lib.pending_after(len(done), arr, device) == pending


def test_threads(lib):
    assert lib.pending_after_threads() == 0


def test_no_source_keeps_attributes_behind_a_process_wide_flag():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, f)).read()
            assert not re.search(r"static bool \w+ = false;[^}]*?cudaFuncSetAttribute", text), f
