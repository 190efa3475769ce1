"""The rules of the dense refinement's steps at their boundaries."""
import ctypes
import math
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    so = tmp_path_factory.mktemp("ir") / "ir.so"
    subprocess.run([cxx, "-std=c++17", "-O2", "-shared", "-fPIC", "-o", str(so),
                    str(ROOT / "tests" / "host" / "ir_tolerance_host.cpp")], check=True)
    L = ctypes.CDLL(str(so))
    L.ir_limit.argtypes, L.ir_limit.restype = [ctypes.c_double, ctypes.c_int], ctypes.c_double
    L.ir_done.argtypes = [ctypes.c_double] * 2 + [ctypes.c_int]
    return L


def test_columns_of_a_step(lib):
    assert lib.ir_limit(3.0, 1) == pytest.approx(3e-6)
    for k in (2, 3, 60):
        assert lib.ir_limit(3.0, k) == pytest.approx(3e-4)


def test_one_step_beyond_the_tolerance(lib):
    assert not lib.ir_done(1.0, 1.1, 0) and not lib.ir_done(1.0, 1.1, 1)
    assert not lib.ir_done(1.0, 0.9, 0) and lib.ir_done(1.0, 0.9, 1)
    assert not lib.ir_done(1.0, 0.051, 0) and lib.ir_done(1.0, 0.05, 0) and lib.ir_done(1.0, 0.0, 0)


def test_degenerate_residuals(lib):
    for rn in (math.inf, math.nan):
        assert not lib.ir_done(1e-12, rn, 1)
    assert lib.ir_done(0.0, 0.0, 0)
