"""The inner tolerance of a refinement step at the boundaries of its rule."""
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
    L.ir_inner.argtypes, L.ir_inner.restype = [ctypes.c_double] * 2, ctypes.c_double
    L.ir_done.argtypes = [ctypes.c_double] * 2 + [ctypes.c_int]
    return L


@pytest.mark.parametrize("need", [1e-13, 1e-12, 9.99e-9, 1.01e-8, 1.9e-8, 2.1e-8, 3.9e-7, 4.1e-7, 1e-6, 1e-4, 1e-2, 0.5])
def test_steps_towards_the_tolerance(lib, need):
    t = lib.ir_inner(need, 1.0)
    assert 2e-8 <= t <= 1e-6
    assert t <= 0.02 * need or t == 2e-8 or need < 1e-8  # a fiftieth, as far as a step goes
    assert lib.ir_inner(3 * need, 3.0) == pytest.approx(t)


def test_one_step_beyond_the_tolerance(lib):
    assert lib.ir_inner(1.0, 0.9) == lib.ir_inner(1.0, 1.0) == 1e-4
    assert not lib.ir_done(1.0, 1.1, 0) and not lib.ir_done(1.0, 1.1, 1)
    assert not lib.ir_done(1.0, 0.9, 0) and lib.ir_done(1.0, 0.9, 1)
    assert not lib.ir_done(1.0, 0.031, 0) and lib.ir_done(1.0, 0.03, 0) and lib.ir_done(1.0, 0.0, 0)


def test_degenerate_residuals(lib):
    for rn in (math.inf, math.nan):
        assert lib.ir_inner(1e-12, rn) == 1e-6
        assert not lib.ir_done(1e-12, rn, 1)
    assert lib.ir_inner(0.0, 1.0) == 1e-6 and lib.ir_done(0.0, 0.0, 0)
