"""Kernel attributes are set on every device that launches the kernel, not once per process."""
import ctypes
import re
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
    so = tmp_path_factory.mktemp("once") / "once.so"
    subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", "-shared", "-fPIC", "-o", str(so),
                    str(ROOT / "tests" / "host" / "device_once_host.cpp")], check=True)
    return ctypes.CDLL(str(so))


def test_each_device_is_set_up_once(lib):
    for dev in (0, 1, 0, 7, 1, 63, 0, 63):
        assert lib.launch_on(dev, 0) == 0
    assert [lib.set_ups(d) for d in (0, 1, 7, 63, 2)] == [1, 1, 1, 1, 0]


def test_a_failed_set_up_is_tried_again(lib):
    assert lib.launch_on(5, 1) == -1 and lib.launch_on(5, 1) == -1
    assert lib.launch_on(5, 0) == 0 and lib.launch_on(5, 1) == 0
    assert lib.set_ups(5) == 3


def test_devices_beyond_the_remembered_ones_and_threads(lib):
    assert lib.launch_on(64, 0) == 0 and lib.launch_on(64, 0) == 0 and lib.set_ups(64) == 2
    lib.launch_threads(9, 8)
    assert 1 <= lib.set_ups(9) <= 8


def test_no_attribute_is_set_once_per_process():
    for p in sorted((ROOT / "fluidlets_gb300" / "csrc").glob("*.cu")):
        text = p.read_text()
        assert not re.search(r"static\s+bool\s+\w*set\w*\s*=\s*false", text), p.name
        for m in re.finditer(r"cudaFuncSetAttribute", text):
            before = text[:m.start()]
            assert before.rfind("FLG_ONCE_PER_DEVICE(") > before.rfind("\n}\n"), (p.name, before.count("\n") + 1)
