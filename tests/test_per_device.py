"""The once-per-device record behind the kernels' shared-memory limits, on the
CPU with a fake of the runtime's call: each device its own, a failure tried
again, several threads."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fltk_sph_ice_gb300", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_each_device_once(tmp_path):
    exe = tmp_path / "per_device"
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-pthread", "-I", CSRC,
                        os.path.join(ROOT, "tests", "cpp", "per_device.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_no_limit_is_raised_once_a_process():
    """Every kernel's limit goes through that record."""
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                n = f.read().count("cudaFuncSetAttribute(")
            assert n == (1 if name == "fsph_kernels.cuh" else 0), name
