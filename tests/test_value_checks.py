"""The rays' conversions off the float64 pipe against plain casts, on the CPU
(tests/kernel_host/value_checks.cpp includes the kernels' ytgb_ray.cuh)."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
HERE = Path(__file__).resolve().parent / "kernel_host"


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    out = tmp_path_factory.mktemp("value_checks") / "libvalue_checks.so"
    cuda_inc = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{ROOT / 'include'}",
                    f"-I{ROOT / 'yt_gb300' / 'csrc'}", f"-I{cuda_inc}", str(HERE / "value_checks.cpp"), "-o",
                    str(out)], check=True)
    return C.CDLL(str(out))


def test_narrow_is_the_conversion(checks):
    checks.check_narrow.restype = C.c_longlong
    assert checks.check_narrow(C.c_longlong(3_000_000), C.c_ulonglong(7)) == 0


def test_ray_values(checks):
    checks.check_rays.restype = C.c_longlong
    assert checks.check_rays(C.c_longlong(300_000), C.c_ulonglong(8)) == 0
