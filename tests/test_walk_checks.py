"""Parts of the per-ray walk against their plain forms, on the CPU
(tests/kernel_host/walk_checks.cpp includes the kernels' ytgb_ray.cuh)."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
HERE = Path(__file__).resolve().parent / "kernel_host"


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    out = tmp_path_factory.mktemp("walk_checks") / "libwalk_checks.so"
    cuda_inc = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", f"-I{ROOT / 'include'}",
                    f"-I{ROOT / 'yt_gb300' / 'csrc'}", f"-I{cuda_inc}", str(HERE / "walk_checks.cpp"), "-o",
                    str(out)], check=True)
    return C.CDLL(str(out))


@pytest.mark.parametrize("aim,least", [(0, 0.5), (1, 0.1), (2, 0.0), (3, 0.0)])
def test_setup_by_entry_face_equals_general(checks, aim, least):
    """Every walk the entry-face set-up decides has the general set-up's enter
    t, tmax, cell and position, bit for bit; and it does decide the common
    walks."""
    n = 200_000
    out = (C.c_longlong * 3)()
    checks.check_setup(C.c_longlong(n), aim, C.c_ulonglong(11 + aim), out)
    decided, left, wrong = out
    assert wrong == 0
    assert decided + left == n and decided >= least * n


@pytest.mark.parametrize("steps", [1, 7, 64, 2000])
@pytest.mark.parametrize("ties", [0, 1])
def test_runs_of_steps_equal_float64_adds(checks, steps, ties):
    """tmax after every step of a run is the float64 sum's bits, across
    binades and exact halves, and the step that leaves the brick is never
    inside a run."""
    n = 2_000_000 // (steps + 10)
    looks = C.c_longlong()
    checks.check_runs.restype = C.c_longlong
    bad = checks.check_runs(C.c_longlong(n), steps, ties, C.c_ulonglong(5 + steps), C.byref(looks))
    assert bad == 0
    assert looks.value > 0


def test_octree_values_equal_float64(checks):
    """Slab midpoints, float32 pairs and dt formed on the integer pipe are the
    float64 operations' (float32 ties, which the pair rounds the other way,
    still sum to the value)."""
    checks.check_octree_values.restype = C.c_longlong
    assert checks.check_octree_values(C.c_longlong(2_000_000), C.c_ulonglong(3)) == 0
