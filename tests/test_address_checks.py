"""Every form of the per-ray walk over exactly sized arrays, on the CPU
(tests/kernel_host/address_checks.cpp includes the kernels' ytgb_ray.cuh).

Both cell loops -- the run-limited one with sample_many, and the loop with every
test in every step, which the batch kernel takes for several samples, masks,
the light source and other table sets -- read nothing outside a brick's arrays
and do nothing undefined, use no variable before it is set, and form the same
images bit for bit."""
import os
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SRC = Path(__file__).resolve().parent / "kernel_host" / "address_checks.cpp"
SANITIZE = ["-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all"]
BUILDS = {
    "sanitized": [*SANITIZE],
    "sanitized-general": [*SANITIZE, "-DYTGB_GENERAL_LOOP"],
    "pattern": ["-O2", "-ftrivial-auto-var-init=pattern"],
    "zero": ["-O2", "-ftrivial-auto-var-init=zero"],
    "pattern-general": ["-O2", "-ftrivial-auto-var-init=pattern", "-DYTGB_GENERAL_LOOP"],
}


@pytest.fixture(scope="module")
def runs(tmp_path_factory):
    d = tmp_path_factory.mktemp("address_checks")
    cuda_inc = os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include"
    probe = d / "probe.cpp"
    probe.write_text("int main() { return 0; }\n")
    sanitizers = subprocess.run(["g++", *SANITIZE, str(probe), "-o", str(d / "probe")], capture_output=True).returncode == 0

    def one(name):
        if name.startswith("sanitized") and not sanitizers:
            return name, None
        exe = d / name
        subprocess.run(["g++", "-std=c++17", "-ffp-contract=off", *BUILDS[name], f"-I{ROOT / 'include'}",
                        f"-I{ROOT / 'yt_gb300' / 'csrc'}", f"-I{cuda_inc}", str(SRC), "-o", str(exe)], check=True)
        return name, subprocess.run([str(exe)], capture_output=True, text=True, timeout=600,
                                    env={**os.environ, "ASAN_OPTIONS": "detect_leaks=0"})

    with ThreadPoolExecutor(len(BUILDS)) as ex:
        return dict(ex.map(one, BUILDS))


@pytest.mark.parametrize("name", [b for b in BUILDS if b.startswith("sanitized")])
def test_reads_inside_the_arrays(runs, name):
    if runs[name] is None:
        pytest.skip("no sanitizer libraries")
    assert runs[name].returncode == 0, runs[name].stderr[-3000:]


def test_every_build_forms_the_same_images(runs):
    done = {n: r for n, r in runs.items() if r is not None}
    for n, r in done.items():
        assert r.returncode == 0, (n, r.stderr[-3000:])
        assert r.stdout == done["zero"].stdout, n
