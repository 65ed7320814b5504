"""CPU check that the non-culling test's FP32 decisions (numba_tail in lyem_device.cuh) equal the numba engine's FP64
ones on inputs concentrated at every decision boundary; the device header is compiled for the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path_factory.mktemp("numba") / "numba_decisions")
    cmd = [nvcc, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off",
           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "lyceanem-python_gb300", "csrc"),
           "-o", exe, os.path.join(ROOT, "tests", "numba_decisions.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("seed", [1, 2])
def test_fp32_decisions_match_the_fp64_ones(checker, seed):
    r = subprocess.run([checker, "4000000", str(seed)], capture_output=True, text=True)
    cases, mismatches, hits = map(int, r.stdout.strip().splitlines()[-1].split())
    assert cases == 4000000 and mismatches == 0, r.stdout
    assert hits > cases // 20
