"""Host rules of the ragged tuning, on the CPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_warp_limit_does_not_depend_on_the_cta_size(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "test_limited_ctas")
    r = subprocess.run([nvcc, "-std=c++17", "-I", os.path.join(ROOT, "cusbf_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "test_limited_ctas.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    assert subprocess.run([exe]).returncode == 0
