"""The disk cache of run-time compiled kernels, on the CPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_cache_file_follows_what_is_compiled(tmp_path):
    from cusbf_b200 import build

    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    build.write_jit_sources(str(tmp_path))
    exe = str(tmp_path / "test_jit_cache")
    r = subprocess.run([nvcc, "-std=c++17", "-I", str(tmp_path),
                        "-I", os.path.join(ROOT, "cusbf_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "test_jit_cache.cpp"), "-o", exe,
                        "-ldl"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
