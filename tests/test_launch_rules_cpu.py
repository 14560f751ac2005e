"""Host rules that choose between kernels or size their grids, checked on the
CPU: tests/cpp/launch_rules_check.cu includes the launch headers and calls the
rules themselves. nvcc compiles it for sm_100a, but nothing runs on a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_launch_rules(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "launch_rules_check")
    cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++20", "-O1", "--expt-relaxed-constexpr",
           "-I", os.path.join(ROOT, "zldsp_fft_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", "cpp", "launch_rules_check.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr
    assert all(f"{rule}: ok" in r.stdout for rule in ("pairs", "launches", "runs", "single")), r.stdout
