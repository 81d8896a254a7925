"""Chained launches that the runtime refuses on the host (no kernel runs)."""
import subprocess

import pytest

from perf_libs_sparse_b200 import build


@pytest.mark.gpu  # without a driver every runtime call reports the missing driver
def test_refused_launch_leaves_no_error(tmp_path):
    exe = tmp_path / "launch_check"
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-o", str(exe), f"{build.ROOT}/tests/launch_check.cu"],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
