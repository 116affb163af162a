"""The library's host-side helpers over a fake CUDA runtime (tests/fake_cuda.hpp):
what they leave behind when any one of their calls fails."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("check", ["stream_fork_check", "ray_order_check", "call_buffer_check"])
def test_helper_survives_every_failing_call(tmp_path, check):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / check
    subprocess.run([gxx, "-O2", "-std=c++20", "-Wall", "-Wextra", "-Werror", "-Wno-unused-parameter", "-isystem",
                    "/usr/local/cuda/include", "-o", str(exe), str(ROOT / "tests" / f"{check}.cpp")], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
    assert int(res.stdout) > 0
