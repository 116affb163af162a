"""Host-side parts of the library checked without a GPU: what the helpers leave
behind when any one of their CUDA calls fails (tests/fake_cuda.hpp stands in for
the runtime), and the SDF cell tables at their size limit."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("check", ["stream_fork_check", "ray_order_check", "call_buffer_check", "sdf_budget_check"])
def test_host_check(tmp_path, check):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / check
    subprocess.run([gxx, "-O2", "-std=c++20", "-pthread", "-isystem", "/usr/local/cuda/include", "-o", str(exe),
                    str(ROOT / "tests" / f"{check}.cpp")], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
    assert int(res.stdout) > 0
