"""A launch's attributes are its own: the shared-memory split that one handle's decode stages ask for does not stay with the
kernel for the next handle (launch.h)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA = Path("/usr/local/cuda")


@pytest.mark.skipif(shutil.which("g++") is None or not (CUDA / "include" / "cuda_runtime.h").exists(),
                    reason="needs g++ and the CUDA headers")
def test_the_shared_memory_split_is_the_launchs_own(tmp_path):
    exe = tmp_path / "launch_check"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CUDA / 'include'}", str(ROOT / "tests" / "cpp" / "launch_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
