"""Which register cap, shared-memory split and hand-over the decode stages take follows from the room on an SM (stage_room.h)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_the_stages_room_by_shared_memory_and_registers(tmp_path):
    exe = tmp_path / "stage_room_check"
    subprocess.run(["g++", "-std=c++17", "-O2", str(ROOT / "tests" / "cpp" / "stage_room_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr
