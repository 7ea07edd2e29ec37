"""The decode stages' hand-over: its tags are new for every call, past the last one too (handover_words.h), and a poll that gives up
leaves no copy in flight (staged_decode.cuh)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA = Path("/usr/local/cuda")


@pytest.mark.skipif(shutil.which("g++") is None or not (CUDA / "include" / "cuda_runtime.h").exists(),
                    reason="needs g++ and the CUDA headers")
def test_no_call_meets_its_tag_in_a_word_of_an_earlier_call(tmp_path):
    exe = tmp_path / "handover_words_check"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CUDA / 'include'}", str(ROOT / "tests" / "cpp" / "handover_words_check.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr


def test_a_poll_that_gives_up_waits_for_the_blocks_copies():
    """The tile of a warp that polls is on its way into the block's shared memory: before the warp leaves, the tile has to be there."""
    src = (ROOT / "nvmai_b200" / "csrc" / "staged_decode.cuh").read_text()
    polls = [m.start() for m in re.finditer(r"if \(!poll_row_part<", src)]
    assert polls
    for at in polls:
        leaves = src.index("return false;", at)
        assert "mbar_wait(bar, 0, status);" in src[at:leaves]
