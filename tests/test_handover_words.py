"""The decode stages' hand-over: a poll that gives up leaves no copy in flight (staged_decode.cuh)."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_a_poll_that_gives_up_waits_for_the_blocks_copies():
    """The tile of a warp that polls is on its way into the block's shared memory: before the warp leaves, the tile has to be there."""
    src = (ROOT / "nvmai_b200" / "csrc" / "staged_decode.cuh").read_text()
    polls = [m.start() for m in re.finditer(r"if \(!poll_row_part<", src)]
    assert polls
    for at in polls:
        leaves = src.index("return false;", at)
        assert "mbar_wait(bar, 0, status);" in src[at:leaves]
