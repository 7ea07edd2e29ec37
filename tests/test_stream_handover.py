"""The streaming kernel's hand-over between the two warps of a tile (stream_gemm.cuh, KS = 2): a slot may be written again,
two units later, only after it has been read, whatever the number of stages and the length of a unit."""
import re
from pathlib import Path

import pytest

SRC = (Path(__file__).resolve().parent.parent / "nvmai_b200" / "csrc" / "stream_gemm.cuh").read_text()


def _ordered(stages: int, chunks: int, scales_after_read: bool) -> bool:
    """Is the first half's write of unit 2 behind the second half's read of unit 0?  What must have happened before an event,
    followed back from the write: a warp's own order, a chunk's fill behind the release of the stage's last use by both
    warps, a unit's scales behind the release of the scales of the unit before the last one."""
    def before(event):
        kind, warp, u, i = event
        if kind == "use":                                    # chunk i of unit u
            yield ("use", warp, u, i - 1) if i else ("scales", warp, u, 0)
            n = u * chunks + i - stages                      # the chunk that had this stage
            if n >= 0:
                yield from (("use", w, n // chunks, n % chunks) for w in (0, 1))
        elif kind == "scales":                               # the unit's scales are there
            if u >= 1:
                yield ("over", warp, u - 1, 0)
            if u >= 2:
                yield from ((("over" if scales_after_read else "use"), w, u - 2, 0 if scales_after_read else chunks - 1) for w in (0, 1))
        else:                                                # hand-over of unit u written (warp 0) or read (warp 1)
            yield ("use", warp, u, chunks - 1)
            if warp == 1:
                yield ("over", 0, u, 0)
    seen, todo = set(), [("over", 0, 2, 0)]
    while todo:
        e = todo.pop()
        if e not in seen:
            seen.add(e)
            todo.extend(before(e))
    return ("over", 1, 0, 0) in seen


def test_the_model_finds_the_unordered_case():
    assert _ordered(6, 4, False) and not _ordered(6, 3, False) and not _ordered(4, 2, False)


@pytest.mark.parametrize("stages", range(1, 17))
@pytest.mark.parametrize("chunks", [1, 2, 3, 4, 8, 16])
def test_a_slot_is_written_again_only_after_it_was_read(stages, chunks):
    read = re.search(r"mbar_wait\(&bars->h_full\[turn & 1u\]", SRC).start()
    release = SRC.index("scales_done();", read) if "scales_done();" in SRC else SRC.index("mbar_arrive(&bars->m_empty")
    assert _ordered(stages, chunks, scales_after_read=release > read)
