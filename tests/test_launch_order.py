"""Rule 1 of launch.h, read from the sources: a kernel waits for the one in front right before it lets the one behind start."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "nvmai_b200" / "csrc"


def test_dependents_start_only_behind_an_unconditional_wait():
    seen = 0
    for path in sorted(CSRC.glob("*.cu*")):
        lines = [re.sub(r"//.*", "", line).strip() for line in path.read_text().splitlines()]
        for i, line in enumerate(lines):
            if "pdl_launch_dependents();" not in line or "__device__" in line:
                continue
            seen += 1
            before = line.split("pdl_launch_dependents();")[0].strip() or next(p for p in reversed(lines[:i]) if p)
            assert re.search(r"(^|[{;]\s*)pdl_wait\(\);$", before), f"{path.name}:{i + 1}"
    assert seen >= 15
