"""Launch shapes follow the device's SM count, not that of one part (a partition of it has fewer)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "helio_b200" / "csrc"


def test_no_launch_shape_is_sized_by_a_constant_sm_count():
    for p in sorted(CSRC.iterdir()):
        if p.suffix in (".cu", ".cuh", ".h"):
            code = re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", p.read_text(), flags=re.S))
            assert not re.search(r"\b148(u|ull|l)?\b", code), p.name
