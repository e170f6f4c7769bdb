"""Chained kernels pass their pointer parameters through the wait for their
predecessor.  Pointers inside struct parameters are not: their loads stay
behind the wait's memory clobber as long as no member is __restrict__."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "skyfall-viewer_gb300" / "csrc"


def test_no_restrict_members():
    found = 0
    for f in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        for body in re.findall(r"\bstruct\b[^;{()]*\{(.*?)\n\};", text, re.S):
            found += 1
            assert "__restrict__" not in body, f.name
    assert found >= 10  # DevBuffers, SortSegment, ViewerParams and the others
