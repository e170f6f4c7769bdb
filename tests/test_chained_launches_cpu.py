"""Kernels launched with programmatic stream serialization wait for their
predecessor before anything else: a kernel that did not would read unfinished
results, and one that ended early would let its successor do so."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "skyfall-viewer_gb300" / "csrc"
TEXT = {f.name: re.sub(r"//[^\n]*", "", f.read_text()) for f in CSRC.glob("*.cu")}
CHAINED = sorted({(f, k) for f, t in TEXT.items()
                  for k in re.findall(r"\bchain(?:_if)?\((?:\w+,\s*)?(k_\w+)", t)})


def test_kernels_are_found():
    assert {"k_onesweep", "k_forward", "k_backward_exact2", "k_geom_adam"} <= {k for _, k in CHAINED}
    calls = sum(len(re.findall(r"\bchain(?:_if)?\(", t)) for t in TEXT.values())
    named = sum(len(re.findall(r"\bchain(?:_if)?\((?:\w+,\s*)?k_\w+", t)) for t in TEXT.values())
    assert calls == named


@pytest.mark.parametrize("file,kernel", CHAINED)
def test_waits_first(file, kernel):
    found = re.findall(r"__global__[^;{]*?\b" + kernel + r"\(([^;{]*?)\)\s*\{\s*([^;]*;)", TEXT[file])
    assert len(found) == 1
    params, first = found[0]
    # every pointer parameter goes through the wait: a load through a const
    # __restrict__ one may otherwise be moved before it
    pointers = [q.split()[-1].lstrip("*") for q in params.split(",") if "*" in q]
    assert first == "chain_wait(" + ", ".join(pointers) + ");"
