"""A step's scan raises the capacity bit at its last item.  Its blocks run in any
order, and a pass that grows its buffers goes on with what they wrote, so no
block may take that bit of its own grid for a reason to write nothing.  Errors
from before the scan (a sort that gave up, more views than launched for) do
stop it.  The library's own predicate, compiled for the host, over every order
of a grid's blocks."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "skyfall-viewer_gb300" / "csrc"

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include "sort.cuh"
using namespace sky;
int main() {
  int order[5] = {0, 1, 2, 3, 4}, missing = 0;
  do {
    uint32_t error = 0;
    for (int block : order) {
      if (scan_without_input(error)) ++missing;
      if (block == 4) error |= SKY_DEVERR_CAPACITY;  // the block of the last item
    }
  } while (std::next_permutation(order, order + 5));
  const uint32_t before[] = {SKY_DEVERR_SORT_TIMEOUT, SKY_DEVERR_LISTS, SKY_DEVERR_VIEWS};
  int stopped = 0, bits = SKY_DEVERR_CAPACITY;
  for (uint32_t e : before) {
    stopped += scan_without_input(e) && scan_without_input(e | SKY_DEVERR_CAPACITY);
    stopped -= (bits & e) != 0;  // the bits are distinct
    bits |= e;
  }
  std::printf("%d %d\n", missing, stopped);
}
"""


def test_blocks_write_whatever_their_order(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "scan.cpp", tmp_path / "scan"
    src.write_text(PROGRAM)
    include = Path(nvcc).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", f"-I{include}", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split() == ["0", "3"]


def test_scan_kernels_ask_only_that():
    text = re.sub(r"//[^\n]*", "", (CSRC / "kernels.cu").read_text())
    skip = re.search(r"bool scan_skipped\([^)]*\) \{(.*?)\n?\}", text, re.S).group(1)
    assert "scan_without_input(" in skip and "capacity_failed" not in skip
    for kernel in ("k_scan_reduce", "k_scan_blocks", "k_scan_final"):
        body = re.search(r"\b" + kernel + r"\(DevBuffers b.*?\n\}\n", text, re.S).group(0)
        assert "scan_skipped(b)" in body and "capacity_failed" not in body
    # the bit is raised by the scan and, once it has run, by the group bounds alone
    raisers = re.findall(r"\b(k_\w+)\([^;{]*\) \{(?:(?!__global__).)*?SKY_DEVERR_CAPACITY", text, re.S)
    assert raisers == ["k_scan_final", "k_group_bounds"]
