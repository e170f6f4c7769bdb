"""The 16x16 backward's variant for steps of few tiles is for launches whose
blocks are all resident at once, so its limit follows the device's
multiprocessors (152 on a whole GB300, fewer on a part of one).  The library's
own rule, compiled for the host."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "skyfall-viewer_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "kernels.cuh"
int main() {
  for (int sms : {1, 38, 76, 132, 152})
    std::printf("%d %d ", (int)sky::few_tiles(5u * sms, sms), (int)sky::few_tiles(5u * sms + 1u, sms));
}
"""


def test_limit_follows_the_multiprocessors(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "few.cpp", tmp_path / "few"
    src.write_text(PROGRAM)
    include = Path(nvcc).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", f"-I{include}", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split() == ["1", "0"] * 5


def test_the_launch_asks_the_device():
    text = re.sub(r"//[^\n]*", "", (CSRC / "kernels.cu").read_text())
    assert re.search(r"few_tiles\(max_tiles, sm_count\(\)\)", text)
    assert "152" not in re.findall(r"\b\d+\b", text)  # no multiprocessor count written out
