"""Alignment batches whose launch groups find no room side by side run with the scratch of one group, as they
did before the groups ran together (host check, tests/native/sw_scratch_check.cpp; no test drives a GPU out
of memory)."""
from __future__ import annotations

import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_scratch_is_shared_when_there_is_no_room_for_all(tmp_path):
    cxx = shutil.which("g++")
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    if cxx is None or not (cuda / "cuda_runtime.h").exists():
        pytest.skip("g++ or the CUDA headers not available")
    exe = tmp_path / "sw_scratch_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", f"-I{cuda}", f"-I{ROOT / 'rovaca_b200' / 'csrc'}",
                    str(ROOT / "tests" / "native" / "sw_scratch_check.cpp"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "ok\n"
