"""The serving loop holds its batches to a share of the memory budget by an estimate of what each request takes
(host check, tests/native/request_bytes_check.cpp): with work items down to one haplotype each, 24 bytes a
rerun slot and the codes of two alignments in a warp it is not below what a region needs, nor twice it."""
from __future__ import annotations

import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_the_estimate_covers_what_a_region_takes(tmp_path):
    cxx = shutil.which("g++")
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    if cxx is None or not (cuda / "cuda_runtime.h").exists():
        pytest.skip("g++ or the CUDA headers not available")
    exe = tmp_path / "request_bytes_check"
    csrc = ROOT / "rovaca_b200" / "csrc"
    subprocess.run([cxx, "-std=c++17", "-O2", "-w", "-pthread", f"-I{cuda}", f"-I{csrc}",
                    str(ROOT / "tests" / "native" / "request_bytes_check.cpp"), str(csrc / "phmm_plan.cpp"),
                    str(csrc / "phmm_tables.cpp"), "-o", str(exe)], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True)
    assert p.returncode == 0 and p.stdout == "ok\n", p.stdout
