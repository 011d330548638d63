"""Host check (no GPU) of the alignments behind the FP64 kernels' asynchronous copies:
tests/native/shared_layout_check.cpp holds them as compile-time checks of the kernels' own headers, and
the kernel declares the type they are checked on."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_the_fp64_table_and_its_ring_are_16_byte_aligned(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    subprocess.run([cxx, "-std=c++20", "-O1", "-mfma", "-w", "-fsyntax-only",
                    str(ROOT / "tests" / "native" / "shared_layout_check.cpp")], check=True)
    kernel = (ROOT / "rovaca_b200" / "csrc" / "phmm_kernels.cu").read_text()
    assert "__shared__ PriorTable64<K> tab;" in kernel and "__shared__ double" not in kernel
