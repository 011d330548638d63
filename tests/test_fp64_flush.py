"""The FP64 pass sweeps a pair without flushes first and again, flushing every result below 2^-1022 as the
reference does, when its sum is below 2^-700 (rovaca_b200/csrc/phmm_device64.cuh).  On the CPU emulator,
whose FP64 lanes keep such values as the GPU does, pairs around and far below that line equal the
reference's FP64 kernel (the oracle's) to 1e-12; the emulator built without the second sweep does not,
so it can tell."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess

import numpy as np
import pytest

from rovaca_b200.pairhmm import PackedBatch, Region
from test_warp_emulator import CSRC, EXACT, LOG10_C_F64, NATIVE, _run, _write, emulator  # noqa: F401

LINE = -700 * np.log10(2.0) - LOG10_C_F64  # the likelihood of a sum of 2^-700


def _batch(kind: str) -> PackedBatch:
    """Reads of 250 and 300 bases (one and two stripes), from a quarter matching their haplotype to not at
    all, at qualities that spread the likelihoods from 1e-300 to below all doubles."""
    rng = np.random.default_rng(5)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    haps = [acgt[rng.integers(0, 4, n)].tobytes() for n in (44, 60, 75)]
    reads, q, i, d, c = [], [], [], [], []
    for r in range(16):
        n = 250 if r % 2 else 300
        x = acgt[rng.integers(0, 4, n)].copy()
        own = np.frombuffer(haps[r % 3], np.uint8)[:10 * (r % 4)]
        x[:len(own)] = own
        if kind == "N":
            x[n // 2] = ord("N")
        reads.append(x.tobytes())
        q.append(rng.integers(20, 41, n).astype(np.uint8).tobytes())
        vary = kind == "per_base"
        i.append((rng.integers(30, 46, n) if vary else np.full(n, 45)).astype(np.uint8).tobytes())
        d.append((rng.integers(30, 46, n) if vary else np.full(n, 45)).astype(np.uint8).tobytes())
        c.append((np.full(n, 10 + r) + (rng.integers(0, 2, n) if vary else 0)).astype(np.uint8).tobytes())
    return PackedBatch.from_regions([Region(haps, reads, q, i, d, c)])


def _reference(oracle, pb: PackedBatch, kernel: int) -> np.ndarray:
    cut = lambda a, off, k: bytes(a[int(off[k]):int(off[k + 1])])
    raw = np.array([[oracle.raw_f64(cut(pb.hap_bases, pb.hap_off, h), *(cut(a, pb.read_off, r) for a in (
        pb.read_bases, pb.read_qual, pb.read_ins, pb.read_del, pb.read_gcp)), kernel=kernel)
        for r in range(int(pb.n_reads[0]))] for h in range(int(pb.n_haps[0]))])
    with np.errstate(divide="ignore"):
        return np.log10(raw).reshape(-1) - LOG10_C_F64


def _differs(a: np.ndarray, b: np.ndarray) -> np.ndarray:
    with np.errstate(invalid="ignore"):
        return ~((a == b) | (np.abs(a - b) <= EXACT))


@pytest.mark.parametrize("kind", ["flat", "per_base", "N"])
def test_tiny_likelihoods_on_the_emulator_equal_the_reference(emulator, oracle, tmp_path, kind):  # noqa: F811
    pb = _batch(kind)
    want = _reference(oracle, pb, 1 if kind == "N" else 0)
    got, _, status = _run(emulator, pb, tmp_path, mode="eq64" if kind == "flat" else "row64")
    assert status == 0
    assert not _differs(got, want).any()
    assert (want > LINE + 20).any() and (np.abs(want - LINE) < 40).any() and (want < LINE - 60).any()
    assert np.isinf(want).any()


def test_the_emulator_can_tell_the_second_sweep_left_out(oracle, tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    binary = tmp_path / "warp_emu_unflushed"
    subprocess.run([gxx, "-std=c++20", "-O2", "-mfma", "-ffp-contract=off", "-pthread", "-w",
                    "-DPHMM_F64_UNFLUSHED_MIN=0.0", str(NATIVE / "warp_emu.cpp"), str(CSRC / "phmm_plan.cpp"),
                    str(CSRC / "phmm_tables.cpp"), "-o", str(binary)], check=True)
    pb = _batch("flat")
    want = _reference(oracle, pb, 0)
    got, _, status = _run(binary, pb, tmp_path, mode="eq64")
    wrong = _differs(got, want)
    assert status == 0 and wrong.any()
    assert not wrong[want >= LINE].any()  # above the line the unflushed sweep alone is enough


def _collectives(binary, pb: PackedBatch, tmp_path) -> int:
    """What the FP64 recompute of every pair of the batch cost: the collectives of its warps' steps."""
    _write(pb, tmp_path / "batch.bin")
    p = subprocess.run([str(binary), str(tmp_path / "batch.bin"), str(tmp_path / "out.bin"), "eq64", "default"],
                       check=True, timeout=900, capture_output=True, text=True)
    return int(p.stdout.split()[1])


def _fit(order: str, reads: int = 1) -> PackedBatch:
    """Haplotypes that hold the reads (g) and foreign ones (f), whose pairs are below the line."""
    rng = np.random.default_rng(17)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    own = acgt[rng.integers(0, 4, 160)]
    foreign = np.frombuffer(b"ACGT", np.uint8)[3 - np.searchsorted(acgt, own)]  # no base of the reads' own place
    haps = [(own if k == "g" else foreign).tobytes() for k in order]
    gap = [bytes([80] * 160)] * reads
    return PackedBatch.from_regions([Region(haps, [own.tobytes()] * reads, [bytes([60] * 160)] * reads, gap, gap, gap)])


def test_only_the_haplotypes_below_the_line_are_swept_again(emulator, oracle, tmp_path):  # noqa: F811
    """Foreign haplotypes at both ends of a run cost what the same ones next to each other cost, but for one
    more fill of the wavefront (a fifth of a haplotype here): those between them are not swept again."""
    want = _reference(oracle, _fit("fggggf"), 0)
    assert (want[[0, 5]] < LINE).all() and (want[1:5] > LINE).all()
    apart, together, none = (_collectives(emulator, _fit(o), tmp_path) for o in ("fggggf", "ffgggg", "gggggg"))
    assert none < together < apart < 1.1 * together


def test_runs_of_foreign_reads_are_not_all_swept_twice(emulator, tmp_path):  # noqa: F811
    """Twelve runs whose pairs are all below the line: the first two are swept both ways."""
    foreign, good = (_collectives(emulator, _fit(o, reads=12), tmp_path) for o in ("ff", "gg"))
    assert 13 / 12 < foreign / good < 16 / 12


def test_no_factor_of_the_cell_update_exceeds_one(oracle):
    """What the flushes take away stays small because every value is multiplied by at most 1 from then on:
    over the whole tables, none negative."""
    lib = oracle.lib
    lib.oracle_ph2pr_f64.restype, lib.oracle_ph2pr_f64.argtypes = C.c_double, [C.c_int]
    lib.oracle_mm_f64.restype, lib.oracle_mm_f64.argtypes = C.c_double, [C.c_int, C.c_int]
    err = [lib.oracle_ph2pr_f64(q) for q in range(128)]
    vals = err + [1.0 - e for e in err] + [e / 3.0 for e in err]
    vals += [lib.oracle_mm_f64(i, j) for i in range(128) for j in range(128)]
    assert min(vals) >= 0.0 and max(vals) <= 1.0
