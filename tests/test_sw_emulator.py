"""The two-alignments-per-warp Smith-Waterman device code on the CPU (tests/native/sw16_emu.cpp) against
the oracle: score, end cell, offset and CIGAR of every alignment, and its stores inside its buffers."""
from __future__ import annotations

import ctypes as C
import random
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import SwOracle
from rovaca_b200 import sw

HERE = Path(__file__).resolve().parent
SRC = HERE / "native" / "sw16_emu.cpp"
CSRC = HERE.parent / "rovaca_b200" / "csrc"


@pytest.fixture(scope="module")
def emu():
    out = HERE / "native" / "_build" / "libsw16_emu.so"
    out.parent.mkdir(exist_ok=True)
    deps = [SRC, CSRC / "phmm_sw16.cuh", CSRC / "phmm_sw.h"]
    if not out.exists() or any(d.stat().st_mtime > out.stat().st_mtime for d in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-w", "-shared", "-fPIC", "-I/usr/local/cuda/include", str(SRC), "-o",
                        str(out), "-lpthread"], check=True)
    lib = C.CDLL(str(out))
    lib.emu_sw16_form.argtypes = [C.c_void_p, C.c_int, C.c_uint32, C.c_uint32, C.c_int]
    return lib


PLAIN, REBASED, ONE_PER_WARP = 0, 1, 2


def _run(lib, k, rebased, params, variant, pairs):
    haps, reads = b"".join(h for h, _ in pairs), b"".join(r for _, r in pairs)
    items = np.zeros(len(pairs), sw.SW_ITEM_DTYPE)
    items["hap_len"], items["read_len"] = [len(h) for h, _ in pairs], [len(r) for _, r in pairs]
    items["hap_offset"] = np.cumsum([0] + [len(h) for h, _ in pairs])[:-1]
    items["read_offset"] = np.cumsum([0] + [len(r) for _, r in pairs])[:-1]
    out, ops = np.zeros(len(pairs), sw.SW_RESULT_DTYPE), np.zeros(4096, np.uint32)
    prm = (C.c_int32 * 4)(*params)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    hb, rb = np.frombuffer(haps + b"\0", np.uint8), np.frombuffer(reads + b"\0", np.uint8)
    assert lib.emu_sw16(k, int(rebased), prm, variant, len(pairs), p(items), p(hb), p(rb), 2047, p(out), p(ops)) == 0
    return [(int(o["score"]), int(o["alignment_offset"]), int(o["max_i"]), int(o["max_j"]),
             [int(x) for x in ops[2047 * q:2047 * q + int(o["cigar_count"])]]) for q, o in enumerate(out)]


def _sequence(rng, n, alphabet):
    return bytes(rng.choice(alphabet) for _ in range(n))


def _read_of(rng, hap, n, rate):
    s = rng.randint(0, max(0, len(hap) - n))
    out = bytearray()
    for c in hap[s:s + n]:
        x = rng.random()
        if x < rate:
            out += rng.choice([b"", bytes([c]) + _sequence(rng, rng.randint(1, 9), b"ACGT"), _sequence(rng, 1, b"ACGT")])
        else:
            out.append(c)
    return bytes(out[:n])


@pytest.mark.parametrize("k", [1, 3, 5, 8, 10, 24])
@pytest.mark.parametrize("alphabet", [b"ACGT", b"AC", b"ACGTN", b"ACGTNacgt."], ids=["acgt", "repeats", "n", "other"])
def test_pairs_equal_the_oracle(emu, k, alphabet):
    """Widths whose scores fill one and several code words and table groups; reads from one base to the
    width's last column, haplotypes shorter and longer than the wavefront, unequal partners, a missing
    partner and empty sequences; few letters, for ties; letters outside A/C/G/T/N (the comparing step)."""
    rng = random.Random(100 * k + len(alphabet))
    oracle = SwOracle()
    lo = 1 if k == 1 else 32 * (k - 1 if k <= 8 else {10: 8, 24: 20}[k])
    shapes = [(1, lo), (31, 32 * k), (40, lo + 1), (260, 32 * k), (33, 32 * k - 1), (150, lo + 7)]
    for params, variant, rebased in ((sw.GENOTYPING, 0, False), ((3, -2, -5, -1), 2, False), ((1, 0, 0, -1), 1, False),
                                     (sw.ASSEMBLY, 1, True), (sw.GENOTYPING, 0, True), ((250, 0, -200, -40), 1, True)):
        pairs = []
        for rows, cols in shapes:
            h = _sequence(rng, rows, alphabet)
            r = _read_of(rng, h, cols, 0.06)
            pairs.append((h, (r + _sequence(rng, cols, alphabet))[:cols] if rng.random() < 0.7 else _sequence(rng, cols, alphabet)))
        groups = [pairs[0:2], pairs[2:4], pairs[4:6], pairs[3:4], [pairs[1], (b"", b"ACG"[:3])], [(b"ACGT", b""), pairs[5]],
                  [(b"", b""), (b"A", b"A")]]
        prm = (C.c_int32 * 4)(*params)
        for g in groups:
            form = {emu.emu_sw16_form(prm, int(variant == 1), len(h), len(r), k) for h, r in g}
            assert form <= ({PLAIN, REBASED} if rebased else {PLAIN})
            assert _run(emu, k, rebased, params, variant, g) == [oracle.align(h, r, params, variant) for h, r in g], (params, g)


def test_forms_of_parameters(emu):
    def form(params, nrow=300, ncol=250, k=8, i32=True):
        return emu.emu_sw16_form((C.c_int32 * 4)(*params), int(i32), nrow, ncol, k)

    assert form(sw.GENOTYPING) == form(sw.GENOTYPING, 2047, 768, 24) == form(sw.GENOTYPING, i32=False) == PLAIN
    assert form(sw.ASSEMBLY) == form(sw.ASSEMBLY, 2047, 768, 24) == REBASED      # 256 columns x 200
    assert form(sw.ASSEMBLY, i32=False) == REBASED
    assert form(sw.ASSEMBLY, 300, 768, 24, i32=False) == ONE_PER_WARP            # its int16 cutoff could bind
    for params, nrow, ncol, k in ((sw.GENOTYPING, 2048, 250, 8), (sw.GENOTYPING, 300, 769, 24),
                                  ((10, -15, 1, -5), 300, 250, 8), ((10, -15, -30, 0), 300, 250, 8),
                                  ((10, 1, -30, -5), 300, 250, 8), ((-1, -15, -30, -5), 300, 250, 8),
                                  ((600, -15, -300, -5), 300, 250, 8), ((200000, -15, -30, -5), 300, 250, 8),
                                  ((10, -15, -2**31, -5), 300, 250, 8), ((10, -15, -30, -2**31), 300, 250, 8)):
        assert form(params, nrow, ncol, k) == ONE_PER_WARP, params
