"""Batches replayed from a captured CUDA graph give the bits of direct launches: small ones with every
batch replayed (use_cuda_graph=2), the default's large ones before and after a small batch laid out
compactly in the same arena, after a change of tile shapes, and region requests with genotyping and
realignment.  A graph holds every class (66 and the preparation and post-processing kernels), a direct
launch only the classes with work, so kernel_launches tells which of the two ran."""
from __future__ import annotations

import random

import numpy as np
import pytest

from rovaca_b200 import synth
from test_gpu_parity import _all_length_batch, _table
from test_gpu_realign import _realign_inputs

pytestmark = pytest.mark.gpu
CLASSES = 66


def _same(a, b):
    assert np.array_equal(a[0], b[0], equal_nan=True) and np.array_equal(a[1], b[1])


def test_small_batches_through_the_graph_equal_direct_launches(engine_direct, ref_regions):
    from rovaca_b200 import Engine

    with Engine(device=0, autotune=False, use_cuda_graph=2) as eng:
        for group in ("debug", "edge", "config1", "debug"):
            pb, _ = ref_regions[group]
            for flags in (True, False):
                a = eng.compute(pb, want_flags=flags)
                b = engine_direct.compute(pb, want_flags=flags)
                assert a[2]["kernel_launches"] > CLASSES > b[2]["kernel_launches"]
                assert np.array_equal(a[0], b[0], equal_nan=True)
                assert not flags or np.array_equal(a[1], b[1])
        with eng.resident(pb, want_flags=True) as res:  # replayed several times
            assert res.run(3)["kernel_launches"] > 3 * CLASSES
            _same(res.results(), engine_direct.compute(pb, want_flags=True))


def test_a_graph_is_captured_again_for_a_new_tile_table(engine_direct):
    """The FP64 classes' dependencies follow the table: with the graph of the old one, pairs of shapes that
    moved would be recomputed before the FP32 classes that report them have run."""
    from rovaca_b200 import Engine

    pb = _all_length_batch(7)
    want = engine_direct.compute(pb, want_flags=True)
    with Engine(device=0, autotune=False, use_cuda_graph=2) as eng:
        for table in (None, _table(lambda m, b: (4, 1) if b > 4 else None), _table(lambda m, b: (8, 1) if b > 8 else None)):
            if table is not None:
                eng.set_tiles(table)
            for _ in range(2):
                got = eng.compute(pb, want_flags=True)
                assert got[2]["kernel_launches"] > CLASSES
                _same(got, want)


def test_large_batches_keep_their_graph_around_compact_ones(engine_direct):
    """... and report its launches, not those of the direct launch before them."""
    from rovaca_b200 import Engine

    big, small = synth.config1(90, seed=21), synth.config1(1, seed=22)
    want_big = engine_direct.compute(big, want_flags=True)
    want_small = engine_direct.compute(small, want_flags=True)
    assert want_big[2]["cells"] >= 2e10
    with Engine(device=0, autotune=False, chunk_cells=2**64 - 1) as eng:
        for step in ("big", "small", "big", "tiles", "big", "small", "small", "big"):
            if step == "tiles":
                eng.set_tiles(_table(lambda m, b: (5, 1) if b > 5 else None))
                continue
            got = eng.compute(big if step == "big" else small, want_flags=True)
            assert (got[2]["kernel_launches"] > CLASSES) == (step == "big")
            _same(got, want_big if step == "big" else want_small)


def test_region_requests_through_the_graph_equal_direct_launches(engine):
    from rovaca_b200 import Engine

    regions = synth.genotyping_regions(12, seed=41)
    rng = random.Random(9)
    inputs = [_realign_inputs(r, rng) for r in regions]

    def run(eng):
        tickets = [eng.submit_region(r["haplotypes"], r["reads"], r["quals"], r["mapq"], 18, k % 4,
                                     events=r["events"], want_allele_lk=True, realign=z)
                   for k, (r, z) in enumerate(zip(regions, inputs))]
        out = []
        for t in tickets:
            mat, keep = t.wait()
            best, sw = t.realignment()
            out += [mat, keep, best, sw.fields, sw.cigars]
            for gl, call, alk in t.genotypes():
                out += [gl, np.array(call), alk]
        return out

    want = run(engine)
    with Engine(device=0, autotune=False, use_cuda_graph=2) as eng:
        for _ in range(2):
            got = run(eng)
            assert len(got) == len(want)
            for a, b in zip(got, want):
                assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")
        stats = eng.server_stats()
        assert stats["graph_captures"] >= 1 and stats["batches"] >= 2
