"""An alignment call stages its sequences and plans its launches side by side, on one thread or two by the
batch's bytes and alignments: every form gives what the resident batch (uploaded piece by piece, planned
before) gives, and the oracle's alignments on a sample."""
from __future__ import annotations

import numpy as np
import pytest

from rovaca_b200 import sw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, hap, read, what", [
    (300, 400, 150, "under 1 MiB: one thread"),
    (900, 1400, 900, "many bytes an alignment: planned on the helper"),
    (20000, 40, 30, "few bytes an alignment: staged on the helper"),
    (9000, 1900, 60, "over 16 MB: copied by several threads"),
])
def test_every_staging_form_gives_the_resident_batch_s_results(engine, sw_oracle, n, hap, read, what):
    rng = np.random.default_rng(n)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    haps = acgt[rng.integers(0, 4, (n, hap))]
    at = rng.integers(0, hap - read + 1, n)
    reads = np.take_along_axis(haps, at[:, None] + np.arange(read), axis=1)
    wrong = rng.random(reads.shape) < 0.01
    reads[wrong] = acgt[rng.integers(0, 4, int(wrong.sum()))]
    batch = sw.SwBatch.from_pairs([(h.tobytes(), r.tobytes()) for h, r in zip(haps, reads)])
    assert {0: n * (hap + read) < 1 << 20, 1: n * (hap + read) >= 128 * n, 2: n * (hap + read) < 128 * n,
            3: n * hap >= 16 << 20}[[300, 900, 20000, 9000].index(n)]
    with engine.sw_resident(batch) as r:
        r.run(1)
        want = r.results()
    for _ in range(2):
        got = engine.sw_align(batch)
        assert np.array_equal(got.fields, want.fields) and np.array_equal(got.cigars, want.cigars)
    for q in range(0, n, max(1, n // 40)):
        assert got.tuple(q) == sw_oracle.align(*batch.pair(q))
