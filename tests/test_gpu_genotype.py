"""The genotype kernel (a warp per genotype, its lanes forming the terms of 32 reads at a time) against the
restatement of the reference's marginalisation and genotype likelihoods (oracle/genotype.py), bit for bit on
the device's own normalised matrix: read counts at and around whole warps, one allele to more genotypes than
a block has warps, alleles without a haplotype and haplotypes without an allele."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import genotype as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_reads", [1, 2, 31, 32, 33, 63, 64, 65, 130])
def test_genotype_likelihoods_equal_the_restatement(engine, n_reads):
    rng = np.random.default_rng(n_reads)
    acgt = np.frombuffer(b"ACGT", np.uint8)
    ref = acgt[rng.integers(0, 4, 260)]
    haps = []
    for h in range(9):
        x = ref.copy()
        x[20 + 25 * h] = acgt[(np.searchsorted(acgt, x[20 + 25 * h]) + 1) % 4]
        haps.append(x.tobytes())
    reads, quals = [], []
    for r in range(n_reads):
        s = int(rng.integers(0, 140))
        reads.append(haps[int(rng.integers(0, 9))][s:s + 120])
        quals.append(rng.integers(20, 41, 120).astype(np.uint8).tobytes())
    if n_reads > 2:  # a read that is dropped
        reads[n_reads // 2] = acgt[rng.integers(0, 4, 120)].tobytes()
    of = lambda m: (np.arange(9) % m).astype(np.int8)
    partial = of(3)
    partial[4] = -1
    events = [(1, of(1)), (2, of(2)), (5, of(5)), (9, of(9)), (4, partial), (3, np.full(9, -1, np.int8))]
    t = engine.submit_region(haps, reads, quals, np.full(n_reads, 60, np.uint8), 18, 0, events=events, want_allele_lk=True)
    mat, keep = t.wait()
    kept = int(keep.sum())
    assert kept == n_reads - (n_reads > 2)
    for (n_alleles, of_hap), (gl, best, alk) in zip(events, t.genotypes()):
        want = G.marginalize(mat, kept, list(of_hap), n_alleles)
        assert np.array_equal(alk[:, :kept], want) and np.isnan(alk[:, kept:]).all()
        likelihoods = G.genotype_likelihoods(want)
        assert np.array_equal(gl, likelihoods)
        assert best == G.best_genotype(likelihoods)
