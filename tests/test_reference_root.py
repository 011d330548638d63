"""Without the reference's sources (no REFERENCE_ROOT) what needs them is skipped, not an error: the source
root is then a path that holds none of them, and the build functions keep the libraries already built."""
from __future__ import annotations

from pathlib import Path

import pytest


def test_an_unset_reference_root_is_a_path_without_sources(monkeypatch):
    from oracle import oracle

    monkeypatch.delenv("REFERENCE_ROOT", raising=False)
    assert not Path(oracle.reference_root(), "src/haplotypecaller/pairhmm").is_dir()
    for build, lib in ((oracle.build_ref, oracle.REF_LIB), (oracle.build_ref_sw, oracle.SW_REF_LIB),
                       (oracle.build_ref_genotype, oracle.GENOTYPE_REF_LIB)):
        assert build() == (lib if lib.exists() else None)


def test_the_binding_s_driver_is_skipped_when_it_cannot_be_built(monkeypatch, tmp_path):
    import test_integration

    monkeypatch.delenv("REFERENCE_ROOT", raising=False)
    monkeypatch.setattr(test_integration, "BIN", tmp_path / "missing")
    with pytest.raises(pytest.skip.Exception):
        test_integration._binary()
