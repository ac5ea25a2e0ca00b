"""Where the reference's kernels are neither built nor buildable, what needs them
says so in a way that pytest counts as skipped."""
import unittest

import pytest

import oracle
from opensayal_gb300.fluid import default_config


def test_missing_reference_is_a_skip(oracle_built, monkeypatch, tmp_path):
    monkeypatch.setattr(oracle, "REF_CUBIN", tmp_path / "none.cubin")
    monkeypatch.setattr(oracle, "_harness", None)
    assert not oracle.reference_available()
    with pytest.raises(unittest.SkipTest, match="none.cubin"):
        oracle.RefFluid(default_config(16, 16))
