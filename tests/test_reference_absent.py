"""Comparisons with a reference build that is not there are skipped: its loader's error is a missing file and a skip."""
import unittest

import pytest

import oracle.oracle as O


@pytest.mark.parametrize("load", [lambda: O.RefCPU(), lambda: O.RefKZM(), lambda: O.RefCUDA()])
def test_a_missing_build_is_a_skip(load, monkeypatch, tmp_path):
    monkeypatch.setattr(O, "REF", str(tmp_path))
    with pytest.raises(FileNotFoundError) as e:
        load()
    assert isinstance(e.value, unittest.SkipTest)
