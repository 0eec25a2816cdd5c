"""Comparisons with the reference's own library are skipped, not failed, where it is not built."""
import unittest

import pytest

from oracle import farfield as F


def test_missing_reference_library_skips(monkeypatch):
    monkeypatch.setattr(F, "ref_lib", lambda: None)
    for call in (lambda: F.ref_through_focus(((), ()), 1.0, 0.5, 1.0),
                 lambda: F.ref_propagate_pillars([0.0], [0.0], [1.0], 0.0, 0.0, 1.0, 0.5, 3, 1.0)):
        with pytest.raises(FileNotFoundError) as e:
            call()
        assert isinstance(e.value, unittest.SkipTest)
