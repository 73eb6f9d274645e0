"""Where the reference library is not built, a test that compares with it live is skipped, as the
tests are that ask for it beforehand: one missing file does not end a run that stops at its first
failure."""
import unittest

import pytest

import refdrive


def test_missing_reference_is_a_skip(monkeypatch, tmp_path):
    monkeypatch.setattr(refdrive, "REF_SO", tmp_path / "libmopref.so")
    monkeypatch.setattr(refdrive, "_libs", {})
    with pytest.raises(unittest.SkipTest, match="not built") as e:
        refdrive.lib()
    assert isinstance(e.value, FileNotFoundError)
