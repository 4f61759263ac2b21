"""A test that compares with a checker is skipped only where the checker cannot be: the reference's library without the
reference's sources.  Whatever could have been built, or shipped with the tree, and is missing fails the test."""
import unittest

import pytest

from oracle import oracle as O


@pytest.fixture
def nothing_built(monkeypatch, tmp_path):
    monkeypatch.setattr(O, "ORACLE_SO", str(tmp_path / "liboracle.so"))
    monkeypatch.setattr(O, "REF_SO", str(tmp_path / "libref.so"))
    monkeypatch.setattr(O, "_libs", {})
    monkeypatch.setattr(O, "build", lambda reference=True: None)


@pytest.mark.parametrize("lib,sources,skipped", [("ref", False, True), ("ref", True, False), ("oracle", False, False),
                                                 ("oracle", True, False)])
def test_missing_library(nothing_built, monkeypatch, lib, sources, skipped):
    monkeypatch.setattr(O, "has_reference", lambda: sources)
    error = None
    try:
        O._load(lib)
    except FileNotFoundError as e:
        error = e
    assert error is not None and isinstance(error, unittest.SkipTest) == skipped
    assert not O.available(lib)
