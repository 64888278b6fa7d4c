"""CPU: the build entry point works beside a reference tree that is missing or empty."""
import importlib
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("there", [False, True])
def test_build_without_reference_sources(lib, tmp_path, monkeypatch, there):
    if there:
        (tmp_path / "reference").mkdir()
    monkeypatch.setenv("SIP_REFERENCE_ROOT", str(tmp_path / "reference"))
    sys.path.insert(0, ROOT)
    entry = importlib.reload(importlib.import_module("__graft_entry__"))
    entry.build()
