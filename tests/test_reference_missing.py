"""Tests that call the reference library, where it is not built."""
import os
import subprocess
import sys

import pytest

import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CALLER = """
import oracle as O

def test_reference(monkeypatch):
    monkeypatch.setattr(O, "_ref", None)
    monkeypatch.setattr(O, "REF_SO", "/nonexistent/libplmref.so")
    O.ref()

def test_other_error():
    raise RuntimeError("not the reference's absence")
"""


def test_missing_reference_raises(monkeypatch):
    monkeypatch.setattr(O, "_ref", None)
    monkeypatch.setattr(O, "REF_SO", "/nonexistent/libplmref.so")
    with pytest.raises(O.ReferenceNotBuilt):
        O.ref()


def test_missing_reference_skips_the_test(tmp_path):
    """One that calls it is skipped; any other error still fails."""
    f = tmp_path / "test_caller.py"
    f.write_text(CALLER)
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(
        [ROOT, os.path.join(ROOT, "tests")]))
    p = subprocess.run([sys.executable, "-m", "pytest", "-q", "-p", "conftest",
                        "-p", "no:cacheprovider", str(f)], cwd=tmp_path,
                       env=env, capture_output=True, text=True)
    assert "1 failed, 1 skipped" in p.stdout, p.stdout
