"""A test that needs a program built from the reference's sources is skipped
where there is none, and does not end a run that stops at the first failure;
one that shares its fixture but not the program runs."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle

SCRIPT = """
import numpy as np
import pytest
import oracle

x = np.arange(64, dtype=np.float32)


@pytest.fixture
def shards():
    with oracle.UcrShards(x) as u:
        yield u


def test_search():
    oracle.ucr_dtw(x, x[:16], "2")


def test_shards(shards):
    shards.search(x[:16], 2)


def test_stream_of_the_shards(shards):
    assert shards.x is x


def test_ldtw():
    oracle.ref_ldtw(x[:16], x, 2)


def test_after():
    pass
"""


def test_missing_programs_skip(tmp_path, monkeypatch):
    (tmp_path / "test_needs_it.py").write_text(SCRIPT)
    (tmp_path / "conftest.py").write_text("import oracle\noracle.REF_DIR = '/nonexistent'\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-p", "no:cacheprovider",
                          str(tmp_path)], capture_output=True, text=True, cwd=tmp_path,
                         env={**os.environ, "PYTHONPATH": root}).stdout
    assert "2 passed, 3 skipped" in out
    monkeypatch.setattr(oracle, "REF_DIR", "/nonexistent")
    with pytest.raises(FileNotFoundError):
        oracle.ucr_ed(np.zeros(8), np.zeros(4))
