"""The builder of the two native libraries, without a compiler run."""

import tomllib
from pathlib import Path

import pytest

from templar_b200.ops import build as B

ROOT = Path(__file__).resolve().parent.parent


def test_everything_the_builder_reads_is_package_data():
    """An installed package holds the files that package-data names and nothing else beside the Python modules."""
    globs = tomllib.loads((ROOT / "pyproject.toml").read_text())["tool"]["setuptools"]["package-data"]["templar_b200.ops"]
    packed = {p for g in globs for p in B.HERE.glob(g)}
    read = [*B.sources(), *B.headers(), *B.host_sources()]
    assert B.sources() and B.headers() and B.host_sources()
    assert not [p.name for p in read if p not in packed]


def test_missing_host_sources_are_named(monkeypatch, tmp_path):
    monkeypatch.setattr(B, "HOST_SRC", tmp_path)
    with pytest.raises(RuntimeError, match="no sources of the autograd nodes"):
        B._build_host(lambda cmd: pytest.fail("the compiler was called without sources"))
