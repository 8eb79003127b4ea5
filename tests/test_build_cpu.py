"""The builder of the two native libraries, with scripts in the compilers' places."""

import os
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


@pytest.fixture
def tree(monkeypatch, tmp_path):
    """A source tree of one kernel file and one host file, and compilers that write what they were called with to their output
    file (and fail when a file ``broken`` lies beside them)."""
    for d in ("csrc", "csrc_host", "_lib"):
        (tmp_path / d).mkdir()
    (tmp_path / "csrc" / "a.cu").write_text("")
    (tmp_path / "csrc" / "entries.h").write_text("")
    (tmp_path / "csrc_host" / "b.cpp").write_text("")
    for name in ("nvcc", "cxx"):
        f = tmp_path / name
        f.write_text(f'#!/bin/bash\n[ -e "{tmp_path}/{name}_broken" ] && exit 1\necho {name} >> "{tmp_path}/calls"\n'
                     'args=("$@")\nfor i in "${!args[@]}"; do [ "${args[$i]}" = -o ] && echo "$@" > "${args[$((i+1))]}"; done\nexit 0\n')
        f.chmod(0o755)
    monkeypatch.setattr(B, "CSRC", tmp_path / "csrc")
    monkeypatch.setattr(B, "HOST_SRC", tmp_path / "csrc_host")
    monkeypatch.setattr(B, "LIBDIR", tmp_path / "_lib")
    monkeypatch.setenv("NVCC", str(tmp_path / "nvcc"))
    monkeypatch.setenv("CXX", str(tmp_path / "cxx"))

    def calls():
        """Compiler calls since the last look."""
        log = tmp_path / "calls"
        got = sorted(log.read_text().split()) if log.exists() else []
        log.unlink(missing_ok=True)
        return got

    return tmp_path, calls


def test_builds_what_has_changed(tree):
    _, calls = tree
    B.build()
    assert calls() == ["cxx", "nvcc", "nvcc"]                  # the module, an object, the link
    B.build()
    assert calls() == []
    B.build(force=True)
    assert calls() == ["cxx", "nvcc", "nvcc"]


def test_another_pytorch_rebuilds_the_extension_module(tree, monkeypatch):
    import torch

    _, calls = tree
    B.build()
    calls()
    monkeypatch.setattr(torch, "__version__", torch.__version__ + "+other")
    assert not B.host_usable()
    B.build()
    assert calls() == ["cxx"] and B.host_usable()


def test_library_is_linked_when_the_extension_module_fails(tree):
    """A failed host compile must not leave new objects beside an old library that the next build takes for current."""
    root, calls = tree
    B.build()
    old = B.lib_path().stat().st_mtime_ns
    for f in ("csrc/a.cu", "csrc_host/b.cpp"):
        os.utime(root / f, (B.lib_path().stat().st_mtime + 10,) * 2)
    (root / "cxx_broken").touch()
    with pytest.raises(RuntimeError, match="compiler failed"):
        B.build()
    assert B.lib_path().stat().st_mtime_ns > old


def test_library_is_linked_again_when_an_object_is_newer(tree):
    root, calls = tree
    B.build()
    calls()
    os.utime(B.LIBDIR / "a.o", (B.lib_path().stat().st_mtime + 10,) * 2)
    B.build()
    assert calls() == ["nvcc"]


def test_missing_host_sources_are_named(tree):
    root, calls = tree
    (root / "csrc_host" / "b.cpp").unlink()
    with pytest.raises(RuntimeError, match="no sources of the autograd nodes"):
        B.build()
    assert calls() == ["nvcc", "nvcc"]                         # the library is built all the same


def test_changed_declarations_rebuild_both(tree):
    root, calls = tree
    B.build()
    calls()
    (root / "csrc" / "entries.h").write_text("int changed();")
    os.utime(root / "csrc" / "entries.h", (B.lib_path().stat().st_mtime + 10,) * 2)
    B.build()
    assert calls() == ["cxx", "nvcc", "nvcc"]


@pytest.mark.parametrize("entry", ["int tplr_abi() { return -1; }", "int other() { return 0; }"])
def test_nodes_refuse_a_library_of_other_declarations(entry, tmp_path):
    """Before any of its entries is taken: a changed argument list would hand shifted arguments to a kernel."""
    import shutil
    import subprocess

    from templar_b200.ops import native

    if shutil.which("gcc") is None:
        pytest.skip("no C compiler for the stand-in library")
    (tmp_path / "l.c").write_text(entry)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "l.so"), str(tmp_path / "l.c")], check=True)
    with pytest.raises(RuntimeError, match="entry declarations|tplr_abi is missing"):
        native.host().bind(str(tmp_path / "l.so"))
    native.host().bind(str(B.lib_path()))


def test_operators_keep_their_python_nodes_without_the_extension_module(monkeypatch):
    """Said once; an error where nothing but the native path is wanted."""
    from templar_b200.ops import native

    def broken(*a):
        raise RuntimeError("compiler failed: no such thing")

    monkeypatch.setattr(native, "_host", None)
    monkeypatch.setattr(B, "host_usable", lambda: False)
    monkeypatch.setattr(B, "build_host", broken)
    monkeypatch.setenv("TPLR_STRICT_NATIVE", "1")
    with pytest.raises(RuntimeError, match="compiler failed"):
        native.host()
    monkeypatch.delenv("TPLR_STRICT_NATIVE")
    with pytest.warns(RuntimeWarning, match="using the Python nodes"):
        assert native.host() is None
    import warnings

    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert native.host() is None
    native.launch_count = 5
    assert native.launch_count == 5
