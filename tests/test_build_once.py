"""Building the libraries: processes that start together on a fresh checkout, and what is left when a build cannot be done (no
GPU, no real compiler: a stand-in writes the library in two halves)."""
import os
import subprocess
import sys
import warnings

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multi-variate-parallel-transformer_b200")
COMPILER = """#!/bin/sh
while [ "$1" != "-o" ]; do shift; done
printf first > "$2"; sleep 3; printf second >> "$2"; echo built >> "$COUNT"
"""
PROCESS = """
import os, sys
sys.path.insert(0, {pkg!r})
import {module} as m
m.LIB_PATH, m.HASH_PATH = {lib!r}, {lib!r} + ".srchash"
{more}
m.build()
assert not m._stale(), "the digest is not that of the sources"
assert open({lib!r}).read() == "firstsecond", "half a library"
"""


@pytest.mark.parametrize("module, more", [
    ("mvpa_host", ""), ("mvpa_native", "m.shutil.which = lambda name: os.environ['CXX']\nm.sources = lambda: []")])
def test_processes_that_start_together(tmp_path, module, more):
    compiler, lib, count = tmp_path / "cc", str(tmp_path / "lib.so"), tmp_path / "count"
    compiler.write_text(COMPILER)
    compiler.chmod(0o755)
    env = dict(os.environ, CXX=str(compiler), COUNT=str(count))
    code = PROCESS.format(pkg=PKG, module=module, lib=lib, more=more)
    ps = [subprocess.Popen([sys.executable, "-c", code], env=env, stderr=subprocess.PIPE, text=True) for _ in range(4)]
    errors = [p.communicate(timeout=300)[1] for p in ps]
    assert all(p.returncode == 0 for p in ps), errors
    assert count.read_text() == "built\n"                                     # the others waited for the first
    assert sorted(os.listdir(tmp_path)) == ["cc", "count", "lib.so", "lib.so.srchash"]


def test_no_compiler_is_an_import_error(tmp_path, monkeypatch):
    sys.path.insert(0, PKG)
    import mvpa_host
    monkeypatch.setattr(mvpa_host, "LIB_PATH", str(tmp_path / "lib.so"))
    monkeypatch.setattr(mvpa_host, "HASH_PATH", str(tmp_path / "lib.so.srchash"))
    monkeypatch.setenv("CXX", str(tmp_path / "none"))
    with pytest.raises(ImportError):
        mvpa_host.build()
    assert not os.listdir(tmp_path)


def test_without_the_extension_python_serves(monkeypatch):
    sys.path.insert(0, PKG)
    import mvpa_host

    def refuse(force=False):
        raise ImportError("no compiler")

    monkeypatch.setattr(mvpa_host, "_module", None)
    monkeypatch.setattr(mvpa_host, "_refused", False)
    monkeypatch.setattr(mvpa_host, "build", refuse)
    with pytest.warns(RuntimeWarning, match="no compiler"):
        assert not mvpa_host.available()
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert not mvpa_host.available()           # (once)
