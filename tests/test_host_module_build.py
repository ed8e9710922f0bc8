"""The compiled host module as a file: its name goes by everything it depends on, it appears whole or not at all, and where it cannot be
built or loaded the calls take the Python way."""
import os
import stat

import pytest
import torch

from test_operator_b200 import build, op


@pytest.fixture
def lib_dir(tmp_path, monkeypatch):
    monkeypatch.setattr(build, "LIB_DIR", str(tmp_path / "lib"))
    os.makedirs(build.LIB_DIR)
    return build.LIB_DIR


def _copied(path, tmp_path, extra):
    new = tmp_path / os.path.basename(path)
    with open(path) as f:
        new.write_text(f.read() + extra)
    return str(new)


def test_the_name_goes_by_torch_and_by_the_sources(monkeypatch, tmp_path):
    here = build.host_path()
    assert build.host_path() == here
    names = {here}
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0.0")
        names.add(build.host_path())
    for what in ("HOST_SOURCE", "HOST_HEADER"):
        with monkeypatch.context() as m:
            m.setattr(build, what, _copied(getattr(build, what), tmp_path, "// another one\n"))
            names.add(build.host_path())
    assert len(names) == 4


@pytest.mark.parametrize("fails", [True, False])
def test_a_file_appears_whole_or_not_at_all(lib_dir, tmp_path, fails):
    path = os.path.join(lib_dir, "out.so")
    seen = str(tmp_path / "seen")
    compiler = tmp_path / "compiler"
    compiler.write_text(f'#!/bin/sh\nprintf half > "$2"\nls "{lib_dir}" > "{seen}"\nprintf whole > "$2"\nexit {int(fails)}\n')
    compiler.chmod(compiler.stat().st_mode | stat.S_IXUSR)
    if fails:
        with pytest.raises(RuntimeError):
            build._compile([str(compiler)], path, "log", False)
    else:
        build._compile([str(compiler)], path, "log", False)
    with open(seen) as f:
        assert "out.so" not in f.read().split()
    assert sorted(os.listdir(lib_dir)) == (["log"] if fails else ["log", "out.so"])
    if not fails:
        with open(path) as f:
            assert f.read() == "whole"


def test_a_module_that_cannot_be_loaded(lib_dir):
    with open(build.host_path(), "wb") as f:
        f.write(b"\x7fELF and then half of a file")
    with pytest.warns(UserWarning, match="host module"):
        assert op._load_host(op.load_library()) is op._NoNativeHost


def test_a_module_that_cannot_be_built_though_another_is_there(lib_dir, monkeypatch):
    with open(os.path.join(lib_dir, "_smla_host.so"), "wb") as f:
        f.write(b"one of other sources")

    def no_compiler(*_):
        raise RuntimeError("no compiler")
    monkeypatch.setattr(build, "build_host", no_compiler)
    with pytest.warns(UserWarning, match="no compiler"):
        assert op._load_host(op.load_library()) is op._NoNativeHost
