"""mflux_b200/_host.so belongs to one torch and one Python: another one's is built again, never called, and never needed."""
import subprocess
import sys
import types

import pytest


@pytest.fixture
def fresh(lib_built, monkeypatch):
    """The loader and the call as in a new process."""
    from mflux_b200 import _lib, ops

    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "_host_module", None)
    monkeypatch.setattr(ops, "_native", None)
    return _lib, ops


def _module(monkeypatch, module):
    import mflux_b200

    monkeypatch.delattr(mflux_b200, "_host", raising=False)
    monkeypatch.setitem(sys.modules, "mflux_b200._host", module)


def test_the_library_loads_without_the_module(fresh, monkeypatch):
    _lib, ops = fresh
    _module(monkeypatch, None)                       # importing it raises ImportError
    assert _lib.load().mfx_version() > 0
    with pytest.warns(RuntimeWarning, match="does not load.*mflux_b200.build"):
        assert ops.plain_qlinear(*[None] * 6, 4, 64, None) is None
    assert ops.plain_qlinear(*[None] * 6, 4, 64, None) is None      # said once


@pytest.mark.parametrize("built_for", ["torch 1.0 cpython-30", None])
def test_a_module_of_another_torch_is_not_called(fresh, monkeypatch, built_for):
    _lib, ops = fresh

    def refuse(*args):
        raise AssertionError("called")

    module = types.ModuleType("mflux_b200._host")
    module.linear = module.bind = refuse
    if built_for:
        module.BUILT_FOR = built_for
    _module(monkeypatch, module)
    with pytest.warns(RuntimeWarning, match=f"was built for {built_for or 'an unknown torch'}"):
        assert ops.plain_qlinear(*[None] * 6, 4, 64, None) is None


def test_the_module_built_here_is_used(fresh, recwarn):
    from mflux_b200 import build

    _lib, _ = fresh
    assert _lib._host().BUILT_FOR == build.host_builds_for()
    assert not [w for w in recwarn if "_host.so" in str(w.message)]


def test_built_again_for_another_torch(lib_built, tmp_path, monkeypatch):
    from mflux_b200 import build

    commands = []

    def run(cmd, **kw):
        commands.append(cmd)
        (tmp_path / "_host.so").write_text("")
        return subprocess.CompletedProcess(cmd, 0, "", "")

    monkeypatch.setattr(build, "HOST", tmp_path / "_host.so")
    monkeypatch.setattr(build, "OBJ", tmp_path)
    monkeypatch.setattr(build.subprocess, "run", run)
    for expected in (1, 1):                          # built once, then up to date
        build.build_host(False, [])
        assert len(commands) == expected
    monkeypatch.setattr(build, "host_builds_for", lambda: "torch 99.0 cpython-30")
    for expected in (2, 2):
        build.build_host(False, [])
        assert len(commands) == expected
    assert any("torch 99.0" in part for part in commands[-1])
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: subprocess.CompletedProcess(cmd, 1, "", "no"))
    monkeypatch.setattr(build, "host_builds_for", lambda: "torch 100.0 cpython-30")
    with pytest.raises(RuntimeError):
        build.build_host(False, [])
    monkeypatch.setattr(build, "host_builds_for", lambda: "torch 99.0 cpython-30")
    monkeypatch.setattr(build.subprocess, "run", run)
    build.build_host(False, [])                      # nothing is taken for granted after a failure
    assert len(commands) == 3
