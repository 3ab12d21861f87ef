"""The build of the optional extension: the library does not depend on it, and another torch or interpreter is noticed."""
import os
import types

import pytest

from bitladder_b200 import bit_decode_interface as I, build as b


@pytest.fixture
def commands(monkeypatch, tmp_path):
    """Every command that a build runs, none of them executed; g++ fails if `failing`."""
    ran = []

    def run(cmd, **_):
        ran.append(cmd)
        broken = cmd[0] == "g++" and run.failing
        if not broken:
            open(cmd[cmd.index("-o") + 1], "w").close()
        return types.SimpleNamespace(returncode=int(broken), stdout="", stderr="no headers")

    run.failing = False
    monkeypatch.delenv("CXX", raising=False)
    monkeypatch.setattr(b.subprocess, "run", run)
    for name, path in (("BUILD_DIR", tmp_path), ("LIB_PATH", tmp_path / "lib.so"), ("CALLS_PATH", tmp_path / "calls.so")):
        monkeypatch.setattr(b, name, str(path))
    ran.append(run)
    return ran


def test_the_library_is_built_where_the_extension_cannot_be(commands):
    commands[0].failing = True
    with pytest.warns(UserWarning, match="no headers"):
        assert b.build() == b.LIB_PATH
    assert any(c[0] != "g++" and "-shared" in c for c in commands[1:]) and os.path.exists(b.LIB_PATH)


def test_a_failed_extension_leaves_no_old_one(commands):
    b.build()
    assert os.path.exists(b.CALLS_PATH)
    commands[0].failing = True
    with pytest.warns(UserWarning):
        b.build(force=True)
    assert not os.path.exists(b.CALLS_PATH)


def test_another_torch_is_noticed(commands, monkeypatch):
    import torch
    b.build()
    del commands[1:]
    b.build()
    assert len(commands) == 1                        # all as it was
    monkeypatch.setattr(torch, "__version__", "0.0")
    b.build()
    assert [c[0] for c in commands[1:]] == ["g++"]


def test_an_extension_for_another_torch_is_not_taken(monkeypatch):
    from bitladder_b200 import _torch_calls
    monkeypatch.setattr(I, "_CALLS", None)
    assert I._calls() is _torch_calls
    monkeypatch.setattr(I, "_CALLS", None)
    monkeypatch.setattr(b, "calls_key", lambda: "torch 0.0")
    with pytest.warns(UserWarning, match="torch 0.0"):
        assert I._calls() is I._InterpretedCalls
