"""When the extension between torch and the C ABI is rebuilt."""
import os

import pytest

from rustorch_b200 import build


@pytest.fixture
def built(tmp_path, monkeypatch):
    """An extension newer than its sources, as a build of it for this interpreter and torch leaves it; a compiler that only
    notes that it was called."""
    calls = []

    class Done:
        returncode, stdout, stderr = 0, "", ""

    def run(cmd, **kw):
        calls.append(cmd[0])
        (tmp_path / "ext.so").write_bytes(b"")
        return Done()

    monkeypatch.setattr(build, "BINDING_PATH", str(tmp_path / "ext.so"))
    monkeypatch.setattr(build.subprocess, "run", run)
    build.build_binding(force=True)
    assert calls == ["g++"]
    calls.clear()
    return calls


def test_extension_in_order_is_left_alone(built):
    build.build_binding()
    assert built == []


@pytest.mark.parametrize("what", ["torch", "python", "source", "no record"])
def test_extension_for_something_else_is_rebuilt(built, monkeypatch, what):
    import torch
    if what == "torch":
        monkeypatch.setattr(torch, "__version__", "0.0.1")
    elif what == "python":
        monkeypatch.setattr(build.sys.implementation, "cache_tag", "cpython-00")
    elif what == "source":
        os.utime(build.BINDING_PATH, (1, 1))
    else:
        for name in os.listdir(os.path.dirname(build.BINDING_PATH)):
            if name.endswith(".stamp"):
                os.remove(os.path.join(os.path.dirname(build.BINDING_PATH), name))
    build.build_binding()
    assert built == ["g++"]
    build.build_binding()
    assert built == ["g++"]
