"""The extension of the compiled entry points is rebuilt when Python or torch changed, and not used with another torch."""
import os
import types

import pytest

from boostr_b200 import build, tensor


def test_current_only_for_this_python_and_torch(monkeypatch, tmp_path):
    build.build()
    assert build._host_current()
    monkeypatch.setattr(build.importlib.metadata, "version", lambda name: "0.0.1")
    assert not build._host_current()  # another torch
    monkeypatch.undo()
    monkeypatch.setattr(build, "HOST_LIB", build.HOST_LIB.replace("cpython-", "cpython-x"))
    assert not build._host_current()  # another Python
    monkeypatch.undo()
    monkeypatch.setattr(build, "HOST_STAMP", str(tmp_path / "none"))
    assert not build._host_current()  # after a forced build has cleared the objects
    monkeypatch.undo()
    assert build._host_current() and not os.path.exists(os.path.join(build.HERE, "_hostops.so"))


def test_module_of_another_torch_is_not_used(monkeypatch):
    import boostr_b200

    other = types.SimpleNamespace(torch_version="0.0.1", make_ref=None)
    monkeypatch.setattr(tensor, "_hostops", None)
    monkeypatch.setitem(__import__("sys").modules, "boostr_b200._hostops", other)
    monkeypatch.setattr(boostr_b200, "_hostops", other, raising=False)
    with pytest.warns(RuntimeWarning, match="compiled against torch 0.0.1"):
        assert tensor.hostops() is tensor._PythonForms
