"""The native module that launches a prompt step's kernels (csrc/host.cpp) as a thing that can be done without, and its build's name."""
from types import SimpleNamespace

import pytest

from qwenforge_b200 import ops
from qwenforge_b200.csrc import KernelLibraryError, build


def _without(monkeypatch):
    """A machine on which host.cpp cannot be compiled; returns what was tried."""
    tried = []

    def refuse(name):
        tried.append(name)
        raise KernelLibraryError(f"{name}: no Python.h")
    monkeypatch.setattr(build, "_modules", {})
    monkeypatch.setattr(build, "_unavailable", {})
    monkeypatch.setattr(build, "_compile", refuse)
    monkeypatch.setattr(ops.host, "_module", None)
    return tried


def test_a_model_is_prepared_without_it(monkeypatch, capsys):
    tried = _without(monkeypatch)
    build.prepare({"host"})
    assert "no Python.h" in capsys.readouterr().err
    build.prepare({"host"})
    assert tried == ["host"]                                   # (one attempt, however many models)
    monkeypatch.setattr(build, "library_names", lambda: ["host"])
    with pytest.raises(KernelLibraryError, match="Python.h"):   # whoever builds everything hears of it
        build.build_all()


def test_its_functions_answer_none_without_it(monkeypatch):
    tried = _without(monkeypatch)
    before, rows = ops.kernels.launches, SimpleNamespace(is_cuda=True)
    assert ops.host.rms_norm(rows, None, None, 1e-6) is None and ops.host.rms_norm(rows, None, None, 1e-6) is None
    assert tried == ["host"] and ops.kernels.launches == before


@pytest.mark.parametrize("name", ["host", "norm"])
def test_changed_flags_are_another_build(name, monkeypatch):
    before, flags = build._digest(name), build._flags
    monkeypatch.setattr(build, "_flags", lambda which: [*flags(which), "-DANOTHER"])
    assert build._digest(name) != before
