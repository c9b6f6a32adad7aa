"""CPU: the build passes on what ptxas says about spilled registers."""
import importlib.util
import os
from types import SimpleNamespace

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _build_module():
    spec = importlib.util.spec_from_file_location(
        "hv_build_notes", os.path.join(ROOT, "hyper-vlasov_b200", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_spill_warnings_are_returned_beside_the_object(monkeypatch, tmp_path):
    b = _build_module()
    warning = "ptxas warning : Registers are spilled to local memory in function 'k', 136 bytes spill stores"
    calls = []

    def run(cmd, **kw):
        calls.append(cmd)
        return SimpleNamespace(returncode=0, stdout="", stderr=f"something else\n{warning}\n")

    monkeypatch.setattr(b.subprocess, "run", run)
    obj, err, notes = b.compile_one(str(tmp_path / "k.cu"), True)
    assert err is None and notes == [f"k.cu: {warning}"]
    assert "-warn-spills" in calls[0]


def test_a_failed_compilation_is_an_error(monkeypatch, tmp_path):
    b = _build_module()
    monkeypatch.setattr(b.subprocess, "run",
                        lambda cmd, **kw: SimpleNamespace(returncode=1, stdout="", stderr="no such file"))
    _, err, notes = b.compile_one(str(tmp_path / "k.cu"), True)
    assert "no such file" in err and notes == []
