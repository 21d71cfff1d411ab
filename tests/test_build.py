"""What `build` does where torch is missing or another one than the module was built with (nothing is compiled here)."""
import sys

import pytest

from cnet_b200 import build


def test_the_library_is_built_without_torch(monkeypatch, tmp_path, capsys):
    monkeypatch.setitem(sys.modules, "torch", None)
    monkeypatch.setattr(build, "OPS", str(tmp_path / "ops_native.so"))
    monkeypatch.setattr(build, "_build_lib", lambda force, verbose: "the library")
    assert build.build() == build.build(force=True) == "the library"
    assert not (tmp_path / "ops_native.so").exists() and "torch" in capsys.readouterr().err


def test_the_module_is_built_anew_for_another_torch_or_python(monkeypatch, tmp_path):
    """Under another key it is out of date, and no half-written file stands in its place meanwhile."""
    monkeypatch.setattr(build, "OPS", str(tmp_path / "ops_native.so"))
    monkeypatch.setattr(build, "OPS_KEY", str(tmp_path / "build" / "key"))
    made = []

    def compiler(cmd, **kw):
        out = cmd[cmd.index("-o") + 1]
        assert out != build.OPS
        made.append(out)
        open(out, "w").write("module %d" % len(made))
        return type("R", (), {"returncode": int(len(made) == 3), "stdout": b"message"})

    monkeypatch.setattr(build.subprocess, "run", compiler)
    assert not build._ops_up_to_date()
    build._build_ops({})
    assert build._ops_up_to_date() and open(build.OPS).read() == "module 1"
    monkeypatch.setattr(build, "ops_key", lambda: "another")
    assert not build._ops_up_to_date()
    build._build_ops({})
    assert build._ops_up_to_date() and open(build.OPS).read() == "module 2"
    with pytest.raises(RuntimeError, match="message"):
        build._build_ops({})
    assert open(build.OPS).read() == "module 2" and sorted(p.name for p in tmp_path.iterdir()) == ["build", "ops_native.so"]


def test_a_module_of_another_torch_or_python_is_not_used(monkeypatch):
    from cnet_b200 import lib, ops
    build.build()
    monkeypatch.setattr(ops, "_native", None)
    assert ops._load_native().built_for == build.ops_key()
    monkeypatch.setattr(ops, "_native", None)
    monkeypatch.setattr(build, "ops_key", lambda: "another")
    with pytest.raises(lib.CnetError, match="built for another"):
        ops._load_native()
