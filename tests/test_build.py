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
