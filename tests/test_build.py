"""The build without a working compiler for the extension module: the library is linked all the same, a word says what is missing, and no older module stays."""
import subprocess

import pytest

from jasmine_b200 import build


@pytest.fixture
def small_tree(tmp_path, monkeypatch):
    """The build of objects that are there already, in a folder of its own."""
    (tmp_path / "one.c").write_text("typedef int nothing;\n")
    subprocess.run(["gcc", "-fPIC", "-c", "one.c", "-o", "one.o"], cwd=tmp_path, check=True)
    for name, path in (("OBJ", "build"), ("LIB", "lib.so"), ("CALLS", "_native.so")):
        monkeypatch.setattr(build, name, tmp_path / path)
    monkeypatch.setattr(build, "_compile", lambda src, force, verbose: tmp_path / "one.o")
    return tmp_path


@pytest.mark.parametrize("cxx", ["/bin/false", "/nowhere/g++"])
def test_the_library_does_without_the_extension(small_tree, monkeypatch, capsys, cxx):
    monkeypatch.setenv("CXX", cxx)
    (small_tree / "_native.so").write_bytes(b"from other sources")
    assert build.build() == small_tree / "lib.so" and (small_tree / "lib.so").exists()
    assert "_native.so was not built" in capsys.readouterr().err
    assert not (small_tree / "_native.so").exists()
