"""What `inferi_b200.build` builds and when: the library alone decides, the Python binding comes with it where there is a torch to compile it against."""
import os
import sys
import types

import pytest
import torch

from inferi_b200 import build, ops

COMPILER = """#!/bin/sh
echo {name} >> {log}
while [ $# -gt 0 ]; do [ "$1" = -o ] && out=$2; shift; done
{act}
"""


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A package folder with one source and compilers that note their calls"""
    csrc, log = tmp_path / "csrc", tmp_path / "log"
    csrc.mkdir()
    for f in ("one.cu", "binding.cpp"):
        (csrc / f).write_text("")

    def compiler(name, act="echo made > $out"):
        path = tmp_path / name
        path.write_text(COMPILER.format(name=name, log=log, act=act))
        path.chmod(0o755)
        return str(path)

    def calls():
        names = log.read_text().split() if log.exists() else []
        log.unlink(missing_ok=True)
        return sorted(names)

    def sources_at(when):
        for f in (csrc / "one.cu", csrc / "binding.cpp"):
            os.utime(f, (when, when))

    sources_at(os.path.getmtime(build.__file__))
    monkeypatch.setattr(build, "PKG_DIR", str(tmp_path))
    monkeypatch.setattr(build, "CSRC", str(csrc))
    monkeypatch.setattr(build, "LIB_PATH", str(tmp_path / "lib.so"))
    monkeypatch.setattr(build, "BINDING_PATH", str(tmp_path / "binding.so"))
    monkeypatch.setattr(build, "BINDING_SOURCES", [str(csrc / "binding.cpp"), build.__file__])
    monkeypatch.setattr(build, "SOURCES", ["one.cu"])
    monkeypatch.setattr(build, "_nvcc", lambda: compiler("nvcc"))
    monkeypatch.setenv("CXX", compiler("cxx", f'echo "{build.binding_stamp()}" > $out'))
    return types.SimpleNamespace(path=tmp_path, csrc=csrc, compiler=compiler, calls=calls)


LIBRARY = ["nvcc", "nvcc"]   # compiled and linked
with_cuda = pytest.mark.skipif(torch.version.cuda is None, reason="a torch without CUDA has no binding")


@with_cuda
def test_nothing_is_built_twice(tree):
    build.build()
    assert tree.calls() == ["cxx"] + LIBRARY
    build.build()
    assert tree.calls() == []
    os.utime(tree.csrc / "binding.cpp")
    build.build()
    assert tree.calls() == ["cxx"]
    os.utime(tree.csrc / "one.cu")
    build.build()
    assert tree.calls() == LIBRARY
    build.build(force=True)
    assert tree.calls() == ["cxx"] + LIBRARY


@with_cuda
@pytest.mark.parametrize("broken", ["fails", "is missing"])
def test_the_library_does_not_depend_on_the_binding(tree, monkeypatch, broken):
    build.build()
    monkeypatch.setenv("CXX", tree.compiler("cxx", "exit 1") if broken == "fails" else str(tree.path / "no such compiler"))
    build.build(force=True)
    assert os.path.exists(build.LIB_PATH) and not os.path.exists(build.BINDING_PATH)   # (nor an old binding)
    tree.calls()
    build.build()
    assert "nvcc" not in tree.calls()


def test_a_library_that_does_not_compile_is_an_error(tree, monkeypatch):
    monkeypatch.setattr(build, "_nvcc", lambda: tree.compiler("nvcc", "exit 1"))
    with pytest.raises(RuntimeError):
        build.build()


@pytest.mark.parametrize("kind", ["without CUDA", "missing"])
def test_a_torch_that_has_no_binding(tree, monkeypatch, kind):
    if kind == "missing":
        monkeypatch.setitem(sys.modules, "torch", None)
    else:
        monkeypatch.setattr(torch.version, "cuda", None)
    build.build()
    assert tree.calls() == LIBRARY
    build.build()
    assert tree.calls() == []


@with_cuda
def test_a_binding_of_another_torch_is_built_again(tree, monkeypatch):
    build.build()
    tree.calls()
    monkeypatch.setattr(build, "binding_stamp", lambda: "torch of tomorrow")
    build.build()
    assert tree.calls() == ["cxx"]


@pytest.mark.parametrize("stamp", [None, "torch of yesterday"])
def test_a_binding_of_another_torch_is_not_used(monkeypatch, stamp):
    other = types.SimpleNamespace(**({"stamp": stamp} if stamp else {}))
    monkeypatch.setitem(sys.modules, "inferi_b200._binding", other)
    assert ops._load_binding() is ops._NoBinding
    other.stamp = build.binding_stamp()
    assert ops._load_binding() is other
