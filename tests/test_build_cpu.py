"""What is built, and when, without running a compiler: the library for callers of the C ABI, who have neither Python nor torch,
and the tensor front end, which fits one interpreter and one build of torch."""
import os
import re
import sys
import types

import pytest

from tracea_b200 import build, ops


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """Targets in an empty folder; compilers that only write their output file. Returns the list of what they were run for."""
    runs = []

    def run(cmd, what):
        runs.append(what)
        with open(cmd[cmd.index("-o") + 1], "w") as f:
            f.write(what)

    monkeypatch.setattr(build, "_run", run)
    for name in ("LIB", "NATIVE", "NATIVE_STAMP", "UNTAGGED_NATIVE"):
        monkeypatch.setattr(build, name, str(tmp_path / os.path.basename(getattr(build, name, name))), raising=False)
    return runs


def test_without_torch_the_library_is_built_alone(tree, monkeypatch):
    monkeypatch.setitem(sys.modules, "torch", None)
    assert build.build() == build.LIB and os.path.exists(build.LIB)
    assert tree == ["nvcc"] and not build.needs_build()


def test_the_library_can_be_asked_for_alone(tree):
    build.build(library_only=True)
    assert tree == ["nvcc"]
    build.build()
    assert tree == ["nvcc", "c++"] and not build.needs_build()


def test_the_front_end_is_rebuilt_for_another_torch_or_interpreter(tree, monkeypatch):
    build.build()
    assert tree == ["nvcc", "c++"]
    build.build()
    assert tree == ["nvcc", "c++"]
    fits = build._torch_build()
    for other in (fits.replace(" torch ", " torch 1."), "." + fits, fits.rstrip()[:-1] + "\n"):
        with open(build.NATIVE_STAMP, "w") as f:
            f.write(other)
        assert build.needs_build()
        del tree[:]
        build.build()
        assert tree == ["c++"] and not build.needs_build()
    with open(build.UNTAGGED_NATIVE, "w") as f:      # every interpreter would import it
        f.write("")
    build.build()
    assert not os.path.exists(build.UNTAGGED_NATIVE)


def test_a_front_end_of_another_torch_is_refused(monkeypatch):
    import tracea_b200
    from tracea_b200 import ffi
    other = types.SimpleNamespace(torch_version="1.0.0")
    monkeypatch.setitem(sys.modules, "tracea_b200._ops_native", other)
    monkeypatch.setattr(tracea_b200, "_ops_native", other, raising=False)
    monkeypatch.setattr(ops, "_native_module", None)
    monkeypatch.setattr(ffi, "load", lambda: None)
    with pytest.raises(ImportError, match="built for torch 1.0.0"):
        ops._native()


def test_kernels_read_tensors_with_ordinary_loads():
    """A programmatic launch is resident while its predecessors write what it reads, which the non-coherent loads do not allow."""
    for path in build.SOURCES + build.HEADERS:
        with open(path) as f:
            code = "\n".join(line.split("//")[0] for line in f)
        assert not re.search(r"\b__ldg\b|ld\.global\S*\.nc|__builtin_nontemporal_load|__ldlu", code), path
