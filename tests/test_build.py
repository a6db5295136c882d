"""What `python -m gelib_b200.build` does about the native host side, whose file is tied to a torch and a Python.  Nothing is
compiled here: the compiler is a stand-in that writes a file."""
import os
import sys
import types

import pytest
import torch


@pytest.fixture
def builder(tmp_path, monkeypatch):
    from gelib_b200 import build as b
    calls = []

    def run(cmd, **kw):
        calls.append(cmd)
        with open(b.NATIVE, "w") as f:
            f.write("made by call %d" % len(calls))
        return types.SimpleNamespace(returncode=0, stdout="", stderr="")

    lib = tmp_path / "lib.so"
    lib.write_text("")
    os.utime(lib, (1, 1))
    monkeypatch.setattr(b, "LIB", str(lib))
    monkeypatch.setattr(b, "NATIVE", str(tmp_path / "_native.so"))
    monkeypatch.setattr(b, "OBJ", str(tmp_path))
    monkeypatch.setattr(b, "build_library", lambda *a: str(lib))
    monkeypatch.setattr(b.subprocess, "run", run)
    return types.SimpleNamespace(b=b, calls=calls, build=b.build)


def test_an_up_to_date_file_is_kept(builder):
    builder.build()
    builder.build()
    assert len(builder.calls) == 1


@pytest.mark.parametrize("change", ["torch", "python", "file"])
def test_a_file_for_another_torch_or_python_or_a_broken_one_is_built_again(builder, monkeypatch, change):
    builder.build()
    if change == "torch":
        monkeypatch.setattr(torch, "__version__", "0.0")
    if change == "python":
        monkeypatch.setattr(sys, "version", "0.0")
    if change == "file":
        with open(builder.b.NATIVE, "w") as f:
            f.write("broken")
    builder.build()
    assert len(builder.calls) == 2


def test_the_toolkits_headers_are_found_from_the_compilers_name_alone(builder, monkeypatch):
    if not os.path.exists(builder.b.NVCC):
        pytest.skip("no CUDA compiler here")
    monkeypatch.setenv("PATH", os.path.dirname(builder.b.NVCC) + os.pathsep + os.environ["PATH"])
    monkeypatch.setattr(builder.b, "NVCC", "nvcc")
    builder.build()
    include = [a[2:] for a in builder.calls[0] if a.startswith("-I")]
    assert any(os.path.exists(os.path.join(d, "cuda_runtime_api.h")) for d in include), include


def test_the_library_is_built_where_pythons_headers_are_missing(builder, monkeypatch, capsys):
    monkeypatch.setattr(builder.b.sysconfig, "get_paths", lambda: {"include": "/nonexistent"})
    assert builder.build() == builder.b.LIB
    assert builder.calls == [] and "Python.h" in capsys.readouterr().err


@pytest.mark.parametrize("how", ["missing", "another torch"])
def test_products_do_without_the_native_host_side(cabi, monkeypatch, how):
    import gelib_b200 as G
    module = None if how == "missing" else types.SimpleNamespace(torch_version="0.0")
    monkeypatch.setitem(sys.modules, "gelib_b200._native", module)
    monkeypatch.setattr(G._lib, "_native", None)
    x = G.SO3vec.randn(2, {0: 2, 1: 2})
    with pytest.warns(RuntimeWarning, match="_native.so"):
        with pytest.raises(RuntimeError, match="CUDA"):  # what the Python code says about CPU tensors
            x.CGproduct(x)
