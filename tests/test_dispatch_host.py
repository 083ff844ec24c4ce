"""Host path of the per-op calls (dispatch.c, or the same over ctypes) without a device: what it refuses, in the order and with the
errors that the ops name, and what an installation without a compiler gets."""
import ctypes
import os
import shutil
import subprocess
import sys

import pytest
import torch

from conftest import ROOT
from wgml_b200 import _lib, ops

CPU = torch.zeros(8)


@pytest.fixture(params=["module", "ctypes"], autouse=True)
def path(request, monkeypatch):
    fast = _lib._dispatch_module() if request.param == "module" else _lib._dispatch_ctypes()
    assert fast is not None
    monkeypatch.setattr(_lib, "_fast", fast)


class FakeMatrix:
    """What the module reads of a matrix or a tile set; no handle behind it."""
    nrows, ncols, _h = 8, 8, None


@pytest.mark.parametrize("call,message", [
    (lambda: ops.GemvQuant().dispatch(CPU, FakeMatrix(), torch.zeros(7)), "Gemv: dimension mismatch."),
    (lambda: ops.GemvQuant().dispatch(torch.zeros(7), FakeMatrix(), CPU), "Gemv: dimension mismatch."),
    (lambda: ops.Q4KTiles.gemm(FakeMatrix(), torch.zeros(2, 8), torch.zeros(3, 8)), "Gemm: dimension mismatch."),
    (lambda: ops.Q6KTiles.gemm(FakeMatrix(), torch.zeros(8), torch.zeros(1, 8)), "Gemm: dimension mismatch."),
    (lambda: ops.Q80Tiles.gemm(FakeMatrix(), torch.zeros(1, 9), torch.zeros(1, 8)), "Gemm: dimension mismatch."),
    (lambda: ops.RmsNorm().dispatch(ops.RmsNormConfig(1e-5), CPU, CPU, torch.zeros(7)), "RmsNorm: dimension mismatch."),
    (lambda: ops.RmsNorm().dispatch(ops.RmsNormConfig(1e-5), torch.zeros(7), CPU, CPU), "RmsNorm: dimension mismatch."),
    (lambda: ops.Silu().dispatch(CPU, torch.zeros(7)), "Silu: dimension mismatch."),
    (lambda: ops.BatchedMultiqueryAttention().dispatch(ops.BatchedMultiqueryAttentionParams(4, 8, 1, 1, 8, 0), CPU, CPU, CPU, None, CPU), "attention: dimension mismatch."),
    (lambda: ops.BatchedMultiqueryAttention().dispatch(ops.BatchedMultiqueryAttentionParams(1, 8, 1, 1, 8, 0), CPU, CPU, CPU, torch.zeros(0), CPU),
     "attention: dimension mismatch."),
])
def test_dimension_mismatches(call, message):
    with pytest.raises(ops.WgbError) as e:
        call()
    assert e.value.status == _lib.ERR_INVALID and e.value.message == message


@pytest.mark.parametrize("call,name", [
    (lambda: ops.Silu().dispatch(CPU, CPU), "in_out_h1"),
    (lambda: ops.Silu().dispatch(CPU.double(), CPU), "in_out_h1"),
    (lambda: ops.GemvQuant().dispatch(CPU, FakeMatrix(), CPU), "v"),                          # a handle of None is the library's to refuse
    (lambda: ops.Q4KTiles.gemm(FakeMatrix(), torch.zeros(2, 8), torch.zeros(2, 8)), "v"),
    (lambda: ops.RmsNorm().dispatch(ops.RmsNormConfig(1e-5), CPU, CPU, CPU), "result"),
    (lambda: ops.RoPE().dispatch(ops.RoPEVariant.Neox, ops.RoPEConfig(8, 8, 0, 1e4), CPU, CPU), "in_out_q"),
    (lambda: ops.BatchedMultiqueryAttention().dispatch(ops.BatchedMultiqueryAttentionParams(1, 8, 1, 1, 8, 0), CPU, CPU, CPU, None, CPU), "q"),
])
def test_tensors_off_the_device_are_refused_by_name(call, name):
    with pytest.raises(TypeError, match=f"^{name}: expected a contiguous float32 CUDA tensor$"):
        call()


def test_other_arguments():
    d = _lib.dispatch()
    with pytest.raises(TypeError):
        d.gemv(CPU, FakeMatrix())
    with pytest.raises(TypeError):
        d.rms_norm(CPU, CPU, CPU, "eps")
    with pytest.raises(TypeError):
        d.attention(b"short", CPU, CPU, CPU, None, CPU)
    with pytest.raises(AttributeError):
        d.silu(object(), CPU)
    with pytest.raises(AttributeError):
        d.gemv(CPU, object(), CPU)


def lookalike(cls, *values):
    """A structure of the same fields as `cls`, of a class of its own."""
    return type("Other", (ctypes.Structure,), {"_fields_": cls._fields_})(*values)


def test_parameter_structures_are_of_their_class_or_a_derived_one():
    """Any buffer of the right size is no parameter structure; one of a derived class with more fields is."""
    d = _lib.dispatch()
    attn, rope = (1, 8, 1, 1, 8, 0), (8, 8, 0, 1e4)
    for p in (bytes(24), lookalike(ops.BatchedMultiqueryAttentionParams, *attn)):
        with pytest.raises(TypeError, match="^params: expected BatchedMultiqueryAttentionParams$"):
            d.attention(p, CPU, CPU, CPU, None, CPU)
    for p in (bytes(16), lookalike(ops.RoPEConfig, *rope)):
        with pytest.raises(TypeError, match="^shape: expected a RoPEConfig$"):
            d.rope(0, p, CPU, CPU)
    for cls, values, call in ((ops.BatchedMultiqueryAttentionParams, attn, lambda p: d.attention(p, CPU, CPU, CPU, None, CPU)),
                              (ops.RoPEConfig, rope, lambda p: d.rope(0, p, CPU, CPU))):
        more = type("More", (cls,), {"_fields_": [("note", ctypes.c_uint32)]})
        with pytest.raises(TypeError, match="expected a contiguous float32 CUDA tensor$"):
            call(more(*values, 5))


def copied_package(tmp_path):
    """A copy of the package as another installation has it: sources, no built module."""
    dst = tmp_path / "wgml_b200"
    shutil.copytree(os.path.join(ROOT, "wgml_b200"), dst, ignore=shutil.ignore_patterns("*.so", "build", "__pycache__"))
    return dst


def in_copy(tmp_path, code, **env):
    return subprocess.run([sys.executable, "-c", code], cwd=tmp_path, capture_output=True, text=True, timeout=300,
                          env=dict(os.environ, PYTHONPATH=str(tmp_path), PYTHONDONTWRITEBYTECODE="1", **env))


def test_a_given_library_needs_no_compiler(tmp_path, path):
    """With the library named by WGML_B200_LIB and neither gcc nor nvcc to be found, the per-op calls reach their own checks."""
    copied_package(tmp_path)
    r = in_copy(tmp_path, "import torch\nfrom wgml_b200 import ops\nz = torch.zeros(8)\nops.Silu().dispatch(z, z)", PATH="/nonexistent",
                CUDA_HOME="/nonexistent", WGML_B200_LIB=_lib.LIB_PATH)
    assert "TypeError: in_out_h1: expected a contiguous float32 CUDA tensor" in r.stderr, r.stderr


def test_the_library_builds_without_python_headers(tmp_path, monkeypatch):
    """build() makes the library alone; the host module is a step of its own."""
    from wgml_b200 import build
    monkeypatch.setattr(build, "EXT", str(tmp_path / "module.so"))
    build.build()
    assert not (tmp_path / "module.so").exists()
    build.build_dispatch()
    assert (tmp_path / "module.so").exists()


def test_a_module_of_another_interpreter_is_left_alone(tmp_path):
    """A file without this interpreter's tag (here not even a library) is not loaded; this one's is built beside it."""
    pkg = copied_package(tmp_path)
    (pkg / "_dispatch.so").write_bytes(b"built for another Python")
    (pkg / "_dispatch.cpython-399-other.so").write_bytes(b"the same")
    r = in_copy(tmp_path, "import torch\nfrom wgml_b200 import _lib, build, ops\nprint(_lib._dispatch_module().__file__ == build.EXT)\n"
                "z = torch.zeros(8)\nops.Silu().dispatch(z, z)", WGML_B200_LIB=_lib.LIB_PATH)
    assert "True" in r.stdout and "TypeError: in_out_h1: expected a contiguous float32 CUDA tensor" in r.stderr, r.stdout + r.stderr


def test_the_module_appears_whole(tmp_path, monkeypatch):
    """The compiler writes beside the module's name, which a finished file takes and a failed one does not."""
    from wgml_b200 import build
    ext = tmp_path / "module.so"
    monkeypatch.setattr(build, "EXT", str(ext))
    for rc in (1, 0):
        def gcc(cmd, **kw):
            assert not ext.exists()
            open(cmd[-1], "wb").write(b"half")
            assert not ext.exists()
            return subprocess.CompletedProcess(cmd, rc, "", "")
        monkeypatch.setattr(build.subprocess, "run", gcc)
        if rc:
            with pytest.raises(RuntimeError):
                build.build_dispatch()
            assert not list(tmp_path.iterdir())
        else:
            build.build_dispatch()
            assert list(tmp_path.iterdir()) == [ext]


def test_the_module_names_what_it_calls():
    """The addresses handed over are those of the module's own list, so a module and a library of different versions cannot disagree on it."""
    assert set(_lib._dispatch_module().ENTRY_POINTS) <= set(_lib.SIGNATURES)
