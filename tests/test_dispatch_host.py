"""Host path of the per-op calls (dispatch.c) without a device: what it refuses, in the order and with the errors that the ops name."""
import pytest
import torch

from wgml_b200 import _lib, ops

CPU = torch.zeros(8)


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
