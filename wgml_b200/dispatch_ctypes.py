"""The calls of dispatch.c over ctypes, for installations where that module cannot be built: the same checks, in the same order, with
the same errors, at 4 to 5 us more of host time a call."""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from ._lib import AttnParams, ERR_INVALID, RopeConfig, WgbError, check


def _f32(t, name):
    if not (isinstance(t, torch.Tensor) and t.is_cuda and t.dtype == torch.float32 and t.is_contiguous()):
        raise TypeError(f"{name}: expected a contiguous float32 CUDA tensor")
    return t.data_ptr()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def gemv(out, m, v):
    if v.numel() != m.ncols or out.numel() != m.nrows:
        raise WgbError(ERR_INVALID, "Gemv: dimension mismatch.")
    check(_lib.load().wgb_gemv_quant(m._h, _f32(v, "v"), _f32(out, "out"), _stream()))


def _gemm(entry, out, m, v):
    if v.dim() != 2 or out.dim() != 2 or v.shape[1] != m.ncols or out.shape[1] != m.nrows or v.shape[0] != out.shape[0]:
        raise WgbError(ERR_INVALID, "Gemm: dimension mismatch.")
    check(entry(m._h, _f32(v, "v"), v.shape[0], _f32(out, "out"), _stream()))


def gemm_q4k(out, m, v):
    _gemm(_lib.load().wgb_gemm_q4k_tiles, out, m, v)


def gemm_q6k(out, m, v):
    _gemm(_lib.load().wgb_gemm_q6k_tiles, out, m, v)


def gemm_q80(out, m, v):
    _gemm(_lib.load().wgb_gemm_q80_tiles, out, m, v)


def rms_norm(result, value, weight, eps):
    n = value.numel()
    if weight.numel() != n or result.numel() != n:
        raise WgbError(ERR_INVALID, "RmsNorm: dimension mismatch.")
    check(_lib.load().wgb_rms_norm(_f32(result, "result"), _f32(value, "value"), _f32(weight, "weight"), n, eps, _stream()))


def rope(variant, config, q, k):
    if not isinstance(config, RopeConfig):
        raise TypeError("shape: expected a RoPEConfig")
    check(_lib.load().wgb_rope(int(variant), C.byref(config), _f32(q, "in_out_q"), q.numel(), _f32(k, "in_out_k"), k.numel(), _stream()))


def attention(params, q, key_cache, value_cache, attn, xb):
    if not isinstance(params, AttnParams):
        raise TypeError("params: expected BatchedMultiqueryAttentionParams")
    need = params.seq_len * params.kv_dim
    if key_cache.numel() < need or value_cache.numel() < need or q.numel() != params.n_heads * params.head_size \
            or xb.numel() != q.numel() or (attn is not None and attn.numel() < params.n_heads * params.seq_len):
        raise WgbError(ERR_INVALID, "attention: dimension mismatch.")
    check(_lib.load().wgb_attention(C.byref(params), _f32(q, "q"), _f32(key_cache, "key_cache"), _f32(value_cache, "value_cache"),
                                    None if attn is None else _f32(attn, "attn"), _f32(xb, "xb"), _stream()))


def silu(h1, h2):
    if h1.numel() != h2.numel():
        raise WgbError(ERR_INVALID, "Silu: dimension mismatch.")
    check(_lib.load().wgb_silu(_f32(h1, "in_out_h1"), _f32(h2, "in_h2"), h1.numel(), _stream()))


def op_assign(variant, lhs, rhs):
    if lhs.numel() != rhs.numel():
        raise WgbError(ERR_INVALID, "OpAssign: dimension mismatch.")
    check(_lib.load().wgb_op_assign(int(variant), _f32(lhs, "lhs"), _f32(rhs, "rhs"), lhs.numel(), _stream()))
