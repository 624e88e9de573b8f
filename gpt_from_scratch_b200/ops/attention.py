"""Causal flash attention (tcgen05 kernels in csrc/attention.cu) and its torch oracle.

Two entry points:

* :func:`apply_flash_attn` - the reference's public API (core/myFlashAttn.py:1321):
  ``q, k, v`` of shape ``[B, nh, S, D]`` -> ``[B, nh, S, D]``.
* :func:`fused_rope_attention` - what the model uses: takes the packed projection
  output ``[S*B, 3*nh*D]`` (row order ``[q|k|v] x heads x D``, the reference's layout,
  core/transformer_layer.py:42-44), rotates q and k in place, and runs attention
  straight out of that buffer, producing ``[S*B, nh*D]``. This removes the four
  permute/contiguous copies per layer that the reference pays
  (core/transformer_layer.py:52-61, core/myFlashAttn.py:206-208).
"""
from __future__ import annotations

import ctypes
import functools
import math

import torch

from . import _lib
from .rope import rope_inplace_native, rope_reference


def attention_reference(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, causal: bool = True,
                        scale: float | None = None) -> torch.Tensor:
    """Eager attention on ``[B, nh, S, D]`` tensors (materialises the S x S matrix)."""
    D = q.shape[-1]
    scale = 1.0 / math.sqrt(D) if scale is None else scale
    s = torch.matmul(q.float(), k.float().transpose(-1, -2)) * scale
    if causal:
        S = q.shape[-2]
        mask = torch.ones(S, S, dtype=torch.bool, device=q.device).tril()
        s = s.masked_fill(~mask, float("-inf"))
    p = torch.softmax(s, dim=-1)
    return torch.matmul(p, v.float()).to(q.dtype)


def _strides3(t: torch.Tensor) -> tuple[int, int, int]:
    """Element strides (sequence, batch, head) of a ``[S, B, nh, D]`` view."""
    s, b, h, d = t.stride()
    assert d == 1, "need a [S,B,nh,D] view with contiguous head_dim"
    return s, b, h


def _strides_bhsd(t: torch.Tensor) -> tuple[int, int, int]:
    """The same of a ``[B, nh, S, D]`` tensor."""
    b, h, s, d = t.stride()
    assert d == 1, "need contiguous head_dim"
    return s, b, h


_Strides12, _Strides24 = ctypes.c_longlong * 12, ctypes.c_longlong * 24


def _pad128(S: int) -> int:
    return (S + 127) // 128 * 128


def flash_fwd_native(q, k, v, out, causal: bool, scale: float) -> torch.Tensor:
    """q, k, v, out: logical ``[S, B, nh, D]`` views (any strides, head_dim contiguous). Returns the LSE
    (base 2), the form the backward wants it in."""
    S, B, nh, D = q.shape
    lse = torch.empty((B, nh, _pad128(S)), dtype=torch.float32, device=q.device)
    st = _Strides12(*_strides3(q), *_strides3(k), *_strides3(v), *_strides3(out))
    with _lib.nvtx("flash_attention_fwd"):
        rc = _lib.lib().gfs_flash_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), 0, lse.data_ptr(),
                                      S, B, nh, D, st, scale, 1 if causal else 0, 0, _lib.stream_ptr())
    _lib.check(rc, "gfs_flash_fwd")
    return lse


def flash_bwd_native(q, k, v, out, dout, lse, dq, dk, dv, causal: bool, scale: float, rope=None) -> None:
    """``rope = (cos, sin)``: dq and dk are rotated back (inverse RoPE) as they are written."""
    S, B, nh, D = q.shape
    dvec = torch.empty_like(lse)      # scratch of the pre-pass: rowsum(dO * O)
    st = _Strides24(*_strides3(q), *_strides3(k), *_strides3(v), *_strides3(out), *_strides3(dout),
                    *_strides3(dq), *_strides3(dk), *_strides3(dv))
    rc = _lib.lib().gfs_flash_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), dout.data_ptr(),
                                  lse.data_ptr(), dvec.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                                  S, B, nh, D, st, scale, 1 if causal else 0,
                                  rope[0].data_ptr() if rope else 0, rope[1].data_ptr() if rope else 0, 0,
                                  _lib.stream_ptr())
    _lib.check(rc, "gfs_flash_bwd")
    _lib.add_launches(2)  # pre-pass + two main kernels


@functools.lru_cache(maxsize=256)
def _contiguous_strides(n: int, B: int, nh: int, S: int, D: int):
    """ctypes array of the strides of ``n`` contiguous ``[B, nh, S, D]`` tensors."""
    return (ctypes.c_longlong * (3 * n))(*([D, nh * S * D, S * D] * n))


def _stride_array(*ts: torch.Tensor):
    for t in ts:
        if not t.is_contiguous():
            return (ctypes.c_longlong * (3 * len(ts)))(*[x for t in ts for x in _strides_bhsd(t)])
    return _contiguous_strides(len(ts), *ts[0].shape)


class _FlashAttnBHSD(torch.autograd.Function):
    """[B, nh, S, D] API on the native kernels, for bf16 tensors and for fp16 ones: the kernels are bf16, so
    fp16 inputs (the dtype of the reference's self-test, core/myFlashAttn.py:28-32) are rounded to bf16, which
    keeps 8 of their 11 significand bits, within the self-test's tolerances; results are stored as fp16."""

    @staticmethod
    def forward(ctx, q, k, v, causal, scale):
        B, nh, S, D = q.shape
        lib, stream = _lib.lib(), _lib.stream_ptr()
        out = torch.empty_like(q)
        lse = torch.empty((B, nh, _pad128(S)), dtype=torch.float32, device=q.device)
        pq, pk, pv = q.data_ptr(), k.data_ptr(), v.data_ptr()
        copy = None
        if q.dtype == torch.float16:
            qkv = torch.empty((3, B, nh, S, D), dtype=torch.bfloat16, device=q.device)
            src, n = (pq, pk, pv), 2 * B * nh * S * D
            pq = qkv.data_ptr()
            pk, pv = pq + n, pq + 2 * n
            _lib.check(lib.gfs_attn_cast_qkv(*src, pq, S, B, nh, D, _stride_array(q, k, v), stream),
                       "gfs_attn_cast_qkv")
            st = _stride_array(qkv[0], qkv[1], qkv[2], out) if not out.is_contiguous() else \
                _contiguous_strides(4, B, nh, S, D)
            # the backward reads a copy of the output: the caller may write to his (out += residual)
            copy = torch.empty_like(out) if any(ctx.needs_input_grad) else None
            ctx.save_for_backward(qkv, copy, lse)
        else:
            st = _stride_array(q, k, v, out)
            ctx.save_for_backward(q, k, v, out, lse)
        rc = lib.gfs_flash_fwd(pq, pk, pv, out.data_ptr(), _lib.ptr(copy), lse.data_ptr(), S, B, nh, D, st, scale, causal,
                               q.dtype == torch.float16, stream)
        _lib.check(rc, "gfs_flash_fwd")
        ctx.args = (causal, scale)
        return out

    @staticmethod
    def backward(ctx, dout):
        *qkv, out, lse = ctx.saved_tensors
        causal, scale = ctx.args
        B, nh, S, D = out.shape
        dout = _tma_ready(dout)
        f16 = len(qkv) == 1
        dob = 0
        if f16:
            qkv = qkv[0].unbind(0)
            copy = torch.empty_like(qkv[0])     # dout rounded to bf16, written by the pre-pass
            dob = copy.data_ptr()
        q, k, v = qkv
        dq, dk, dv = (torch.empty_like(t, dtype=out.dtype) for t in qkv)
        dvec = torch.empty_like(lse)
        rc = _lib.lib().gfs_flash_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), dout.data_ptr(),
                                      lse.data_ptr(), dvec.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                                      S, B, nh, D, _stride_array(q, k, v, out, dout, dq, dk, dv), scale, causal, 0, 0,
                                      dob, _lib.stream_ptr())
        _lib.check(rc, "gfs_flash_bwd")
        _lib.add_launches(2)  # pre-pass + two main kernels
        return dq, dk, dv, None, None


def _tma_ready(t: torch.Tensor) -> torch.Tensor:
    """``t`` itself if the kernels can read its layout, else a contiguous copy."""
    b, h, s, d = t.stride()
    if d == 1 and not ((b | h | s) & 7) and not t.data_ptr() & 15:
        return t
    return t.clone(memory_format=torch.contiguous_format)   # a copy also where t is contiguous, but at an odd address


def _first_keys(q: torch.Tensor, t: torch.Tensor) -> torch.Tensor:
    """The rows of a longer k or v that the kernels read: one per query. Anything shorter they would read past."""
    B, nh, S, D = q.shape
    if t.dim() != 4 or t.shape[:2] != (B, nh) or t.shape[2] < S or t.shape[3] != D:
        raise ValueError(f"apply_flash_attn: k and v of shape {tuple(t.shape)} do not cover q of shape {tuple(q.shape)}")
    return t[:, :, :S]


def apply_flash_attn(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, causal_mask: bool = True) -> torch.Tensor:
    """Flash attention on ``[B, nh, S, D]`` tensors (reference API, core/myFlashAttn.py:1321)."""
    D = q.shape[-1]
    scale = 1.0 / math.sqrt(D)
    if q.is_cuda and q.dtype in (torch.float16, torch.bfloat16):
        if D not in (64, 128):
            raise ValueError(f"apply_flash_attn: head_dim {D} has no native kernel (64 and 128 do); "
                             "use attention_reference for other sizes")
        if k.is_cuda and v.is_cuda and q.dtype == k.dtype == v.dtype:
            if k.shape != q.shape or v.shape != q.shape:
                k, v = _first_keys(q, k), _first_keys(q, v)
            return _FlashAttnBHSD.apply(_tma_ready(q), _tma_ready(k), _tma_ready(v), 1 if causal_mask else 0, scale)
    return attention_reference(q, k, v, causal_mask, scale)


class _FusedRopeAttention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv2d, cos, sin, S, B, nh, D, pre_rotated):
        qkv = qkv2d.view(S, B, 3, nh, D)
        if not pre_rotated:
            rope_inplace_native(qkv, cos, sin, S, B, nh, D, parts=2, token_stride=3 * nh * D, backward=False)
        out = torch.empty((S, B, nh, D), dtype=qkv2d.dtype, device=qkv2d.device)
        scale = 1.0 / math.sqrt(D)
        lse = flash_fwd_native(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], out, True, scale)
        ctx.save_for_backward(qkv2d, out, lse, cos, sin)
        ctx.dims = (S, B, nh, D, scale)
        return out.view(S * B, nh * D)

    @staticmethod
    def backward(ctx, dout2d):
        qkv2d, out, lse, cos, sin = ctx.saved_tensors
        S, B, nh, D, scale = ctx.dims
        qkv = qkv2d.view(S, B, 3, nh, D)
        dout = dout2d.contiguous().view(S, B, nh, D)
        dqkv = torch.empty_like(qkv)
        # the inverse rotation of dq / dk happens in the backward kernels' epilogues
        flash_bwd_native(qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], out, dout, lse,
                         dqkv[:, :, 0], dqkv[:, :, 1], dqkv[:, :, 2], True, scale, rope=(cos, sin))
        return dqkv.view(S * B, 3 * nh * D), None, None, None, None, None, None, None


def fused_rope_attention(qkv2d: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, S: int, B: int, nh: int,
                         D: int, pre_rotated: bool = False) -> torch.Tensor:
    """RoPE on q,k + causal attention from the packed ``[S*B, 3*nh*D]`` projection output.

    ``cos``/``sin`` are fp32 ``[>=S, D/2]`` tables. On CUDA bf16 the input buffer is
    rotated in place (it is an intermediate owned by the caller's projection), unless
    ``pre_rotated`` says the producing GEMM already rotated q and k in its epilogue; either
    way the returned gradient is w.r.t. the un-rotated projection output.
    """
    if qkv2d.is_cuda and qkv2d.dtype == torch.bfloat16 and D in (64, 128):
        return _FusedRopeAttention.apply(qkv2d.contiguous(), cos, sin, S, B, nh, D, pre_rotated)
    assert not pre_rotated, "pre_rotated inputs exist only on the native path"
    qkv = qkv2d.view(S, B, 3, nh, D)
    q, k, v = qkv.unbind(2)
    q = rope_reference(q, cos[:S], sin[:S])
    k = rope_reference(k, cos[:S], sin[:S])
    o = attention_reference(q.permute(1, 2, 0, 3), k.permute(1, 2, 0, 3), v.permute(1, 2, 0, 3), True)
    return o.permute(2, 0, 1, 3).reshape(S * B, nh * D)
