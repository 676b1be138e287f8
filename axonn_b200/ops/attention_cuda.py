"""Bindings of the flash-attention kernels (``csrc/flash_attn.cu``).

Forward and backward run on the package's tcgen05 kernels directly on the packed
QKV tensor (no split, no head repetition for grouped-query attention).
"""

import ctypes
import os

import torch
from torch.autograd.function import once_differentiable

from . import _lib
from .direct import host_paths, no_graph

_BWD_DEFAULT = "split"


def available():
    return hasattr(_lib.lib(), "axb_flash_attn_fwd") and os.environ.get("AXONN_FLASH", "1") == "1"


def supported(qkv, scale=1.0):
    """Whether the kernels take this packed tensor: bf16, head_dim 64 or 128, dense and 16-byte aligned, any sequence
    length, a positive softmax scale.  Traced, vmapped or subclassed tensors have no storage that a kernel could be
    given.  The scale: masked scores are -inf before they are multiplied by it and the row maximum is taken before the
    multiplication, so it has to be positive, and a normal fp32 number after the change to base 2 (the kernels flush
    denormals)."""
    B, S, G, n, D = qkv.shape
    if not 2.0 ** -100 < scale < 2.0 ** 100:
        return False
    if qkv.dtype != torch.bfloat16 or D not in (64, 128) or not qkv.is_contiguous() or qkv.numel() == 0 or n < 3:
        return False
    if S % 128:
        if torch.compiler.is_compiling() or torch._C._functorch.peek_interpreter_stack() is not None:
            return False
        if type(qkv) not in (torch.Tensor, torch.nn.Parameter):
            return False
    return qkv.data_ptr() % 16 == 0


def flash_fwd_packed(qkv, scale):
    """qkv [B, S, G, qpk+2, D] -> (out [B, S, G*qpk, D], lse [B, G*qpk, S])."""
    B, S, G, n, D = qkv.shape
    qpk = n - 2
    out = torch.empty((B, S, G * qpk, D), dtype=qkv.dtype, device=qkv.device)
    lse = torch.empty((B, G * qpk, S), dtype=torch.float32, device=qkv.device)
    st = _lib.lib().axb_flash_attn_fwd(_lib.addr(qkv), _lib.addr(out), _lib.addr(lse), B, S,
                                       G, qpk, D, scale,
                                       qkv.device.index, _lib.stream())
    _lib.check(st, "axb_flash_attn_fwd")
    return out, lse


def _bwd_split(qkv, out, d_out, lse, dqkv, scale, which):
    B, S, G, n, D = qkv.shape
    L = _lib.lib()
    words = L.axb_flash_attn_bwd_scratch(B, S, G * (n - 2))
    scratch = torch.empty(words, dtype=torch.float32, device=qkv.device)
    st = L.axb_flash_attn_bwd_split(
        _lib.addr(qkv), _lib.addr(out), _lib.addr(d_out), _lib.addr(lse), _lib.addr(scratch), _lib.addr(dqkv),
        B, S, G, n - 2, D,
        scale, which, qkv.device.index, _lib.stream())
    _lib.check(st, "axb_flash_attn_bwd_split")
    _lib.add_launches(1 if which != 3 else 2)


def flash_bwd_packed(qkv, out, d_out, lse, scale):
    """Gradient of the packed QKV tensor for ``flash_fwd_packed``.

    ``AXONN_FA_BWD`` selects the implementation: ``split`` (default) - the two-kernel backward without atomics
    (``csrc/flash_attn_bwd_split.cu``: one kernel for dQ, one for dK and dV); ``fused`` - the one-kernel form
    (``csrc/flash_attn.cu``) with its fp32 dQ accumulator, for sequence lengths that are multiples of 128;
    ``split_dq`` / ``split_dkv`` take only dQ or only dK, dV from the two-kernel form (A/B runs)."""
    B, S, G, n, D = qkv.shape
    qpk = n - 2
    H = G * qpk
    mode = os.environ.get("AXONN_FA_BWD", _BWD_DEFAULT)
    d_out = d_out if d_out.is_contiguous() else d_out.contiguous()
    if d_out.data_ptr() % 16:
        d_out = d_out.clone()
    dqkv = torch.empty_like(qkv)
    if mode == "split" or S % 128:
        _bwd_split(qkv, out, d_out, lse, dqkv, scale, 3)
        return dqkv
    delta = torch.empty((B, H, S), dtype=torch.float32, device=qkv.device)
    dq_acc = torch.zeros((B, S, H, D), dtype=torch.float32, device=qkv.device)
    st = _lib.lib().axb_flash_attn_bwd(_lib.ptr(qkv), _lib.ptr(out), _lib.ptr(d_out), _lib.ptr(lse), _lib.ptr(delta),
                                       _lib.ptr(dq_acc), _lib.ptr(dqkv), ctypes.c_int(B), ctypes.c_int(S),
                                       ctypes.c_int(G), ctypes.c_int(qpk), ctypes.c_int(D), ctypes.c_float(scale),
                                       ctypes.c_int(qkv.device.index), _lib.stream_ptr())
    _lib.check(st, "axb_flash_attn_bwd")
    _lib.add_launches(1)
    dqkv[:, :, :, :qpk].copy_(dq_acc.view(B, S, G, qpk, D))
    if mode == "split_dq":
        _bwd_split(qkv, out, d_out, lse, dqkv, scale, 1)
    elif mode == "split_dkv":
        _bwd_split(qkv, out, d_out, lse, dqkv, scale, 2)
    return dqkv


class _FlashPacked(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, scale):
        out, lse = flash_fwd_packed(qkv, scale)
        ctx.save_for_backward(qkv, out, lse)
        ctx.scale = scale
        return out

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        qkv, out, lse = ctx.saved_tensors
        return flash_bwd_packed(qkv, out, g, lse, ctx.scale), None


def flash_attention_packed_cuda(qkv, causal, scale):
    assert causal
    host = host_paths()
    if host is not None:
        out = host.attention(qkv, scale)
        if out is not None:
            return out
    if no_graph(qkv):
        return flash_fwd_packed(qkv, scale)[0]
    return _FlashPacked.apply(qkv, scale)
