"""Autograd-aware dense linear algebra on the package's GEMM kernels for layers
that are not tensor parallel (router, expert MLPs)."""

import torch
from torch.autograd.function import once_differentiable

from . import _lib
from .activation import swiglu
from .gemm import as_written, bmm_nn, bmm_nt, bmm_tn, matmul_nn, matmul_nt, matmul_tn


class _LinearFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        x2 = x.reshape(-1, x.shape[-1])
        return matmul_nt(x2, w).reshape(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, g):
        x, w = ctx.saved_tensors
        g2 = g.reshape(-1, g.shape[-1])
        g2 = g2 if g2.is_contiguous() else g2.contiguous()
        x2 = x.reshape(-1, x.shape[-1])
        gx = matmul_nn(g2, w).reshape(x.shape) if ctx.needs_input_grad[0] else None
        gw = matmul_tn(g2, x2, out_dtype=w.dtype) if ctx.needs_input_grad[1] else None
        return gx, gw


def linear(x, w):
    """``x @ w.T`` for ``w`` of shape ``[out, in]``."""
    if x.shape[0] == 0 or x.numel() == 0:
        return x.new_zeros(*x.shape[:-1], w.shape[0]) + 0 * w.sum()
    return _LinearFn.apply(x, w)


class _BatchedLinearFn(torch.autograd.Function):
    """``y[e] = x[e] @ w[e].T`` for all ``e`` with one kernel launch per GEMM of forward and backward."""

    @staticmethod
    def forward(ctx, x, w, seg, seg_rows):
        ctx.save_for_backward(x, w)
        ctx.seg, ctx.seg_rows = seg, seg_rows
        return bmm_nt(x, w, seg=seg, seg_rows=seg_rows)

    @staticmethod
    def backward(ctx, g):
        x, w = ctx.saved_tensors
        g = g if g.is_contiguous() else g.contiguous()
        gx = bmm_nn(g, w, seg=ctx.seg, seg_rows=ctx.seg_rows) if ctx.needs_input_grad[0] else None
        gw = bmm_tn(g, x, out_dtype=w.dtype, seg=ctx.seg, seg_rows=ctx.seg_rows) if ctx.needs_input_grad[1] else None
        return gx, gw, None, None


def linear_batched(x, w, seg=None, seg_rows=0):
    """``x[E, rows, in] @ w[E, out, in].T`` -> ``[E, rows, out]``: the expert GEMMs of a mixture-of-experts layer
    as one launch over the tiles of all experts (instead of one launch per expert).

    ``seg`` (int32 ``[E, rows / seg_rows]``, on the device): the rows of every problem are segments of ``seg_rows``
    rows of which only the first ``seg[e, s]`` hold data and the rest are ZERO (capacity padding).  The kernels
    then skip the tiles without data - the output rows of skipped tiles are zeros, which is what the full product
    would give when the layer has no bias."""
    return _BatchedLinearFn.apply(x, w, seg, seg_rows)


def _swiglu_gemm(backward, a, b, out, saved, seg, seg_rows):
    """``axb_gemm_swiglu`` over the problems of ``a[E, M, K]`` (forward ``b[E, N, K]``, backward ``b[E, K, N]``)."""
    E, M, K = a.shape
    N = b.shape[2] if backward else b.shape[1]
    if seg is not None:
        assert seg.dtype == torch.int32 and seg.is_cuda and seg.is_contiguous() and seg.shape[0] == E
    _lib.check(_lib.lib().axb_gemm_swiglu(1 if backward else 0, _lib.addr(a), _lib.addr(b), _lib.addr(out), _lib.addr(saved), E, M,
                                          N, K, _lib.addr(seg), seg_rows, 0 if seg is None else seg.shape[1], a.device.index,
                                          _lib.stream()), "axb_gemm_swiglu")
    return out


class _SwiGLUExpertsFn(torch.autograd.Function):
    """``swiglu(x @ w1.T) @ w2.T`` per expert with the activation and its adjoint in the epilogues of the GEMMs around them:
    the gated product is written once and read once, the activation's gradient is never stored.  One B200, adjoint in the GEMM /
    after it: 8 experts of 2560 rows, hidden 2048, ffn 8192 483 / 696 us, hidden 512, ffn 2048 82 / 107, from 16 M elements (rows of
    all experts x ffn) on 0.69 - 0.98, below 0.83 - 1.25 (8 of 128 rows, hidden 64, ffn 256 11.4 / 9.1; of 320 rows, hidden 512,
    ffn 2048 22.0 / 19.8), where the layer, forward and backward, is bound by the host's launches: 623 / 648.  A single block
    (ops/mlp.py) the same: 0.82 - 0.99 where ffn fills its tiles, otherwise up to 1.16 below 16 M elements (16384 x 320, hidden 384
    20.6 / 17.7; forward and backward 211 / 222)."""

    @staticmethod
    def forward(ctx, x, w1, w2, seg, seg_rows, keep):
        E, rows, _ = x.shape
        gu = torch.empty((E, rows, w1.shape[1]), dtype=x.dtype, device=x.device) if keep else None
        h = _swiglu_gemm(False, x, w1, torch.empty((E, rows, w2.shape[2]), dtype=x.dtype, device=x.device), gu, seg, seg_rows)
        ctx.save_for_backward(x, w1, w2, gu, h)
        ctx.seg, ctx.seg_rows = seg, seg_rows
        return bmm_nt(h, w2, seg=seg, seg_rows=seg_rows)

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        x, w1, w2, gu, h = ctx.saved_tensors
        seg = dict(seg=ctx.seg, seg_rows=ctx.seg_rows)
        g = as_written(g)
        gx = gw1 = gw2 = None
        if ctx.needs_input_grad[0] or ctx.needs_input_grad[1]:
            gu = as_written(gu, 32)
            dgu = _swiglu_gemm(True, g, as_written(w2), torch.empty_like(gu), gu, **seg)
            gx = bmm_nn(dgu, w1, **seg) if ctx.needs_input_grad[0] else None
            gw1 = bmm_tn(dgu, x, out_dtype=w1.dtype, **seg) if ctx.needs_input_grad[1] else None
        if ctx.needs_input_grad[2]:
            gw2 = bmm_tn(g, h, out_dtype=w2.dtype, **seg)
        return gx, gw1, gw2, None, None, None


def swiglu_experts(x, w1, w2, seg=None, seg_rows=0):
    """``swiglu(x[E, rows, hidden] @ w1[E, 2 * ffn, hidden].T) @ w2[E, hidden, ffn].T``; ``seg`` / ``seg_rows`` as in
    ``linear_batched``."""
    E, rows, hidden = x.shape
    ffn = w2.shape[2]
    ts = (x, w1, w2)
    # the GEMMs of the backward reduce over rows, hidden and 2 * ffn in blocks of 64 that must not reach the next problem
    if (all(t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous() and t.data_ptr() % 16 == 0 for t in ts)
            and x.numel() > 0 and rows % 64 == 0 and hidden % 64 == 0 and ffn % 32 == 0
            and w1.shape == (E, 2 * ffn, hidden) and w2.shape == (E, hidden, ffn)):
        keep = torch.is_grad_enabled() and any(t.requires_grad for t in ts)
        return _SwiGLUExpertsFn.apply(x, w1, w2, seg, seg_rows, keep)
    return linear_batched(swiglu(linear_batched(x, w1, seg, seg_rows)), w2, seg, seg_rows)
