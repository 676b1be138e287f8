"""Softmax cross-entropy on (optionally vocabulary-parallel) logits.

The GPU path reads the bf16 logits once for the row statistics and rewrites
them in place with the gradient in backward, so no fp32 copy of the
``[tokens, vocab]`` matrix is ever materialised (``csrc/loss.cu``).
"""

import ctypes

import torch
import torch.distributed as dist
from torch.autograd.function import once_differentiable

from . import _lib
from .gemm import as_written, matmul_nn, matmul_nt, matmul_tn


class _CrossEntropyFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, targets, group, ignore_index):
        V = logits.shape[-1]
        z = logits.reshape(-1, V)
        t = targets.reshape(-1).contiguous()
        rows = z.shape[0]
        n = 1 if group is None else dist.get_world_size(group)
        start = 0 if n == 1 else dist.get_rank(group) * V
        if z.is_cuda:
            if z.dtype != torch.bfloat16:
                raise TypeError("cross-entropy kernel needs bf16 logits")
            z = z.contiguous()
            stats = torch.empty((rows, 3), dtype=torch.float32, device=z.device)
            if n == 1 and rows > 0:
                lse = torch.empty(rows, dtype=torch.float32, device=z.device)
                # two tensors: the loss is returned, and a view made in here could not be modified in place later
                mean, kept = (torch.empty((), dtype=torch.float32, device=z.device) for _ in range(2))
                _lib.check(_lib.lib().axb_ce_fwd_mean(_lib.addr(z), _lib.addr(t), _lib.addr(stats), _lib.addr(lse),
                                                      _lib.addr(mean), _lib.addr(kept), rows, V,
                                                      ignore_index, _lib.stream()),
                           "axb_ce_fwd_mean")
                _lib.add_launches(1)
                ctx.save_for_backward(z, t, lse, kept)
                ctx.start, ctx.ignore_index, ctx.shape = start, ignore_index, logits.shape
                return mean
            _lib.check(_lib.lib().axb_ce_fwd(_lib.ptr(z), _lib.ptr(t), _lib.ptr(stats), ctypes.c_int(rows),
                                             ctypes.c_int(V), ctypes.c_int(start), _lib.stream_ptr()), "axb_ce_fwd")
            m, s, tl = stats[:, 0], stats[:, 1], stats[:, 2]
        else:
            zf = z.float()
            m = zf.max(-1).values
            s = (zf - m[:, None]).exp().sum(-1)
            loc = t - start
            inside = (loc >= 0) & (loc < V)
            tl = torch.where(inside, zf.gather(1, loc.clamp(0, V - 1)[:, None])[:, 0], torch.zeros_like(m))
        if n > 1:
            gm = m.clone()
            dist.all_reduce(gm, op=dist.ReduceOp.MAX, group=group)
            st = torch.stack([s * (m - gm).exp(), tl])
            dist.all_reduce(st, group=group)
            s, tl, m = st[0], st[1], gm
        lse = m + s.log()
        valid = t != ignore_index
        count = valid.sum().clamp_min(1).float()
        loss = ((lse - tl) * valid).sum() / count
        ctx.save_for_backward(z, t, lse.contiguous(), count)
        ctx.start, ctx.ignore_index, ctx.shape = start, ignore_index, logits.shape
        return loss

    @staticmethod
    def backward(ctx, g):
        z, t, lse, count = ctx.saved_tensors
        V = z.shape[-1]
        scale = (g.float() / count).reshape(1).contiguous()
        if z.is_cuda:
            _lib.check(_lib.lib().axb_ce_bwd(_lib.addr(z), _lib.addr(t), _lib.addr(lse), _lib.addr(scale),
                                             z.shape[0], V, ctx.start,
                                             ctx.ignore_index, _lib.stream()), "axb_ce_bwd")
            torch.autograd.graph.increment_version(z)      # written through its address: a second backward has to notice
            return z.reshape(ctx.shape), None, None, None
        p = (z.float() - lse[:, None]).exp()
        loc = t - ctx.start
        inside = (loc >= 0) & (loc < V)
        onehot = torch.zeros_like(p)
        onehot[inside, loc[inside]] = 1.0
        valid = (t != ctx.ignore_index).float()[:, None]
        return ((p - onehot) * valid * scale).to(z.dtype).reshape(ctx.shape), None, None, None


def cross_entropy(logits, targets, group=None, ignore_index=-100):
    """Mean token cross-entropy.  With ``group`` the last dimension of ``logits``
    is this rank's contiguous slice of the vocabulary (rank order = slice order).
    On GPU the logits buffer is consumed: backward overwrites it with the gradient, and a second backward raises an error."""
    return _CrossEntropyFn.apply(logits, targets, group, ignore_index)


def _statistics_in_epilogue(rows, V, H, device):
    return bool(_lib.lib().axb_gemm_ce_pays(rows, V, H, device))


class _ProjectedCrossEntropyFn(torch.autograd.Function):
    """``cross_entropy(x @ w.T, targets)``; the softmax statistics come from the epilogue of the projection where that is faster,
    so that the logits are written once, read and overwritten by their gradient once, and read by the two GEMMs of the backward."""

    @staticmethod
    def forward(ctx, x, weight, targets, shape, ignore_index):
        V, H = shape
        x2 = x.reshape(-1, H)
        t = targets.reshape(-1).contiguous()
        rows = x2.shape[0]
        dev = x.device
        L = _lib.lib()
        stats = torch.empty((rows, 3), dtype=torch.float32, device=dev)
        lse = torch.empty(rows, dtype=torch.float32, device=dev)
        # two tensors: the loss is returned, and a view made in here could not be modified in place later
        mean, kept = (torch.empty((), dtype=torch.float32, device=dev) for _ in range(2))
        if _statistics_in_epilogue(rows, V, H, dev.index):
            z = torch.empty((rows, V), dtype=x.dtype, device=dev)
            part = torch.empty(((V + 255) // 256, rows, 2), dtype=torch.float32, device=dev)
            _lib.check(L.axb_gemm_ce(_lib.addr(x2), _lib.addr(weight), _lib.addr(z), _lib.addr(part), rows, V, H, dev.index,
                                     _lib.stream()), "axb_gemm_ce")
            _lib.check(L.axb_ce_fwd_parts(_lib.addr(part), _lib.addr(z), _lib.addr(t), _lib.addr(stats), _lib.addr(lse),
                                          _lib.addr(mean), _lib.addr(kept), rows, V, ignore_index, _lib.stream()),
                       "axb_ce_fwd_parts")
        else:
            z = matmul_nt(x2, weight.view(V, H))
            _lib.check(L.axb_ce_fwd_mean(_lib.addr(z), _lib.addr(t), _lib.addr(stats), _lib.addr(lse), _lib.addr(mean),
                                         _lib.addr(kept), rows, V, ignore_index, _lib.stream()), "axb_ce_fwd_mean")
        _lib.add_launches(1)
        ctx.save_for_backward(x, weight, z, t, lse, kept)
        ctx.shape, ctx.ignore_index = shape, ignore_index
        return mean

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        x, weight, z, t, lse, kept = ctx.saved_tensors
        z, t, lse = as_written(z), t.contiguous(), lse.contiguous()
        V, H = ctx.shape
        scale = (g.float() / kept).reshape(1).contiguous()
        _lib.check(_lib.lib().axb_ce_bwd(_lib.addr(z), _lib.addr(t), _lib.addr(lse), _lib.addr(scale), z.shape[0], V, 0,
                                         ctx.ignore_index, _lib.stream()), "axb_ce_bwd")
        torch.autograd.graph.increment_version(z)
        gx = matmul_nn(z, weight.reshape(V, H)).view(x.shape) if ctx.needs_input_grad[0] else None
        gw = matmul_tn(z, x.reshape(-1, H)).view(weight.shape) if ctx.needs_input_grad[1] else None
        return gx, gw, None, None, None


def projected_cross_entropy(x, weight, targets, shape, ignore_index=-100):
    """Mean cross-entropy of the logits ``x[..., H] @ weight.T`` with ``weight`` holding ``shape = (V, H)``; ``None`` when the
    projection is not one of those whose kernel has the statistics in its epilogue (few rows, other types).  As in
    ``cross_entropy``, the backward overwrites the logits with their gradient, and a second one raises an error."""
    V, H = shape
    if (x.is_cuda and weight.is_cuda and targets.is_cuda and x.dtype == weight.dtype == torch.bfloat16 and V % 8 == 0 and H % 8 == 0
            and x.dim() > 0 and x.shape[-1] == H and weight.numel() == V * H and x.numel() > 0 and targets.dtype == torch.int64
            and targets.numel() * H == x.numel() and x.is_contiguous() and weight.is_contiguous() and x.data_ptr() % 16 == 0
            and weight.data_ptr() % 16 == 0 and _lib.lib().axb_gemm_on_pairs(x.numel() // H, V, x.device.index)):
        return _ProjectedCrossEntropyFn.apply(x, weight, targets, shape, ignore_index)
    return None
