"""Two-layer feed-forward block on one GPU as one autograd function, with the activation's adjoint in the GEMM before it."""

import torch
from torch.autograd.function import once_differentiable

from . import _lib
from .direct import no_graph
from .gemm import EPI_BIAS, EPI_BIAS_GELU, EPI_GELU, EPI_NONE, as_written, gemm_on_pairs, matmul_nn, matmul_nt, matmul_tn
from .linear import _swiglu_gemm
from .norm import column_sum

_OUT = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}


def _dgelu_gemm(g, w2, z, bias_dtype):
    """``(g @ w2) * gelu'(z)`` and its column sums.  One B200, against the product and the pass after it: 16384 x 8192 x 2048 445 / 488
    us, 4096 rows 117 / 126, hidden 4096 and ffn 16384 378 / 414.  Few tiles leave the epilogue in sight (2048 x 2048 x 2048 46.5 / 42.3,
    1300 x 8192 x 2048 53.4 / 52.1); such blocks, forward and backward, are bound by the host's launches, of which it saves one:
    246 / 257 and 303 / 303."""
    rows, ffn = z.shape
    L = _lib.lib()
    dz = torch.empty_like(z)
    part = torch.empty(((rows + 31) // 32, ffn), dtype=torch.float32, device=z.device)
    _lib.check(L.axb_gemm_dgelu(_lib.addr(g), _lib.addr(w2), _lib.addr(dz), _lib.addr(z), _lib.addr(part), rows, ffn, g.shape[1],
                                z.device.index, _lib.stream()), "axb_gemm_dgelu")
    if bias_dtype is None:
        return dz, None
    db = torch.empty(ffn, dtype=bias_dtype, device=z.device)
    _lib.check(L.axb_fold_columns(_lib.addr(part), _lib.addr(db), part.shape[0], ffn, _OUT[bias_dtype], _lib.stream()),
               "axb_fold_columns")
    return dz, db


class _MLPFn(torch.autograd.Function):
    """``act(x @ w1.T + b1) @ w2.T + b2`` with ``act`` GELU (tanh form) or SwiGLU (no bias in front of it)."""

    @staticmethod
    def forward(ctx, x, w1, b1, w2, b2, hidden, act):
        x2 = x.reshape(-1, hidden)
        v1, v2 = w1.view(-1, hidden), w2.view(hidden, -1)
        z = torch.empty((x2.shape[0], v1.shape[0]), dtype=x.dtype, device=x.device)
        if act == "swiglu":
            h = torch.empty((x2.shape[0], v2.shape[1]), dtype=x.dtype, device=x.device)
            _swiglu_gemm(False, x2[None], v1[None], h, z, None, 0)
        else:
            h = matmul_nt(x2, v1, bias=b1, epilogue=EPI_GELU if b1 is None else EPI_BIAS_GELU, aux=z)
        # a view made in here could not be modified in place later: the result has its shape from the beginning
        y = torch.empty((*x.shape[:-1], hidden), dtype=x.dtype, device=x.device)
        matmul_nt(h, v2, bias=b2, epilogue=EPI_NONE if b2 is None else EPI_BIAS, out=y.view(-1, hidden))
        ctx.save_for_backward(x, w1, w2, z, h)
        ctx.hidden, ctx.act, ctx.b1, ctx.b2 = hidden, act, None if b1 is None else b1.dtype, None if b2 is None else b2.dtype
        return y

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        x, w1, w2, z, h = ctx.saved_tensors
        need = ctx.needs_input_grad
        g2 = as_written(g.reshape(-1, ctx.hidden))
        z = as_written(z, 32)
        v1, v2 = w1.reshape(-1, ctx.hidden), as_written(w2).view(ctx.hidden, -1)
        gx = gw1 = gb1 = gw2 = gb2 = None
        if need[3]:
            gw2 = matmul_tn(g2, h).view(w2.shape)
        if ctx.b2 is not None and need[4]:
            gb2 = column_sum(g2, out_dtype=ctx.b2)
        if need[0] or need[1] or need[2]:
            if ctx.act == "swiglu":
                dz = _swiglu_gemm(True, g2[None], v2[None], torch.empty_like(z), z, None, 0)
            else:
                dz, gb1 = _dgelu_gemm(g2, v2, z, ctx.b1 if ctx.b1 is not None and need[2] else None)
            if need[1]:
                gw1 = matmul_tn(dz, x.reshape(-1, ctx.hidden)).view(w1.shape)
            if need[0]:
                gx = matmul_nn(dz, v1).reshape(x.shape)
        return gx, gw1, gb1, gw2, gb2, None, None


def mlp_takes(rows, hidden, ffn, act, device):
    """Are the sizes ones for which ``mlp`` has its kernels?  (Few elements are turned away without asking the library.)"""
    # GELU: below this the gradient GEMM's main loop is shorter than the epilogue's arithmetic.  One B200, ffn 4 * hidden, with the
    # adjoint in the GEMM / after it, 4096 and 16384 rows: hidden 1024 53.3 / 46.1 and 175 / 162 us, 1280 68.3 / 61.8 and 227 / 226,
    # 1536 82.9 / 81.6 and 290 / 300, 1792 100 / 103 and 365 / 385, 2048 117 / 126 and 445 / 488
    if act == "gelu" and hidden < 2048:
        return False
    return rows * ffn >= 1 << 20 and gemm_on_pairs(rows, ffn, device) and (act == "gelu" or gemm_on_pairs(rows, 2 * ffn, device))


def mlp(x, w1, b1, w2, b2, hidden, ffn, act):
    """The block for a training step (``w1`` holds ``[ffn, hidden]``, ``[2 * ffn, hidden]`` with SwiGLU; ``w2`` ``[hidden, ffn]``;
    flat tensors are fine), or ``None`` where its kernels do not apply: other types, few rows, no gradient needed."""
    wide = 2 * ffn if act == "swiglu" else ffn
    ts = [t for t in (x, w1, b1, w2, b2) if t is not None]
    if (act not in ("gelu", "swiglu") or (act == "swiglu" and b1 is not None) or not torch.is_grad_enabled()
            or not any(t.requires_grad for t in ts)
            or not all(t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous() and t.data_ptr() % 16 == 0 for t in ts)
            or x.dim() == 0 or x.shape[-1] != hidden or x.numel() == 0 or hidden % 64 or ffn % 16
            or w1.numel() != wide * hidden or w2.numel() != ffn * hidden):
        return None
    if not mlp_takes(x.numel() // hidden, hidden, ffn, act, x.device.index):
        return None
    return _MLPFn.apply(x, w1, b1, w2, b2, hidden, act)


def swiglu_projection(x, w1, hidden):
    """``swiglu(x[..., hidden] @ w1.T)`` without gradients as one launch that never stores the gated product (``w1`` holds
    ``[2 * ffn, hidden]``), or ``None`` where the kernel does not apply.  One B200, two-layer block without gradients, three launches /
    two: 4096 rows, 4096 -> 14336 -> 4096 1099 / 1038 us, 1000 rows 316 / 290, 2000, 2048 -> 8192 188 / 164, 777, 1024 -> 4096
    53 / 45."""
    if not (no_graph(x, w1) and x.dtype == w1.dtype == torch.bfloat16 and x.is_contiguous() and w1.is_contiguous() and x.dim() > 0
            and x.shape[-1] == hidden and x.numel() > 0 and w1.numel() % (16 * hidden) == 0 and hidden % 8 == 0
            and x.data_ptr() % 16 == 0 and w1.data_ptr() % 16 == 0):
        return None
    rows, wide = x.numel() // hidden, w1.numel() // hidden
    if not gemm_on_pairs(rows, wide, x.device.index):
        return None
    h = x.new_empty(x.shape[:-1] + (wide // 2,))
    return _swiglu_gemm(False, x.view(1, rows, hidden), w1.view(1, wide, hidden), h, None, None, 0)
