"""LayerNorm and RMSNorm (forward + backward kernels in ``csrc/norm.cu``).

Both accept a hidden dimension that is sharded over a process group
(``group``): the per-row statistics are then partial sums that are all-reduced
between a "statistics" launch and an "apply" launch, in forward and backward.
They stand in for the apex fused LayerNorm and the HF RMSNorm that the
reference's models rely on (``external/models/nvidia_transformer.py:57-95``,
``axonn/models/transformers/modify_llama.py``).
"""

import torch
import torch.distributed as dist

from . import _lib
from .direct import first_derivative_only, host_paths, no_graph

_DT = {torch.bfloat16: 0, torch.float16: 1, torch.float32: 2}


def _group_size(group):
    return 1 if group is None else (group.size() if isinstance(group, dist.ProcessGroup) else dist.get_world_size(group))


def _dense_rows(t, H):
    """``t`` itself when it is dense (the kernels see rows of ``H``) and on 16 bytes, otherwise a copy of its rows that is."""
    return _on_16_bytes(t if t.is_contiguous() else t.reshape(-1, H).contiguous())


def _on_16_bytes(t):
    """``t`` where the kernels can read 16 bytes at a time: a view into a buffer at another offset is copied."""
    return t.clone() if t is not None and t.is_cuda and t.data_ptr() % 16 else t


def _shaped(t, shape):
    return t if t.shape == shape else t.reshape(shape)


def _torch_norm_fwd(x, gamma, beta, eps, rms, group):
    xf = x.float()
    n = _group_size(group)
    H_total = x.shape[-1] * n
    s2 = xf.pow(2).sum(-1, keepdim=True)
    s1 = torch.zeros_like(s2) if rms else xf.sum(-1, keepdim=True)
    if n > 1:
        st = torch.cat([s1, s2], -1)
        dist.all_reduce(st, group=group)
        s1, s2 = st[..., :1], st[..., 1:]
    mean = s1 / H_total
    var = s2 / H_total - (0 if rms else mean * mean)
    rstd = torch.rsqrt(var.clamp_min(0) + eps)
    y = (xf - mean) * rstd * gamma.float()
    if beta is not None:
        y = y + beta.float()
    return y.to(x.dtype), mean, rstd


class _NormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gamma, beta, eps, rms, group):
        shape = x.shape
        H = shape[-1]
        n = _group_size(group)
        ctx.rms, ctx.group, ctx.n, ctx.shape, ctx.has_beta = rms, group, n, shape, beta is not None
        if not x.is_cuda:
            x2 = x.reshape(-1, H).contiguous()
            y, mean, rstd = _torch_norm_fwd(x2, gamma, beta, eps, rms, group)
            ctx.save_for_backward(x, gamma, mean, rstd)
            return y.reshape(shape)
        x2 = _dense_rows(x, H)
        rows = x2.numel() // H
        L = _lib.lib()
        dev = x2.device.index
        y = torch.empty_like(x2)
        stats = torch.empty((rows, 2), dtype=torch.float32, device=x2.device)
        g = _on_16_bytes(gamma.to(x2.dtype) if gamma.dtype != x2.dtype else gamma)
        b = None if beta is None else _on_16_bytes(beta.to(x2.dtype) if beta.dtype != x2.dtype else beta)

        def call(mode):
            st = L.axb_norm_fwd(_lib.addr(x2), _lib.addr(g), _lib.addr(b), _lib.addr(y), _lib.addr(stats),
                                rows, H, H * n, eps,
                                1 if rms else 0, mode, _DT[x2.dtype],
                                dev, _lib.stream())
            _lib.check(st, "axb_norm_fwd")

        if n == 1:
            call(0)
        else:
            call(1)                              # partial (sum x, sum x^2) of my slice of the hidden dimension
            dist.all_reduce(stats, group=group)
            call(3)                              # finishes (mean, rstd) in place and applies them
        ctx.save_for_backward(x2, g, stats, *(i for i, t in ((x, x2), (gamma, g)) if i is not t))
        return _shaped(y, shape)

    @staticmethod
    @first_derivative_only
    def backward(ctx, dy):
        rms, group, n = ctx.rms, ctx.group, ctx.n
        H = ctx.shape[-1]
        if not dy.is_cuda:
            dy2 = dy.reshape(-1, H).contiguous()
            x, gamma, mean, rstd = ctx.saved_tensors
            xh = (x.reshape(-1, H).float() - mean) * rstd
            gd = dy2.float() * gamma.float()
            s1 = torch.zeros_like(mean) if rms else gd.sum(-1, keepdim=True)
            s2 = (gd * xh).sum(-1, keepdim=True)
            if n > 1:
                st = torch.cat([s1, s2], -1)
                dist.all_reduce(st, group=group)
                s1, s2 = st[..., :1], st[..., 1:]
            Ht = H * n
            dx = rstd * (gd - s1 / Ht - xh * s2 / Ht)
            dgamma = (dy2.float() * xh).sum(0).to(gamma.dtype)
            dbeta = dy2.float().sum(0).to(gamma.dtype) if ctx.has_beta else None
            return dx.to(dy.dtype).reshape(ctx.shape), dgamma, dbeta, None, None, None
        x2, g, stats = ctx.saved_tensors[:3]
        dy2 = _dense_rows(dy, H)
        rows = stats.shape[0]
        L = _lib.lib()
        dev = x2.device.index
        grid = L.axb_norm_grid(dev, rows)
        dx = torch.empty_like(x2)
        sums = torch.empty((rows, 2), dtype=torch.float32, device=x2.device) if n > 1 else None
        part = torch.empty((2, grid, H), dtype=torch.float32, device=x2.device)
        pa = part.data_ptr()
        # written in the parameter's dtype: no cast kernel
        dg, db = torch.empty_like(g), (None if rms else torch.empty_like(g))

        def call(mode):
            st = L.axb_norm_bwd(_lib.addr(dy2), _lib.addr(x2), _lib.addr(g), _lib.addr(stats), _lib.addr(dx),
                                _lib.addr(sums), pa, pa + grid * H * 4, _lib.addr(dg), _lib.addr(db), rows, H, H * n,
                                1 if rms else 0, mode, _DT[x2.dtype],
                                _DT[g.dtype], dev, _lib.stream())
            _lib.check(st, "axb_norm_bwd")
            if mode != 1:
                _lib.add_launches(1)

        if n == 1:
            call(0)
        else:
            call(1)
            dist.all_reduce(sums, group=group)
            call(2)
        return _shaped(dx, ctx.shape), dg, (db if ctx.has_beta else None), None, None, None


class _AddNormFn(torch.autograd.Function):
    """``h = x + delta``; ``y = norm(h)``; returns ``(h, y)``.  On CUDA the add is done inside the norm kernel
    (one read of ``x`` and ``delta``, one write of ``h`` and ``y``) and the backward adds the gradient of the
    residual path to the norm's input gradient inside the backward kernel; elsewhere it is the two plain steps."""

    @staticmethod
    def forward(ctx, x, delta, gamma, beta, eps, rms, group):
        shape = x.shape
        H = shape[-1]
        n = _group_size(group)
        ctx.rms, ctx.group, ctx.n, ctx.shape, ctx.has_beta = rms, group, n, shape, beta is not None
        if not x.is_cuda:
            x2 = x.reshape(-1, H).contiguous()
            d2 = delta.reshape(-1, H).contiguous()
            h = (x2 + d2).reshape(shape)
            y, mean, rstd = _torch_norm_fwd(h.reshape(-1, H), gamma, beta, eps, rms, group)
            ctx.save_for_backward(h, gamma, mean, rstd)
            return h, y.reshape(shape)
        x2, d2 = _dense_rows(x, H), _dense_rows(delta, H)
        rows = x2.numel() // H
        L = _lib.lib()
        dev = x2.device.index
        h, y = (torch.empty(shape, dtype=x2.dtype, device=x2.device) for _ in range(2))
        stats = torch.empty((rows, 2), dtype=torch.float32, device=x2.device)
        g = _on_16_bytes(gamma.to(x2.dtype) if gamma.dtype != x2.dtype else gamma)
        b = None if beta is None else _on_16_bytes(beta.to(x2.dtype) if beta.dtype != x2.dtype else beta)

        def call(mode, src, dl):
            st = L.axb_add_norm_fwd(_lib.addr(src), _lib.addr(dl), _lib.addr(h if dl is not None else None), _lib.addr(g),
                                    _lib.addr(b), _lib.addr(y), _lib.addr(stats), rows, H,
                                    H * n, eps, 1 if rms else 0,
                                    mode, _DT[x2.dtype], dev, _lib.stream())
            _lib.check(st, "axb_add_norm_fwd")

        if n == 1:
            call(0, x2, d2)
        else:
            call(1, x2, d2)                      # writes h and the partial row sums
            dist.all_reduce(stats, group=group)
            call(3, h, None)                     # finishes (mean, rstd) in place and applies them
        ctx.save_for_backward(h, g, stats, *(() if g is gamma else (gamma,)))
        return h, y

    @staticmethod
    @first_derivative_only
    def backward(ctx, dh, dy):
        rms, group, n = ctx.rms, ctx.group, ctx.n
        H = ctx.shape[-1]
        if not dy.is_cuda:
            dy2 = dy.reshape(-1, H).contiguous()
            dh2 = None if dh is None else dh.reshape(-1, H).contiguous()
            h, gamma, mean, rstd = ctx.saved_tensors
            xh = (h.reshape(-1, H).float() - mean) * rstd
            gd = dy2.float() * gamma.float()
            s1 = torch.zeros_like(mean) if rms else gd.sum(-1, keepdim=True)
            s2 = (gd * xh).sum(-1, keepdim=True)
            if n > 1:
                st = torch.cat([s1, s2], -1)
                dist.all_reduce(st, group=group)
                s1, s2 = st[..., :1], st[..., 1:]
            Ht = H * n
            dx = rstd * (gd - s1 / Ht - xh * s2 / Ht)
            if dh2 is not None:
                dx = dx + dh2.float()
            dgamma = (dy2.float() * xh).sum(0).to(gamma.dtype)
            dbeta = dy2.float().sum(0).to(gamma.dtype) if ctx.has_beta else None
            dx = dx.to(dy.dtype).reshape(ctx.shape)
            return dx, dx, dgamma, dbeta, None, None, None
        x2, g, stats = ctx.saved_tensors[:3]
        dy2 = _dense_rows(dy, H)
        dh2 = None if dh is None else _dense_rows(dh, H)
        rows = stats.shape[0]
        L = _lib.lib()
        dev = x2.device.index
        grid = L.axb_norm_grid(dev, rows)
        dx = torch.empty_like(x2)
        sums = torch.empty((rows, 2), dtype=torch.float32, device=x2.device) if n > 1 else None
        part = torch.empty((2, grid, H), dtype=torch.float32, device=x2.device)
        pa = part.data_ptr()
        dg, db = torch.empty_like(g), (None if rms else torch.empty_like(g))

        def call(mode):
            st = L.axb_add_norm_bwd(_lib.addr(dy2), _lib.addr(dh2), _lib.addr(x2), _lib.addr(g), _lib.addr(stats), _lib.addr(dx),
                                    _lib.addr(sums), pa, pa + grid * H * 4, _lib.addr(dg), _lib.addr(db), rows, H, H * n,
                                    1 if rms else 0, mode, _DT[x2.dtype],
                                    _DT[g.dtype], dev, _lib.stream())
            _lib.check(st, "axb_add_norm_bwd")
            if mode != 1:
                _lib.add_launches(1)

        if n == 1:
            call(0)
        else:
            call(1)
            dist.all_reduce(sums, group=group)
            call(2)
        dx = _shaped(dx, ctx.shape)
        return dx, dx, dg, (db if ctx.has_beta else None), None, None, None


def _norm_direct(x, delta, gamma, beta, eps, rms, group):
    """``(h, norm(h))`` with ``h = x + delta`` (``delta`` None: ``h = x``) as one launch, when neither a gradient nor a
    reduction over ``group`` is needed; ``None`` when the general path has to run."""
    H = x.shape[-1] if x.dim() else 0
    if (not no_graph(x, delta, gamma, beta) or x.dtype not in _DT or gamma.dtype != x.dtype or gamma.shape != (H,)
            or (beta is not None and (beta.dtype != x.dtype or beta.shape != (H,) or not beta.is_contiguous()))
            or x.numel() == 0 or _group_size(group) != 1 or not x.is_contiguous() or not gamma.is_contiguous()
            or (delta is not None and (delta.shape != x.shape or delta.dtype != x.dtype or not delta.is_contiguous()))
            or any(t is not None and t.data_ptr() % 16 for t in (x, delta, gamma, beta))):
        return None
    rows = x.numel() // H
    y = torch.empty_like(x)
    stats = torch.empty((rows, 2), dtype=torch.float32, device=x.device)
    if delta is None:
        _lib.check(_lib.lib().axb_norm_fwd(x.data_ptr(), gamma.data_ptr(), _lib.addr(beta), y.data_ptr(), stats.data_ptr(), rows,
                                           H, H, eps, 1 if rms else 0, 0, _DT[x.dtype], x.device.index, _lib.stream()),
                   "axb_norm_fwd")
        return x, y
    h = torch.empty_like(x)
    _lib.check(_lib.lib().axb_add_norm_fwd(x.data_ptr(), delta.data_ptr(), h.data_ptr(), gamma.data_ptr(), _lib.addr(beta),
                                           y.data_ptr(), stats.data_ptr(), rows, H, H, eps, 1 if rms else 0, 0, _DT[x.dtype],
                                           x.device.index, _lib.stream()), "axb_add_norm_fwd")
    return h, y


def _norm(x, delta, gamma, beta, eps, rms, group):
    """``norm(x)``, or ``(h, norm(h))`` of ``h = x + delta``.  On one rank the questions, the launches and the autograd node are native
    (one B200, host-bound, forward and backward of 16 rows: RMSNorm 111 -> 74 us, LayerNorm with the residual 131 -> 91)."""
    host = host_paths() if x.is_cuda and _group_size(group) == 1 else None
    if host is not None:
        out = host.norm(x, delta, gamma, beta, eps, rms)
        if out is not None:
            return out
    direct = _norm_direct(x, delta, gamma, beta, eps, rms, group)
    if delta is not None:
        return direct or _AddNormFn.apply(x, delta, gamma, beta, eps, rms, group)
    # made dense outside of the function: what it saves is its input then
    return _NormFn.apply(x.contiguous(), gamma, beta, eps, rms, group) if direct is None else direct[1]


def add_layer_norm(x, delta, gamma, beta, eps=1e-5, group=None):
    """``h = x + delta; y = LayerNorm(h)`` in one kernel; returns ``(h, y)``."""
    return _norm(x, delta, gamma, beta, eps, False, group)


def add_rms_norm(x, delta, gamma, eps=1e-6, group=None):
    """``h = x + delta; y = RMSNorm(h)`` in one kernel; returns ``(h, y)``."""
    return _norm(x, delta, gamma, None, eps, True, group)


def layer_norm(x, gamma, beta, eps=1e-5, group=None):
    """LayerNorm over the last dimension; with ``group`` the last dimension is one
    shard of a hidden dimension split over that process group."""
    return _norm(x, None, gamma, beta, eps, False, group)


def rms_norm(x, gamma, eps=1e-6, group=None):
    """RMSNorm over the last dimension; with ``group`` the last dimension is one shard of a hidden dimension
    split over that process group."""
    return _norm(x, None, gamma, None, eps, True, group)


def column_sum(x, out_dtype=torch.float32):
    """``x.sum(0)`` of a 2-D tensor, accumulated in fp32 and returned as ``out_dtype`` (bias gradients).  One
    pass over ``x`` at memory bandwidth on CUDA (partial sums per row split, then a fold that writes the
    requested dtype); plain PyTorch elsewhere."""
    if not (_lib.use_cuda_kernels(x) and x.dim() == 2 and x.shape[1] % 8 == 0 and x.is_contiguous() and x.data_ptr() % 16 == 0
            and x.dtype in (torch.bfloat16, torch.float16, torch.float32) and x.shape[0] > 0
            and out_dtype in _DT):
        return x.sum(0, dtype=torch.float32).to(out_dtype)
    rows, n = x.shape
    L = _lib.lib()
    dev = x.device.index
    splits = L.axb_colsum_splits(dev, rows, n)
    part = torch.empty((splits, n), dtype=torch.float32, device=x.device)
    out = torch.empty(n, dtype=out_dtype, device=x.device)
    _lib.check(L.axb_colsum(_lib.addr(x), _lib.addr(part), _lib.addr(out), rows, n,
                            _DT[x.dtype], _DT[out_dtype], dev,
                            _lib.stream()), "axb_colsum")
    _lib.add_launches(1)
    return out
