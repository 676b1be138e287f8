"""GEMM epilogues at the edges of their rules: alignment of the output, remainders of tiles, masked rows."""

import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16 = torch.bfloat16


def _rel(got, want):
    return float((got.detach().double() - want.detach().double()).norm() / want.detach().double().norm().clamp_min(1e-30))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(1, 16, 64), (77, 264, 128), (130, 1048, 72), (1031, 2064, 256), (2500, 4104, 192),
                                   (2500, 4112, 192), (2049, 4096, 64)])
@pytest.mark.parametrize("shift", [0, 8])
def test_gemm_store_alignment(M, N, K, shift, dtype):
    """Outputs whose rows start on a 32-byte boundary and ones that do not (N = 8 mod 16, or a base 16 bytes off), the
    last chunk of 32 columns cut at 8, 16 and 24.  Tolerance: one rounding of the result (2^-9 / 2^-11) after fp32 sums;
    the saved pre-activation has the same, and nothing outside the output is written."""
    from axonn_b200 import ops

    torch.manual_seed(M + N)
    a, b = torch.randn(M, K, device=DEV).to(dtype), torch.randn(N, K, device=DEV).to(dtype)
    bias = torch.randn(N, device=DEV).to(dtype)
    bufs = [torch.full((M * N + 64,), 7.0, device=DEV, dtype=dtype) for _ in range(2)]
    out, aux = (t[shift:shift + M * N].view(M, N) for t in bufs)
    ops.matmul_nt(a, b, bias=bias, epilogue=ops.EPI_BIAS_GELU, out=out, aux=aux)
    z = a.double() @ b.double().t() + bias.double()
    tol = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10}[dtype]
    assert _rel(aux, z) < tol
    assert _rel(out, torch.nn.functional.gelu(z, approximate="tanh")) < tol
    for t in bufs:
        assert bool((t[:shift] == 7).all()) and bool((t[shift + M * N:] == 7).all())


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K", [(776, 6144, 512), (1032, 4616, 136), (1000, 5656, 1992), (1024, 4872, 264), (3000, 1560, 72)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_halved_tiles(layout, M, N, K, dtype):
    """A last wave of a few tiles, which are computed as halves of their columns: N that ends inside the first half, the
    second one, and on the seam; a ragged M and K; every epilogue.  Tolerance: one rounding of the result (2^-9 / 2^-11)."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib

    torch.manual_seed(M)
    a, b = torch.randn(M, K, device=DEV).to(dtype), torch.randn(N, K, device=DEV).to(dtype)
    z = a.double() @ b.double().t()
    tol = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10}[dtype]
    fn, x, y = {"nt": (ops.matmul_nt, a, b), "nn": (ops.matmul_nn, a, b.t().contiguous()),
                "tn": (ops.matmul_tn, a.t().contiguous(), b.t().contiguous())}[layout]
    got = fn(x, y)
    assert _lib.device_status() == 0
    for r in range(0, M, 128):                       # a wrong tile must not hide in the norm of the whole
        for c in range(0, N, 128):
            assert _rel(got[r:r + 128, c:c + 128], z[r:r + 128, c:c + 128]) < tol, (r, c)
    acc = torch.randn(M, N, device=DEV, dtype=torch.float32)
    want = acc.double() + z
    assert _rel(fn(x, y, out=acc, accumulate=True), want) < 1e-5
    if layout == "nt":
        bias = torch.randn(N, device=DEV).to(dtype)
        aux = torch.empty(M, N, device=DEV, dtype=dtype)
        out = ops.matmul_nt(x, y, bias=bias, epilogue=ops.EPI_BIAS_GELU, aux=aux)
        assert _rel(aux, z + bias.double()) < tol
        assert _rel(out, torch.nn.functional.gelu(z + bias.double(), approximate="tanh")) < tol


@pytest.mark.parametrize("E,rows,hidden,ffn,counts", [(1, 64, 64, 32, None), (3, 192, 128, 96, [[0], [64], [191]]), (2, 640, 192, 160, [[1], [500]]),
                                                      (2, 512, 256, 288, [[70, 0], [256, 3]]), (8, 2560, 512, 1024, None)])
def test_swiglu_experts(E, rows, hidden, ffn, counts):
    """Gated feed-forward layers with the activation in the GEMMs: tiles with and without data rows, N that ends inside a
    chunk, one segment and two, against the layer in 64 bits.  Memory that no kernel writes holds NaN, so that reading a
    row without data would show.  Tolerance: the stored product, the activation and its gradient are rounded to bf16 (three
    roundings of 2^-9 forward, five backward)."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib

    torch.manual_seed(rows)
    x = torch.randn(E, rows, hidden, device=DEV).bfloat16()
    w1 = (torch.randn(E, 2 * ffn, hidden, device=DEV) * hidden ** -0.5).bfloat16().requires_grad_(True)
    w2 = (torch.randn(E, hidden, ffn, device=DEV) * ffn ** -0.5).bfloat16().requires_grad_(True)
    dy = torch.randn(E, rows, hidden, device=DEV).bfloat16()
    seg, seg_rows = None, 0
    if counts is not None:
        seg, seg_rows = torch.tensor(counts, dtype=torch.int32, device=DEV), rows // len(counts[0])
        live = (torch.arange(seg_rows, device=DEV)[None, None] < seg[:, :, None]).view(E, rows, 1)
        x, dy = x * live, dy * live
    x.requires_grad_(True)
    poison = [torch.full((n * E * rows,), float("nan"), device=DEV, dtype=BF16) for n in (ffn, 2 * ffn, ffn, 2 * ffn, hidden)]
    del poison
    y = ops.swiglu_experts(x, w1, w2, seg, seg_rows)
    poison = [torch.full((n * E * rows,), float("nan"), device=DEV, dtype=BF16) for n in (ffn, 2 * ffn, ffn, 2 * ffn, hidden)]
    del poison
    got = torch.autograd.grad(y, [x, w1, w2], dy)
    with torch.no_grad():
        assert torch.equal(ops.swiglu_experts(x, w1, w2, seg, seg_rows), y)
    assert _lib.device_status() == 0
    x64, a64, b64 = (t.detach().double().requires_grad_(True) for t in (x, w1, w2))
    v = (x64 @ a64.transpose(1, 2)).reshape(E, rows, ffn // 8, 2, 8)
    y64 = (torch.nn.functional.silu(v[..., 0, :]) * v[..., 1, :]).reshape(E, rows, ffn) @ b64.transpose(1, 2)
    want = torch.autograd.grad(y64, [x64, a64, b64], dy.double())
    for e in range(E):
        assert _rel(y[e], y64[e]) < 3 * 2.0 ** -9
        for g, w in zip(got, want):
            assert bool(torch.isfinite(g[e]).all()) and _rel(g[e], w[e]) < 5 * 2.0 ** -9


@pytest.mark.parametrize("in_gemm", [True, False])
@pytest.mark.parametrize("T,H,V", [(2048, 256, 4104), (1031, 264, 12808), (300, 64, 40000), (4096, 128, 50304)])
def test_projected_cross_entropy(T, H, V, in_gemm, monkeypatch):
    """Projection and loss in one, statistics in the epilogue or in a pass of their own: a vocabulary that ends inside a chunk of 32 and inside a tile, rows that are no multiple of
    anything, ignored and out-of-range targets, a row of -inf logits' neighbours.  The logits are bf16, so the loss is
    compared with the unfused operations on the same product (fp32 sums: 1e-5) and the gradients with 64 bits (2^-8)."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib

    assert _lib.lib().axb_gemm_on_pairs(T, V, 0)
    monkeypatch.setattr(sys.modules["axonn_b200.ops.loss"], "_statistics_in_epilogue", lambda *_: in_gemm)
    torch.manual_seed(T)
    x = torch.randn(1, T, H, device=DEV).bfloat16().requires_grad_(True)
    w = (torch.randn(V * H, device=DEV) * 0.2).bfloat16().requires_grad_(True)
    t = torch.randint(0, V, (1, T), device=DEV)
    t[0, ::7] = -100
    t[0, 1], t[0, 2], t[0, 3], t[0, 4], t[0, 5] = V - 1, 0, V, V + 5, -1
    loss = ops.projected_cross_entropy(x, w, t, (V, H))
    ref = ops.cross_entropy(ops.matmul_nt(x.detach()[0], w.detach().view(V, H)), t)
    assert abs(float(loss.detach()) - float(ref)) <= 1e-5 * abs(float(ref))
    got = torch.autograd.grad(loss, [x, w], torch.full((), 3.0, device=DEV))
    x64, w64 = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    z = x64[0] @ w64.view(V, H).t()
    z = z + (z.detach().float().bfloat16().double() - z.detach())
    # a target outside the vocabulary has the loss of a target whose logit is zero, and counts
    kept, inside = t[0] != -100, (t[0] >= 0) & (t[0] < V)
    own = z.gather(1, torch.where(inside, t[0], 0)[:, None])[:, 0] * inside
    want = torch.autograd.grad(3 * ((z.logsumexp(1) - own) * kept).sum() / kept.sum(), [x64, w64])
    for a, b in zip(got, want):
        assert a.shape == b.shape and _rel(a, b) < 2.0 ** -8
    assert _lib.device_status() == 0


def test_projected_cross_entropy_odd_rows(monkeypatch):
    """All logits of a row -inf: a NaN loss, as without fusion; a NaN input reaches the loss; -inf in single columns."""
    from axonn_b200 import ops

    monkeypatch.setattr(sys.modules["axonn_b200.ops.loss"], "_statistics_in_epilogue", lambda *_: True)
    T, H, V = 512, 64, 12800
    for kind in ("inf", "nan", "columns"):
        x, w = torch.ones(1, T, H, device=DEV).bfloat16(), torch.zeros(V, H, device=DEV).bfloat16()
        w[:, 0] = torch.linspace(-3, 3, V, device=DEV).bfloat16()
        if kind == "inf":
            x[0, 5, 0] = float("inf")
            w[:, 0] = -1.0
        elif kind == "nan":
            x[0, 5, 0] = float("nan")
        else:
            w[100:900, 0] = float("-inf")
        t = torch.full((1, T), V - 1, device=DEV)
        a = ops.projected_cross_entropy(x, w.view(-1), t, (V, H))
        b = ops.cross_entropy(ops.matmul_nt(x[0], w), t)
        assert bool(a.isnan()) == bool(b.isnan()) and (kind == "columns") != bool(a.isnan())
        if kind == "columns":
            assert abs(float(a) - float(b)) <= 1e-5 * abs(float(b))


def test_lm_head_with_hooks():
    """The head takes the fused path only when calling the projection is nothing but the product."""
    import torch.distributed as dist

    from axonn_b200 import axonn as ax
    from axonn_b200.models import blocks

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    if not ax.is_initialized:
        ax.init(G_inter=1, G_data=1, G_intra_r=1, G_intra_c=1, G_intra_d=1)
    torch.manual_seed(0)
    head = blocks.ParallelLMHead(128, 12800, dtype=BF16)
    x, t = torch.randn(2, 200, 128, device=DEV, dtype=BF16, requires_grad=True), torch.randint(0, 12800, (2, 200), device=DEV)
    assert blocks._is_plain_product(head.proj, x)
    fused = head(x, t)
    assert type(fused.grad_fn).__name__.startswith("_ProjectedCrossEntropy")
    gf = torch.autograd.grad(fused, [x, head.proj.weight])
    seen = []
    handle = head.proj.register_forward_hook(lambda m, i, o: seen.append(o.shape))
    plain = head(x, t)
    handle.remove()
    assert seen == [torch.Size([2, 200, 12800])] and abs(float(plain.detach()) - float(fused.detach())) < 1e-5 * float(plain.detach())
    for a, b in zip(gf, torch.autograd.grad(plain, [x, head.proj.weight])):
        assert a.shape == b.shape and _rel(a, b) < 2.0 ** -8
    own = head.proj.forward
    head.proj.forward = lambda *a, **k: own(*a, **k)                   # replaced on the instance
    assert not blocks._is_plain_product(head.proj, x) and float(head(x, t).detach()) == float(plain.detach())


@pytest.mark.parametrize("act,bias", [("gelu", True), ("gelu", False), ("swiglu", False)])
@pytest.mark.parametrize("rows,hidden,ffn", [(2500, 2048, 4112), (1031, 2112, 8208), (300, 2048, 20000), (2300, 2048, 2192), (800, 2048, 6416)])
def test_mlp_function(act, bias, rows, hidden, ffn):
    """The feed-forward block as one function: rows that end inside a group of 32, columns inside a chunk, with and without
    bias, each gradient by itself, against 64 bits (roundings of 2^-9: three forward, five backward; bias sums are fp32)."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib

    torch.manual_seed(rows)
    wide = 2 * ffn if act == "swiglu" else ffn
    x = torch.randn(1, rows, hidden, device=DEV).bfloat16().requires_grad_(True)
    w1 = (torch.randn(wide * hidden, device=DEV) * hidden ** -0.5).bfloat16().requires_grad_(True)
    w2 = (torch.randn(ffn * hidden, device=DEV) * ffn ** -0.5).bfloat16().requires_grad_(True)
    b1 = torch.randn(wide, device=DEV).bfloat16().requires_grad_(True) if bias else None
    b2 = torch.randn(hidden, device=DEV).bfloat16().requires_grad_(True) if bias else None
    y = ops.mlp(x, w1, b1, w2, b2, hidden, ffn, act)
    assert y is not None and y.shape == x.shape
    leaves = [t for t in (x, w1, b1, w2, b2) if t is not None]
    dy = torch.randn_like(y)
    got = torch.autograd.grad(y, leaves, dy, retain_graph=True)
    for t, g in zip(leaves, got):                    # one at a time gives the same bits
        assert torch.equal(torch.autograd.grad(y, t, dy, retain_graph=True)[0], g)
    assert _lib.device_status() == 0
    l64 = [t.detach().double().requires_grad_(True) for t in leaves]
    it = iter(l64)
    x64, a64 = next(it), next(it)
    c64 = next(it) if bias else 0
    d64 = next(it)
    e64 = next(it) if bias else 0
    z = x64 @ a64.view(wide, hidden).t() + c64
    if act == "swiglu":
        v = z.reshape(1, rows, ffn // 8, 2, 8)
        h = (torch.nn.functional.silu(v[..., 0, :]) * v[..., 1, :]).reshape(1, rows, ffn)
    else:
        h = torch.nn.functional.gelu(z, approximate="tanh")
    y64 = h @ d64.view(hidden, ffn).t() + e64
    assert _rel(y, y64) < 3 * 2.0 ** -9
    for g, w in zip(got, torch.autograd.grad(y64, l64, dy.double())):
        assert g.shape == w.shape and _rel(g, w) < 5 * 2.0 ** -9


def test_mlp_module_routes():
    """The module takes the function in training and its two layers everywhere else, with the same values."""
    import torch.distributed as dist

    from axonn_b200 import axonn as ax
    from axonn_b200 import ops
    from axonn_b200.models.blocks import ParallelMLP

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    if not ax.is_initialized:
        ax.init(G_inter=1, G_data=1, G_intra_r=1, G_intra_c=1, G_intra_d=1)
    torch.manual_seed(0)
    x = torch.randn(2, 1000, 2048, device=DEV, dtype=BF16, requires_grad=True)
    for act in ("gelu", "swiglu"):
        m = ParallelMLP(2048, 2048, act, bias=act == "gelu", dtype=BF16)
        y = m(x)
        assert "MLP" in type(y.grad_fn).__name__
        grads = torch.autograd.grad(y, [x, *m.parameters()], torch.ones_like(y))
        seen = []
        handle = m.fc2.register_forward_pre_hook(lambda mod, i: seen.append(i[0].shape))
        z = m(x)
        handle.remove()
        assert seen == [torch.Size([2, 1000, 2048])] and _rel(y, z) < 2.0 ** -8
        for a, b in zip(grads, torch.autograd.grad(z, [x, *m.parameters()], torch.ones_like(z))):
            assert a.shape == b.shape and _rel(a, b) < 2.0 ** -7
        with torch.no_grad():
            assert _rel(m(x), y) < 2.0 ** -8
        assert ops.mlp(x[:, :1], m.fc1.weight, m.fc1.bias, m.fc2.weight, m.fc2.bias, 2048, 2048, act) is None


@pytest.mark.parametrize("layout", ["gaps", "shifted"])
@pytest.mark.parametrize("op", ["gelu", "swiglu", "experts", "loss", "route"])
def test_saved_tensors_in_other_layouts(op, layout):
    """Hooks on saved tensors give them back with gaps between the elements, or dense but 16 bytes off: the same gradients."""
    from axonn_b200 import ops
    from axonn_b200.parallel import moe

    torch.manual_seed(0)

    def leaf(*shape):
        return (torch.randn(shape, device=DEV) * 0.05).bfloat16().requires_grad_(True)

    if op in ("gelu", "swiglu"):
        leaves = [leaf(4, 1024, 2048), leaf((2 if op == "swiglu" else 1) * 4096 * 2048), leaf(2048 * 4096)]
        call = lambda: ops.mlp(leaves[0], leaves[1], None, leaves[2], None, 2048, 4096, op)  # noqa: E731
    elif op == "experts":
        leaves = [leaf(2, 4096, 64), leaf(2, 4096, 64), leaf(2, 64, 2048)]
        call = lambda: ops.swiglu_experts(*leaves)  # noqa: E731
    elif op == "loss":
        leaves = [leaf(1, 4096, 64), leaf(4096 * 64)]
        t = torch.randint(0, 4096, (1, 4096), device=DEV)
        call = lambda: ops.projected_cross_entropy(*leaves, t, (4096, 64))  # noqa: E731
    else:
        leaves = [leaf(300, 8)]
        call = lambda: (lambda g, a: (g * torch.arange(600, device=DEV).view(300, 2)).sum() + a)(  # noqa: E731
            *moe._LocalRoute.apply(leaves[0], 2, 40, 64)[:2])

    def unpack(t):
        if layout == "gaps":
            return torch.stack([t, t], -1)[..., 0]
        buf = torch.empty(t.numel() + 16 // t.element_size(), dtype=t.dtype, device=t.device)
        return buf[16 // t.element_size():].view(t.shape).copy_(t)

    y = call()
    dy = torch.randn_like(y)
    want = torch.autograd.grad(y, leaves, dy)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach().clone(), unpack):
        y = call()
    for a, b in zip(torch.autograd.grad(y, leaves, dy), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("fused", [True, False])
def test_logits_are_consumed(fused):
    """The backward of the loss overwrites the logits, so that a second one is refused instead of taking gradients for
    logits - unless hooks keep a copy of them."""
    from axonn_b200 import ops

    torch.manual_seed(0)
    x, w = (torch.randn(4096, 64, device=DEV).bfloat16().requires_grad_(True) for _ in range(2))
    t = torch.randint(0, 4096, (4096,), device=DEV)

    def call():
        return ops.projected_cross_entropy(x, w, t, (4096, 64)) if fused else ops.cross_entropy(ops.linear(x, w), t)

    loss = call()
    want = torch.autograd.grad(loss, [x, w], retain_graph=True)
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        torch.autograd.grad(loss, [x, w])
    with torch.autograd.graph.saved_tensors_hooks(lambda s: s.detach().clone(), lambda s: s.clone()):
        loss = call()
    for _ in range(2):
        for a, b in zip(torch.autograd.grad(loss, [x, w], retain_graph=True), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("op", ["gelu", "experts", "loss"])
def test_second_derivatives_are_refused(op):
    """... not left out: the fused backwards are kernels that no graph sees."""
    from axonn_b200 import ops

    def leaf(*shape):
        return (torch.randn(shape, device=DEV) * 0.05).bfloat16().requires_grad_(True)

    if op == "gelu":
        leaves = [leaf(4096, 2048), leaf(4096 * 2048), leaf(2048 * 4096)]
        y = ops.mlp(leaves[0], leaves[1], None, leaves[2], None, 2048, 4096, op)
    elif op == "experts":
        leaves = [leaf(2, 512, 64), leaf(2, 256, 64), leaf(2, 64, 128)]
        y = ops.swiglu_experts(*leaves)
    else:
        leaves = [leaf(4096, 64), leaf(4096 * 64)]
        y = ops.projected_cross_entropy(*leaves, torch.randint(0, 4096, (4096,), device=DEV), (4096, 64))
    (g,) = torch.autograd.grad((y * y).sum(), leaves[-1], create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        g.float().sum().backward()
