"""Edges of the kernels' tiles and of the rules that choose between them: remainders, the smallest and largest sizes of
a range, against 64-bit (or integer) references."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(got, want):
    return float((got.detach().double() - want.detach()).norm() / want.detach().norm().clamp_min(1e-30))


# ------------------------------------------------------------------------------------------------ norm backward
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,H", [(1, 8), (3, 256), (17, 264), (301, 512), (5, 520), (2048, 1024), (77, 1032), (4099, 2048),
                                    (9, 2056), (1001, 4096), (6, 4104), (613, 8192), (5, 8200), (128, 768), (129, 768), (443, 512),
                                    (445, 512), (591, 2056), (593, 1032), (5921, 1536), (8141, 1024)])
@pytest.mark.parametrize("rms,residual", [(True, False), (False, True)])
def test_norm_backward_sizes(rows, H, rms, residual, dtype):
    """Thread groups per row change at hidden 256, 512, 1024, 2048, 4096; the batch of rows per block and the ring of
    loads end at any row.  Tolerance: results are rounded once to the storage type (2^-9 bf16, 2^-11 fp16), on top of
    fp32 arithmetic (1e-5)."""
    from axonn_b200 import ops

    torch.manual_seed(rows + H)
    x, dl, dy, dh = (torch.randn(rows, H, device=DEV).to(dtype) for _ in range(4))
    g = (1 + 0.1 * torch.randn(H, device=DEV)).to(dtype).requires_grad_(True)
    b = None if rms else (0.1 * torch.randn(H, device=DEV)).to(dtype).requires_grad_(True)
    x.requires_grad_(True)
    leaves = [x, g] + ([] if rms else [b])
    if residual:
        h, y = ops.add_rms_norm(x, dl, g, 1e-5) if rms else ops.add_layer_norm(x, dl, g, b, 1e-5)
        got = torch.autograd.grad([h, y], leaves, [dh, dy])
        base = h.detach().double()
    else:
        y = ops.rms_norm(x, g, 1e-5) if rms else ops.layer_norm(x, g, b, 1e-5)
        got = torch.autograd.grad(y, leaves, dy)
        base = x.detach().double()
    g64 = g.detach().double()
    mean = torch.zeros(rows, 1, device=DEV, dtype=torch.float64) if rms else base.mean(-1, keepdim=True)
    rstd = (base.pow(2).mean(-1, keepdim=True) - mean * mean + 1e-5).rsqrt()
    xh, d = (base - mean) * rstd, dy.double()
    gd = d * g64
    want = [rstd * (gd - (0 if rms else gd.mean(-1, keepdim=True)) - xh * (gd * xh).mean(-1, keepdim=True)), (d * xh).sum(0)]
    if residual:
        want[0] = want[0] + dh.double()
    if not rms:
        want.append(d.sum(0))
    tol = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10, torch.float32: 2e-5}[dtype]
    for a, w in zip(got, want):
        assert _rel(a, w) < tol, _rel(a, w)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,H", [(1, 8), (17, 264), (301, 512), (5, 520), (77, 1032), (4099, 2048), (9, 2056), (1001, 4096),
                                    (6, 4104), (613, 8192), (5, 8200), (2500, 1024), (887, 520), (889, 520), (591, 1032), (593, 1032),
                                    (601, 2056), (601, 2048), (148, 5120), (149, 5120), (2963, 6144)])
@pytest.mark.parametrize("rms", [True, False])
@pytest.mark.parametrize("residual", [True, False])
def test_norm_forward_sizes(rows, H, rms, residual, dtype):
    """Outputs of the forward at the sizes where its thread groups, rings and kernels change.  The residual sum is exact
    (one rounding of an fp32 sum); the normalised rows are rounded once to the storage type (2^-9 bf16, 2^-11 fp16) on
    top of fp32 arithmetic (1e-5), row by row."""
    from axonn_b200 import ops

    torch.manual_seed(rows + H)
    x, dl = (torch.randn(rows, H, device=DEV).to(dtype) for _ in range(2))
    g = (1 + 0.1 * torch.randn(H, device=DEV)).to(dtype)
    b = None if rms else (0.1 * torch.randn(H, device=DEV)).to(dtype)
    if residual:
        h, y = ops.add_rms_norm(x, dl, g, 1e-5) if rms else ops.add_layer_norm(x, dl, g, b, 1e-5)
        assert torch.equal(h, (x.float() + dl.float()).to(dtype))
    else:
        h, y = x, (ops.rms_norm(x, g, 1e-5) if rms else ops.layer_norm(x, g, b, 1e-5))
    z = h.double()
    mean = 0 if rms else z.mean(-1, keepdim=True)
    want = (z - mean) * ((z - mean).pow(2).mean(-1, keepdim=True) + 1e-5).rsqrt() * g.double() + (0 if rms else b.double())
    tol = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10, torch.float32: 2e-5}[dtype]
    assert float(((y.double() - want).norm(dim=-1) / want.norm(dim=-1)).max()) < tol


# ------------------------------------------------------------------------------------------------ attention, any length
@pytest.mark.parametrize("B,S,G,qpk,D", [(1, 1, 1, 1, 64), (2, 5, 2, 1, 128), (3, 127, 1, 2, 64), (2, 129, 2, 2, 128),
                                         (2, 255, 1, 4, 128), (1, 257, 2, 1, 64), (3, 300, 2, 2, 128), (2, 511, 1, 1, 128),
                                         (2, 128, 2, 2, 64), (2, 384, 2, 1, 128), (1, 1531, 2, 4, 128)])
def test_attention_any_length(B, S, G, qpk, D):
    """Sequence ends inside either query tile of a pair, on a tile edge, and before the first one.  Rows of the next
    batch element must not leak in: every element of the batch is compared.  Tolerance: probabilities and score
    gradients are bf16 MMA operands, results are bf16 (a few 2^-9)."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib, attention_cuda

    torch.manual_seed(S)
    qkv = torch.randn(B, S, G, qpk + 2, D, device=DEV).bfloat16().requires_grad_(True)
    dout = torch.randn(B, S, G * qpk, D, device=DEV).bfloat16()
    assert attention_cuda.supported(qkv)
    out = ops.flash_attention_packed(qkv)
    (grad,) = torch.autograd.grad(out, qkv, dout)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    x = qkv.detach().double().requires_grad_(True)
    q = x[:, :, :, :qpk]
    s = torch.einsum("bsgqd,btgd->bgqst", q, x[:, :, :, qpk]) / math.sqrt(D)
    s = s.masked_fill(torch.ones(S, S, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
    ref = torch.einsum("bgqst,btgd->bsgqd", s.softmax(-1), x[:, :, :, qpk + 1]).reshape(B, S, G * qpk, D)
    (gref,) = torch.autograd.grad(ref, x, dout.double())
    for bb in range(B):
        assert _rel(out[bb], ref.detach()[bb]) < 1e-2
        for sl in (slice(0, qpk), slice(qpk, qpk + 1), slice(qpk + 1, qpk + 2)):
            want = gref[bb, :, :, sl]
            err = float((grad[bb, :, :, sl].double() - want).norm())
            # with one key the score gradients vanish: compare with the size of dV, the gradient that is left
            assert err < 1.5e-2 * max(float(want.norm()), float(gref[bb].norm()) * 1e-2), (bb, sl, err)


@pytest.mark.parametrize("B,S,G,qpk,D", [(2, 777, 4, 2, 128), (4, 640, 4, 1, 64), (2, 1531, 4, 1, 128), (2, 896, 2, 2, 128)])
def test_attention_precision_off_256(B, S, G, qpk, D):
    """Lengths that are not multiples of 256: the log-sum-exp to fp32 rounding (sums of at most 1531 positive terms and
    two logarithms of magnitude 10: below 1e-5), and outputs no further from 64 bits than the library's attention,
    which rounds the same probabilities to bf16 (0.3 % for the sampling of the rounding errors)."""
    from axonn_b200.ops.attention_cuda import flash_fwd_packed

    torch.manual_seed(S)
    qkv = torch.randn(B, S, G, qpk + 2, D, device=DEV).bfloat16()
    out, lse = flash_fwd_packed(qkv, 1 / math.sqrt(D))
    x = qkv.double()
    s = torch.einsum("bsgqd,btgd->bgqst", x[:, :, :, :qpk], x[:, :, :, qpk]) / math.sqrt(D)
    s = s.masked_fill(torch.ones(S, S, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
    assert float((lse.double() - s.logsumexp(-1).reshape(B, G * qpk, S)).abs().max()) < 1e-5
    ref = torch.einsum("bgqst,btgd->bsgqd", s.softmax(-1), x[:, :, :, qpk + 1]).reshape(B, S, G * qpk, D)
    q, k, v = qkv[:, :, :, :qpk].reshape(B, S, G * qpk, D), qkv[:, :, :, qpk], qkv[:, :, :, qpk + 1]
    k, v = (t.repeat_interleave(qpk, 2) for t in (k, v))
    lib = torch.nn.functional.scaled_dot_product_attention(*(t.transpose(1, 2) for t in (q, k, v)), is_causal=True).transpose(1, 2)
    assert _rel(out, ref) < 1.003 * _rel(lib, ref)


@pytest.mark.parametrize("S", [77, 300, 384])
def test_attention_lets_nan_through(S):
    """A NaN key reaches every query that sees it, and no other."""
    from axonn_b200 import ops

    for at in (0, 2, 9, S - 1):
        qkv = torch.randn(1, S, 2, 3, 64, device=DEV).bfloat16()
        qkv[0, at, 0, 1, 5] = float("nan")
        out = ops.flash_attention_packed(qkv)
        assert bool(out[0, at:, 0].isnan().all()) and bool(out[0, :at, 0].isfinite().all())
        assert bool(out[0, :, 1].isfinite().all())


@pytest.mark.parametrize("S", [77, 128, 256])
@pytest.mark.parametrize("scale", [0.0, -0.3])
def test_attention_other_scales(S, scale):
    """A scale that is not positive takes the general path: forward and backward against 64 bits (bf16 results and
    probabilities, as above)."""
    from axonn_b200 import ops

    torch.manual_seed(S)
    B, G, qpk, D = 2, 2, 2, 64
    qkv = torch.randn(B, S, G, qpk + 2, D, device=DEV).bfloat16().requires_grad_(True)
    dout = torch.randn(B, S, G * qpk, D, device=DEV).bfloat16()
    out = ops.flash_attention_packed(qkv, scale=scale)
    (grad,) = torch.autograd.grad(out, qkv, dout)
    x = qkv.detach().double().requires_grad_(True)
    s = torch.einsum("bsgqd,btgd->bgqst", x[:, :, :, :qpk], x[:, :, :, qpk]) * scale
    s = s.masked_fill(torch.ones(S, S, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
    ref = torch.einsum("bgqst,btgd->bsgqd", s.softmax(-1), x[:, :, :, qpk + 1]).reshape(B, S, G * qpk, D)
    (gref,) = torch.autograd.grad(ref, x, dout.double())
    assert _rel(out, ref) < 1e-2 and _rel(grad, gref) < 1.5e-2


# ------------------------------------------------------------------------------------------------ split-K GEMM
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("M,N,K", [(8, 128, 256), (24, 2048, 8192), (24, 8192, 2048), (120, 136, 1000), (136, 264, 520),
                                   (128, 1024, 4096), (256, 256, 16384), (1, 512, 2048), (33, 40, 4104),
                                   (120, 136, 8200), (100, 264, 3080), (128, 2056, 2568), (40, 8200, 1544)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gemm_few_tiles(layout, M, N, K, dtype):
    """Problems of few tiles (K split over a cluster), rows and columns that end inside a tile, K blocks that do not
    divide evenly; bias, GELU, accumulation and fp32 output go through the shared epilogue."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib

    if layout == "tn" and M % 8:
        M = 8 * ((M + 7) // 8)
    torch.manual_seed(M + N + K)
    a = torch.randn((M, K) if layout != "tn" else (K, M), device=DEV).to(dtype)
    b = torch.randn((N, K) if layout == "nt" else (K, N), device=DEV).to(dtype)
    want = (a.double() if layout != "tn" else a.double().t()) @ (b.double().t() if layout == "nt" else b.double())
    f = {"nt": ops.matmul_nt, "nn": ops.matmul_nn, "tn": ops.matmul_tn}[layout]
    one = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10
    assert _rel(f(a, b), want) < one
    got = f(a, b, out_dtype=torch.float32)
    assert got.dtype == torch.float32 and _rel(got, want) < 1e-5
    base = torch.randn(M, N, device=DEV)
    assert _rel(f(a, b, out=base.clone(), accumulate=True), want + base.double()) < 1e-5
    if layout == "nt":
        bias = torch.randn(N, device=DEV).to(dtype)
        pre = torch.empty(M, N, device=DEV, dtype=dtype)
        act = ops.matmul_nt(a, b, bias=bias, epilogue=ops.EPI_BIAS_GELU, aux=pre)
        w = want + bias.double()
        assert _rel(pre, w) < one
        assert _rel(act, torch.nn.functional.gelu(w, approximate="tanh")) < 2 * one
    torch.cuda.synchronize()
    assert _lib.device_status() == 0


@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(777, 4104, 1000), (1500, 2056, 520), (136, 16136, 512)])
def test_gemm_one_wave_of_pairs(M, N, K, dtype, layout):
    """Two waves of single tiles that one wave of CTA pairs replaces: rows, columns and K blocks end inside a tile, the
    last column chunk of a row is 8 wide, and the bias starts off a 16-byte boundary.  Tolerance: one rounding to the
    storage type; fp32 sums."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib

    if layout == "tn":
        M = M // 8 * 8
    torch.manual_seed(M + N + K)
    a = torch.randn((M, K) if layout != "tn" else (K, M), device=DEV).to(dtype)
    b = torch.randn((N, K) if layout == "nt" else (K, N), device=DEV).to(dtype)
    want = (a.double() if layout != "tn" else a.double().t()) @ (b.double().t() if layout == "nt" else b.double())
    f = {"nt": ops.matmul_nt, "nn": ops.matmul_nn, "tn": ops.matmul_tn}[layout]
    one = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10
    assert _rel(f(a, b), want) < one
    base = torch.randn(M, N, device=DEV)
    assert _rel(f(a, b, out=base.clone(), accumulate=True), want + base.double()) < 1e-5
    if layout == "nt":
        for off in (0, 1):
            bias = torch.randn(N + 1, device=DEV).to(dtype)[off:N + off]
            pre = torch.empty(M, N, device=DEV, dtype=dtype)
            act = ops.matmul_nt(a, b, bias=bias, epilogue=ops.EPI_BIAS_GELU, aux=pre)
            w = want + bias.double()
            assert _rel(pre, w) < one
            assert _rel(act, torch.nn.functional.gelu(w, approximate="tanh")) < 2 * one
            assert _rel(ops.matmul_nt(a, b, bias=bias, epilogue=ops.EPI_BIAS), w) < one
    torch.cuda.synchronize()
    assert _lib.device_status() == 0


@pytest.mark.parametrize("rows,N,K", [(192, 320, 328), (512, 264, 128)])
def test_batched_gemm_one_segment(rows, N, K):
    """One segment per problem: the weight gradient loops over the K blocks with data only.  Counts at the edges of a
    block, none and all; rows past a count are zero and stay so."""
    from axonn_b200.ops import _lib, gemm

    torch.manual_seed(rows)
    counts = [0, 1, 63, 64, 65, 128, rows - 1, rows]
    seg = torch.tensor(counts, dtype=torch.int32, device=DEV).view(-1, 1)
    live = torch.arange(rows, device=DEV)[None, :] < seg.long()
    E = len(counts)
    a = torch.randn(E, rows, K, device=DEV).bfloat16() * live[:, :, None]
    b = torch.randn(E, N, K, device=DEV).bfloat16()
    g = torch.randn(E, rows, N, device=DEV).bfloat16() * live[:, :, None]
    y, gx = gemm.bmm_nt(a, b, seg=seg, seg_rows=rows), gemm.bmm_nn(g, b, seg=seg, seg_rows=rows)
    gw = gemm.bmm_tn(g, a, out_dtype=torch.float32, seg=seg, seg_rows=rows)
    assert bool((y[~live] == 0).all()) and bool((gx[~live] == 0).all()) and bool((gw[0] == 0).all())
    for e in range(1, E):
        a64, b64, g64 = a[e].double(), b[e].double(), g[e].double()
        assert _rel(y[e], a64 @ b64.t()) < 2.0 ** -8
        assert _rel(gx[e], g64 @ b64) < 2.0 ** -8
        assert _rel(gw[e], g64.t() @ a64) < 1e-5
    torch.cuda.synchronize()
    assert _lib.device_status() == 0


# ------------------------------------------------------------------------------------------------ threads
@pytest.mark.parametrize("op", ["gemm", "batched", "attention"])
def test_first_call_of_a_thread(op):
    """A new thread (autograd's worker at the start of a backward, for one) has no context before its first runtime call;
    the tensor maps of these kernels are encoded before anything is launched."""
    import threading

    from axonn_b200 import ops
    from axonn_b200.ops.gemm import bmm_nt

    a, b = (torch.randn(2, 256, 256, device=DEV).bfloat16() for _ in range(2))
    qkv = torch.randn(1, 256, 2, 3, 64, device=DEV).bfloat16()
    call = {"gemm": lambda: ops.matmul_nt(a[0], b[0]), "batched": lambda: bmm_nt(a, b),
            "attention": lambda: ops.flash_attention_packed(qkv)}[op]
    want, got = call(), []                        # the allocator holds blocks of the sizes that the thread will ask for
    torch.cuda.synchronize()
    keep = want.clone()
    del want
    th = threading.Thread(target=lambda: got.append(call()))
    th.start()
    th.join()
    assert got and torch.equal(got[0], keep)


# ------------------------------------------------------------------------------------------------ cross-entropy
@pytest.mark.parametrize("rows,V", [(1, 8), (3, 4096), (5, 4104), (7, 16384), (2, 16392), (1030, 50304)])
def test_cross_entropy_rows(rows, V):
    """Rows shorter than one batch of vectors, exactly one, one more; ignored targets, a row whose first vectors are all
    -inf, maxima that grow along the row.  Tolerance: fp32 sums."""
    from axonn_b200 import ops

    torch.manual_seed(V)
    z = (torch.randn(rows, V, device=DEV) * 3 + torch.linspace(-20, 20, V, device=DEV)).bfloat16()
    z[0, : V // 2] = float("-inf")
    t = torch.randint(V // 2, V, (rows,), device=DEV)
    if rows > 2:
        t[1] = -100
    ref = torch.nn.functional.cross_entropy(z.double(), t)
    x = z.clone().requires_grad_(True)
    loss = ops.cross_entropy(x, t)
    assert abs(float(loss) - float(ref)) < 1e-5 * abs(float(ref)) + 1e-6
    (g,) = torch.autograd.grad(loss * 2.0, x)
    zr = z.double().requires_grad_(True)
    (gr,) = torch.autograd.grad(torch.nn.functional.cross_entropy(zr, t) * 2.0, zr)
    assert _rel(g, gr) < 2.0 ** -8


# ------------------------------------------------------------------------------------------------ in-place scale
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_scale_sizes_and_offsets(dtype):
    """Chunk edges, vector remainders and tensors that do not start on a 16-byte boundary; one is the identity."""
    from axonn_b200 import ops

    torch.manual_seed(1)
    sizes = [1, 7, 8, 9, 65535, 65536, 65537, 200003]
    base = [torch.randn(n + 1, device=DEV).to(dtype) for n in sizes]
    tensors = [t[:-1] for t in base] + [t[1:] for t in base]
    for s in (0.37, 1.0):
        work = [t.clone() if t.data_ptr() % 16 == 0 else torch.cat([t[:1], t])[1:] for t in tensors]
        want = [(t.float() * s).to(dtype) for t in work]
        ops.multi_tensor_scale_(work, s)
        assert all(torch.equal(a, b) for a, b in zip(work, want))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 1023, 1024, 1025, 2500])
def test_tables_of_many_tensors(n):
    """The search for a unit's tensor narrows 32-fold per round: table lengths around powers of 32, tensors without
    elements, of less than a unit, of exactly one chunk and of several.  Scale: each product rounded once (exact).  Norm:
    fp32 sums.  AdamW: fp32 arithmetic against the plain update (5e-6 of the size of a parameter and its step)."""
    from axonn_b200.ops import _lib
    from axonn_b200.ops.multi_tensor import _PtrTable
    from axonn_b200.ops.optim_step import adamw_reference_
    from axonn_b200.optim import FusedAdamW

    torch.manual_seed(n)
    kinds = [5, 16384, 0, 16385, 3, 65536, 0, 0, 70001, 1]
    sizes = [kinds[(i * 7 + i // 10) % 10] if n < 1000 or i % 50 == 0 else (i * 37) % 3000 for i in range(n)]
    sizes[0] = sizes[0] or 9
    ts = [torch.randn(m, device=DEV) for m in sizes]
    want = [t * 0.37 for t in ts]
    tab = _PtrTable(ts)
    norm = torch.zeros((), device=DEV)
    L = _lib.lib()
    _lib.check(L.axb_multi_l2norm_sq(_lib.addr(tab.dev), tab.n, tab.total_chunks, _lib.addr(norm), _lib.stream()), "norm")
    ref = sum(float(t.double().pow(2).sum()) for t in ts)
    assert abs(float(norm) - ref) < 1e-5 * ref
    s = torch.full((), 0.37, device=DEV)
    _lib.check(L.axb_multi_scale(_lib.addr(tab.dev), tab.n, tab.total_chunks, _lib.addr(s), _lib.stream()), "scale")
    assert all(torch.equal(a, b) for a, b in zip(ts, want))
    ps = [torch.nn.Parameter(t.clone()) for t in ts if t.numel()]
    for p in ps:
        p.grad = torch.randn_like(p)
    ref = [(p.detach().clone(), torch.zeros_like(p), torch.zeros_like(p)) for p in ps]
    FusedAdamW(ps, lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1).step()
    for p, (w, m, v) in zip(ps, ref):
        adamw_reference_(w, p.grad, m, v, 1e-2, 0.9, 0.95, 1e-8, 0.1, 1)
    got, ref = torch.cat([p.detach() for p in ps]), torch.cat([r[0] for r in ref])
    assert float((got - ref).abs().max()) < 5e-6 * max(1.0, float(ref.abs().max()))


# ------------------------------------------------------------------------------------------------ gradient pruning
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("offset", [0, 2, 4])
def test_prune_workspace_of_8_byte_alignment(offset, dtype):
    """The C entry point takes scratch at any 8-byte boundary (``offset``: 32-bit words); values are kept or zeroed, so
    the comparison is exact."""
    from axonn_b200.ops import _lib
    from axonn_b200.ops.optim_step import _LIB_DTYPE

    torch.manual_seed(offset)
    L = _lib.lib()
    g = torch.randn(300_001, device=DEV).to(dtype)
    k = 30_000
    ws = torch.empty(L.axb_prune_workspace_words() + 4, dtype=torch.int32, device=DEV)[offset:]
    want = torch.where(g.abs().float() >= g.abs().float().sort(descending=True)[0][k - 1], g, torch.zeros_like(g))
    _lib.check(L.axb_prune_topk(_lib.addr(g), g.numel(), _LIB_DTYPE[dtype], k, _lib.addr(ws), 0, _lib.stream()), "axb_prune_topk")
    assert torch.equal(g, want)


def test_prune_on_two_streams():
    """Calls that overlap on two streams have their own scratch: histograms, ranks and the block counter of one are not
    touched by the other.  Exact."""
    from axonn_b200 import ops

    torch.manual_seed(0)
    new = [torch.randn(n, device=DEV).bfloat16() * s for n, s in ((24_000_000, 1.0), (16_000_003, 1e-3))]
    want = [torch.where(g.abs().float() >= g.abs().float().sort(descending=True)[0][g.numel() // 10 - 1], g,
                        torch.zeros_like(g)) for g in (t[: t.numel() // 10 * 10] for t in new)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    work = [[t[: t.numel() // 10 * 10].clone() for _ in range(8)] for t in new]
    torch.cuda.synchronize()
    for i in range(8):
        for st, ts in zip(streams, work):
            with torch.cuda.stream(st):
                ops.prune_topk_(ts[i], 0.1)
    torch.cuda.synchronize()
    for w, ts in zip(want, work):
        assert all(torch.equal(t, w) for t in ts)


# ------------------------------------------------------------------------------------------------ local experts
@pytest.mark.parametrize("T,E,k,C", [(1, 4, 2, 8), (5, 8, 2, 8), (1000, 8, 2, 312), (4097, 4, 2, 2048), (8192, 8, 2, 2560),
                                     (3000, 5, 1, 64)])
def test_moe_slots(T, E, k, C):
    """Slots are running counts per expert in assignment order (integers: exact), also past one chunk of the scan and
    for experts that overflow their capacity."""
    import ctypes

    from axonn_b200.ops import _lib

    torch.manual_seed(T)
    idx = torch.rand(T, E, device=DEV).mul_(torch.linspace(0.5, 1.5, E, device=DEV)).topk(k, -1)[1].contiguous()
    n, rows = T * k, (C + 63) // 64 * 64
    dest, inv, cnt = (torch.full((m,), -7, dtype=torch.int32, device=DEV) for m in (n, E * rows, E))
    assigned = torch.empty(E, device=DEV)
    _lib.check(_lib.lib().axb_moe_slots(_lib.ptr(idx), ctypes.c_longlong(n), ctypes.c_int(E), ctypes.c_int(C),
                                        ctypes.c_int(rows), _lib.ptr(dest), _lib.ptr(inv), _lib.ptr(cnt),
                                        _lib.ptr(assigned), _lib.stream_ptr()), "axb_moe_slots")
    flat = idx.reshape(-1).tolist()
    seen, want, winv = [0] * E, [], [-1] * (E * rows)
    for a, e in enumerate(flat):
        ok = seen[e] < C
        want.append(e * rows + seen[e] if ok else -1)
        if ok:
            winv[e * rows + seen[e]] = a
        seen[e] += 1
    assert dest.tolist() == want and inv.tolist() == winv
    assert cnt.tolist() == [min(s, C) for s in seen] and assigned.tolist() == [float(s) for s in seen]


@pytest.mark.parametrize("T,k,rows,H", [(1, 1, 64, 8), (77, 2, 128, 264), (500, 3, 512, 2048)])
def test_moe_permutations(T, k, rows, H):
    """Dispatch, combine and their adjoints against indexing in 64 bits, with dropped assignments and empty rows."""
    from axonn_b200.parallel import moe

    torch.manual_seed(H)
    E = 4
    n = T * k
    perm = torch.randperm(E * rows, device=DEV)[:n].int()
    dest = torch.where(torch.rand(n, device=DEV) < 0.2, torch.full_like(perm, -1), perm)
    inv = torch.full((E * rows,), -1, dtype=torch.int32, device=DEV)
    kept = dest >= 0
    inv[dest[kept].long()] = torch.arange(n, device=DEV, dtype=torch.int32)[kept]
    x = torch.randn(T, H, device=DEV).bfloat16().requires_grad_(True)
    gate = torch.rand(T, k, device=DEV).requires_grad_(True)
    buf = moe._LocalDispatch.apply(x, dest, inv, E, rows, k)
    ref = torch.zeros(E * rows, H, device=DEV, dtype=torch.bfloat16)
    tok = torch.arange(T, device=DEV).repeat_interleave(k)
    ref[dest[kept].long()] = x.detach()[tok[kept]]
    assert torch.equal(buf.detach().view(-1, H), ref)
    gbuf = torch.randn_like(buf)
    (dx,) = torch.autograd.grad(buf, x, gbuf)
    rows64 = gbuf.double().view(-1, H)
    want = torch.zeros(T, H, device=DEV, dtype=torch.float64).index_add(0, tok[kept], rows64[dest[kept].long()])
    assert _rel(dx, want) < 2.0 ** -8
    out = torch.randn(E, rows, H, device=DEV).bfloat16().requires_grad_(True)
    y = moe._LocalCombine.apply(out, gate, dest, inv, T, k)
    o64, g64 = out.detach().double().requires_grad_(True), gate.detach().double().requires_grad_(True)
    y64 = torch.zeros(T, H, device=DEV, dtype=torch.float64).index_add(
        0, tok[kept], o64.view(-1, H)[dest[kept].long()] * g64.view(-1)[kept][:, None])
    assert _rel(y.detach(), y64.detach()) < 2.0 ** -8
    dy = torch.randn_like(y)
    got, want = torch.autograd.grad(y, [out, gate], dy), torch.autograd.grad(y64, [o64, g64], dy.double())
    assert _rel(got[0], want[0]) < 2.0 ** -8 and _rel(got[1], want[1]) < 1e-5


def _local_moe(rank, world, T, hidden, ffn, E, k):
    from axonn_b200 import axonn as ax
    from axonn_b200 import ops
    from axonn_b200.ops import _lib
    from axonn_b200.parallel.moe import ExpertParallelMoE, route_top_k

    ax.init(G_inter=1, G_data=world)
    torch.manual_seed(T)
    layer = ExpertParallelMoE(hidden, ffn, n_experts=E, top_k=k, dtype=torch.bfloat16)
    with torch.no_grad():                          # the first expert overflows, the last one is never chosen
        layer.router[0, 0], layer.router[-1, 0] = 0.5, -50.0
    x = torch.randn(T, hidden, device=DEV).bfloat16()
    x[:, 0] = 1.0
    x.requires_grad_(True)
    y = layer(x)
    dy = torch.randn_like(y)
    params = [x, layer.router, layer.w1, layer.w2]
    got = torch.autograd.grad([y, layer.last_aux_loss], params, [dy, torch.full((), 0.02, device=DEV)])
    assert _lib.device_status() == 0

    C = layer.capacity(T)
    with torch.no_grad():
        idx, _, slot, keep, aux = route_top_k(ops.linear(x, layer.router), k, C)
    per = torch.zeros(E, device=DEV).index_add(0, idx.reshape(-1), torch.ones(T * k, device=DEV))
    assert float(per.max()) > C and float(per[-1]) == 0
    assert torch.equal(layer.last_assignments_per_expert, per)
    assert torch.equal(layer.last_dropped_per_expert, (per - C).clamp_min(0))
    assert abs(float(layer.last_drop_fraction) - float((~keep).float().mean())) < 1e-6
    x64, r64, w1, w2 = (p.detach().double().requires_grad_(True) for p in params)
    z = x64 @ r64.t()
    z = z + (z.to(torch.bfloat16).double() - z).detach()          # the router's logits are bf16 values
    probs = z.softmax(-1)
    gate = probs.gather(1, idx)
    gate = gate / gate.sum(-1, keepdim=True)
    ref = torch.zeros(T, hidden, dtype=torch.float64, device=DEV)
    for e in range(E):
        tok, which = ((idx == e) & keep).nonzero(as_tuple=True)
        v = (x64[tok] @ w1[e].t()).reshape(-1, ffn // 8, 2, 8)    # gate and up rows interleave in blocks of 8
        h = (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(-1, ffn)
        ref = ref.index_add(0, tok, (h @ w2[e].t()) * gate[tok, which][:, None])
    aux64 = E * (per.double() / (T * k) * probs.mean(0)).sum()
    want = torch.autograd.grad([ref, aux64], [x64, r64, w1, w2], [dy.double(), torch.full((), 0.02, dtype=torch.float64, device=DEV)])
    assert abs(float(layer.last_aux_loss) - float(aux64)) < 1e-4 * abs(float(aux64))
    return [_rel(y, ref)] + [_rel(a, b) for a, b in zip(got, want)], bool((got[3][-1] == 0).all() and (got[2][-1] == 0).all())


@pytest.mark.parametrize("T,hidden,ffn,E,k", [(517, 256, 512, 4, 2), (96, 136, 72, 5, 1), (2000, 512, 1024, 8, 2)])
def test_local_moe_layer(T, hidden, ffn, E, k):
    """The whole layer with all experts on one GPU, an expert past its capacity and one without tokens, against routing in
    torch and 64-bit experts.  Tolerance: the layer's intermediates are bf16 (four roundings of 2^-9 forward, twice as
    many backward; the router's gradient is a difference of such sums)."""
    from _dist import run_distributed

    errors, empty = run_distributed(_local_moe, 1, T, hidden, ffn, E, k, backend="nccl", timeout=300)[0]
    assert empty
    assert errors[0] < 1e-2 and max(errors[1], errors[3], errors[4]) < 1.5e-2 and errors[2] < 2e-2, errors
