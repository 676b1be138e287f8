"""Layers that launch their kernel without an autograd function when no gradient can be asked for: the same results as with
one, and the general path wherever something else looks at the operation."""

import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16 = torch.bfloat16


@pytest.fixture(scope="module", autouse=True)
def _grid():
    from axonn_b200 import axonn as ax

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    if not ax.is_initialized:
        ax.init(G_inter=1, G_data=1, G_intra_r=1, G_intra_c=1, G_intra_d=1)


def _views(shape, dtype):
    """A dense tensor, one 16 bytes into a buffer, one with gaps, one with permuted dimensions."""
    n = 1
    for d in shape:
        n *= d
    base = torch.randn(n + 8, device=DEV).to(dtype)
    wide = torch.randn(*shape[:-1], shape[-1] * 2, device=DEV).to(dtype)
    out = [base[:n].view(shape), base[8:].view(shape), wide[..., :shape[-1]]]
    if len(shape) == 3:
        out.append(torch.randn(shape[1], shape[0], shape[2], device=DEV).to(dtype).transpose(0, 1))
    return out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(16,), (5, 16), (2, 3, 264), (0, 16)])
def test_norms(shape, dtype):
    from axonn_b200 import ops

    H = shape[-1]
    g, b = torch.randn(H, device=DEV).to(dtype), torch.randn(H, device=DEV).to(dtype)
    gg = g.clone().requires_grad_(True)
    for x, d in zip(_views(shape, dtype), reversed(_views(shape, dtype))):
        for rms in (False, True):
            norm = (lambda t, w: ops.rms_norm(t, w)) if rms else (lambda t, w: ops.layer_norm(t, w, b))
            add = (lambda t, w: ops.add_rms_norm(t, d, w)) if rms else (lambda t, w: ops.add_layer_norm(t, d, w, b))
            ref, ref_h, ref_y = norm(x, gg), *add(x, gg)
            assert ref.requires_grad
            with torch.no_grad():
                got, (h, y) = norm(x, gg), add(x, gg)
            assert not got.requires_grad and torch.equal(got, ref) and torch.equal(h, ref_h) and torch.equal(y, ref_y)
            assert got.shape == h.shape == y.shape == x.shape
            if x.numel() == 0:
                continue
            h2, y2 = add(x, g)                       # grad mode on, nothing requires a gradient
            assert torch.equal(h2, ref_h) and not y2.requires_grad
            x3 = x.detach().clone().requires_grad_(True)
            h3, y3 = add(x3, gg)
            (gx,) = torch.autograd.grad([h3, y3], x3, [torch.ones_like(h3), torch.ones_like(y3)])
            assert gx.shape == x.shape


@pytest.mark.parametrize("expert,bias,skip", [(True, True, False), (True, False, False), (False, True, False), (True, True, True)])
@pytest.mark.parametrize("k,n,dtype", [(64, 24, BF16), (264, 520, torch.float16), (24, 20, BF16), (32, 32, torch.float32)])
def test_linear(expert, bias, skip, k, n, dtype):
    from axonn_b200.intra_layer import Linear

    torch.manual_seed(k)
    layer = Linear(k, n, bias=bias, skip_bias_add=skip, expert_mode=expert, dtype=dtype)
    if bias:
        with torch.no_grad():
            layer.bias.normal_()
    for shape in [(k,), (3, k), (2, 5, k), (200, k)]:
        for x in _views(shape, dtype):
            for act in (None, "gelu"):
                if act and (not expert or skip or (not bias and n % 8) or dtype == torch.float32):
                    continue
                try:
                    ref = layer(x, activation=act)
                except Exception as e:               # what the general path refuses stays refused
                    with torch.no_grad(), pytest.raises(type(e)):
                        layer(x, activation=act)
                    continue
                with torch.no_grad():
                    got = layer(x, activation=act)
                for a, r in zip(got, ref) if skip and bias else [(got, ref)]:
                    assert a.shape == r.shape and torch.equal(a, r)
    with torch.no_grad(), torch.autocast("cuda", dtype=BF16):
        assert (layer(torch.randn(4, k, device=DEV))[0] if skip and bias else layer(torch.randn(4, k, device=DEV))).dtype == BF16
    with torch.no_grad(), pytest.raises(Exception):
        layer(torch.randn(4, k + 8, device=DEV).to(dtype))


def test_general_path_is_kept():
    """Forward-mode tangents, function transforms and tracing reach the autograd function, as before."""
    import torch.autograd.forward_ad as fw

    from axonn_b200 import ops
    from axonn_b200.ops.direct import no_graph

    x, w = torch.randn(4, 64, device=DEV, dtype=BF16), torch.ones(64, device=DEV, dtype=BF16)
    assert no_graph(x, w, None) and not no_graph(x.cpu()) and not no_graph(x, w.clone().requires_grad_(True))
    with torch.no_grad():
        assert no_graph(x, w.clone().requires_grad_(True))
        with fw.dual_level():
            assert not no_graph(fw.make_dual(x, torch.ones_like(x)))
            with pytest.raises(RuntimeError):
                ops.rms_norm(fw.make_dual(x, torch.ones_like(x)), w)
        with pytest.raises(RuntimeError):
            torch.func.vmap(lambda t: ops.rms_norm(t, w))(x[None])

    class Sub(torch.Tensor):
        pass

    assert not no_graph(x.as_subclass(Sub))


def test_rope_counts_as_in_place():
    """A tensor saved for a backward and then rotated without a graph is noticed."""
    from axonn_b200 import ops

    table = ops.rope_table(8, 64, 1e4, torch.device("cuda", 0))
    x = torch.randn(1, 8, 2, 64, device=DEV, dtype=BF16, requires_grad=True)
    y = x * 1
    z = y * y
    with torch.no_grad():
        out = ops.apply_rope(y.detach(), table)
    assert out.shape == y.shape
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        z.sum().backward()
    with torch.inference_mode():
        kept = ops.apply_rope(torch.randn(1, 8, 2, 64, device=DEV, dtype=BF16), table)
    with torch.no_grad(), pytest.raises(RuntimeError, match="inference"):
        ops.apply_rope(kept, table)
    y = x * 1
    with torch.no_grad():
        out = ops.apply_rope(y, table)               # rotated outside the graph, so it is not part of it
    assert out.data_ptr() == y.data_ptr() and not out.requires_grad and out.grad_fn is None


def test_embedding_rows(monkeypatch):
    """Rows of consecutive positions: a slice of the table without gradients, the layer itself with them, with a hook, and
    past the ends of the table (what it makes of them is its own; the look-up is a stub here)."""
    from axonn_b200.intra_layer import Embedding, embedding

    e = Embedding(40, 64, expert_mode=True, transpose=True, dtype=BF16)
    dev = torch.device("cuda", 0)
    ref = e(torch.arange(3, 20, device=dev))
    assert ref.requires_grad and e.rows(3, 17, dev).requires_grad
    with torch.no_grad():
        got = e.rows(3, 17, dev)
        assert torch.equal(got, ref) and got.data_ptr() == e.weight.data_ptr() + 3 * 64 * 2 and e.rows(0, 0, dev).shape == (0, 64)
        seen = []
        handle = e.register_forward_hook(lambda m, i, o: seen.append(o.shape))
        assert torch.equal(e.rows(3, 17, dev), ref) and seen == [torch.Size([17, 64])]
        handle.remove()
        asked = []
        monkeypatch.setattr(embedding.F, "embedding", lambda x, *_: asked.append(x.tolist()) or x)
        assert e.rows(23, 17, dev).shape == (17, 64) and not asked
        e.rows(24, 17, dev), e.rows(-1, 2, dev)
        assert asked == [list(range(24, 41)), [-1, 0]]


@pytest.mark.parametrize("rows,hidden,ffn", [(129, 64, 40000), (1000, 256, 2056), (2048, 136, 4104), (777, 512, 8),
                                             (800, 64, 3080), (200, 64, 4096), (1100, 64, 2456)])
def test_swiglu_block(rows, hidden, ffn):
    """The gated block without gradients, rows and columns that end inside tiles and chunks, on the fused product and (few
    columns, few rows) without it: the bits of the layers with their activation between them."""
    from axonn_b200 import ops
    from axonn_b200.models.blocks import ParallelMLP

    torch.manual_seed(rows)
    m = ParallelMLP(hidden, ffn, "swiglu", bias=False, dtype=BF16)
    for x in (torch.randn(rows, hidden, device=DEV, dtype=BF16), torch.randn(1, rows, 2 * hidden, device=DEV, dtype=BF16)[..., :hidden],
              torch.randn(2, 3, hidden, device=DEV, dtype=BF16)):
        with torch.no_grad():
            want = m.fc2(ops.swiglu(m.fc1(x)))
            got = m(x)
        assert got.shape == want.shape and torch.equal(got, want)
    from axonn_b200.ops import _lib

    with torch.no_grad():
        h = ops.swiglu_projection(torch.randn(rows, hidden, device=DEV, dtype=BF16), m.fc1.weight, hidden)
        assert (h is not None) == bool(_lib.lib().axb_gemm_on_pairs(rows, 2 * ffn, 0))


def test_replaced_first_layer():
    """A gated block whose first layer was replaced by a module of any kind runs that module, with gradients and without."""
    from axonn_b200.models.blocks import ParallelMLP

    torch.manual_seed(0)
    m = ParallelMLP(64, 4096, "swiglu", bias=False, dtype=BF16)
    x = torch.randn(2000, 64, device=DEV, dtype=BF16)
    want = m(x)
    m.fc1 = torch.nn.Sequential(m.fc1, torch.nn.Identity())
    assert torch.equal(m(x), want)
    with torch.no_grad():
        assert torch.equal(m(x), want)


def test_replaced_forwards(monkeypatch):
    """A forward replaced on the instance or on the class is called, whatever could stand in for the original."""
    from axonn_b200.intra_layer import Embedding, Linear
    from axonn_b200.models import blocks
    from axonn_b200.ops.direct import plain_layer

    dev = torch.device("cuda", 0)
    e, head = Embedding(40, 64, expert_mode=True, dtype=BF16), blocks.ParallelLMHead(64, 12800, dtype=BF16)
    m = blocks.ParallelMLP(64, 4096, "swiglu", bias=False, dtype=BF16)
    x, t = torch.randn(2000, 64, device=DEV, dtype=BF16), torch.randint(0, 12800, (2000,), device=DEV)

    def calls():
        with torch.no_grad():
            e.rows(3, 4, dev), m(x), head(x, t)
        m(x), head(x, t)

    seen = []
    calls()
    for layer in (e, m.fc1, m.fc2, head.proj):
        assert plain_layer(layer)
        own = layer.forward
        layer.forward = lambda *a, own=own, **k: (seen.append(own), own(*a, **k))[1]
        assert not plain_layer(layer)
    calls()
    assert len(seen) == 1 + 2 * 3
    for layer in (e, m.fc1, m.fc2, head.proj):
        del layer.forward
    seen.clear()
    for cls in (Embedding, Linear):
        own = cls.forward
        monkeypatch.setattr(cls, "forward", lambda self, *a, own=own, **k: (seen.append(own), own(self, *a, **k))[1])
    calls()
    assert len(seen) == 1 + 2 * 3
    monkeypatch.undo()
    assert all(plain_layer(layer) for layer in (e, m.fc1, m.fc2, head.proj))


def test_small_training_steps_are_not_asked(monkeypatch):
    """Blocks of few rows are bound by host time: in a training step they do not go through the questions of the fused
    operations, which could not take them."""
    from axonn_b200.intra_layer import fully_connected
    from axonn_b200.models import blocks

    def asked(*_):
        raise AssertionError("asked")

    monkeypatch.setattr(blocks, "plain_layer", asked)
    monkeypatch.setattr(blocks, "plain_tensors", asked)
    monkeypatch.setattr(fully_connected, "no_graph", asked)
    x, t = torch.randn(1, 64, 256, device=DEV, dtype=BF16, requires_grad=True), torch.randint(0, 512, (1, 64), device=DEV)
    for act in ("gelu", "swiglu"):
        blocks.ParallelMLP(256, 1024, act, bias=act == "gelu", dtype=BF16)(x)
    blocks.ParallelLMHead(256, 512, dtype=BF16)(x, t)
