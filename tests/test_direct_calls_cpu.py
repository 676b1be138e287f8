"""When a layer may launch its kernel by itself: the decision, asked on CPU ranks with the launch replaced by a record."""

import torch

from _dist import run_distributed


def _without_gradients(rank, world, grid, transpose, bias, expert):
    """Tensors of these ranks count as CUDA tensors and the GEMM is a stub that writes zeros."""
    import torch.distributed as dist

    from axonn_b200 import axonn as ax
    from axonn_b200.intra_layer import Linear
    from axonn_b200.intra_layer import fully_connected as fc
    from axonn_b200.intra_layer.communication import _drop

    ax.init(G_inter=1, G_data=1, G_intra_r=grid[0], G_intra_c=grid[1], G_intra_d=1)
    launches = []

    class Lib:
        def axb_gemm(self, *args):
            launches.append(args)
            return 0

    fc.no_graph = lambda *ts: not (torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in ts))
    fc._lib.lib, fc._lib.stream = lambda: Lib(), lambda: None
    torch.manual_seed(1)
    seq = torch.nn.Linear(64, 128, bias=bias).bfloat16()
    layer = Linear(64, 128, bias=bias, transpose=transpose, expert_mode=expert, dtype=torch.bfloat16)
    layer.load_state_dict(seq.state_dict())
    X = torch.randn(8, 64).bfloat16()
    x = _drop(X, 1, layer.inner_group) if expert else _drop(X, 0, dist.group.WORLD)
    with_grad = layer(x)
    assert not launches
    with torch.no_grad():
        y = layer(x)
    assert y.shape == with_grad.shape
    if not launches:
        assert torch.equal(y, with_grad)
        if not expert:
            want = _drop(seq(X), 0, dist.group.WORLD)
            assert (y.float() - want.float()).norm() <= 2 ** -7 * want.float().norm()
    return len(launches)


def _cases(rank, world, cases):
    return [_without_gradients(rank, world, *case) for case in cases]


def test_easy_mode_on_a_grid_is_not_one_launch():
    """Easy mode trades batch for channels whichever group is larger than one: the output is this rank's rows of the whole
    product, without gradients too."""
    cases = [(grid, transpose, bias, False) for grid in ((2, 1), (1, 2)) for transpose in (False, True) for bias in (False, True)]
    assert run_distributed(_cases, 2, cases) == [[0] * 8] * 2


def test_expert_mode_on_a_grid():
    """Expert mode keeps the shard of the outer group, so only the inner group's sum rules the launch out."""
    cases = [((2, 1), False, False, True), ((2, 1), True, False, True), ((1, 2), True, False, True), ((1, 2), False, False, True)]
    assert run_distributed(_cases, 2, cases) == [[1, 0, 1, 0]] * 2


def _other_position_embedding(rank, world):
    from axonn_b200 import axonn as ax
    from axonn_b200.models import GPT, GPTConfig
    from axonn_b200.models.gpt import DistributedGPT

    ax.init(G_inter=1, G_data=1, G_intra_r=1, G_intra_c=1, G_intra_d=1)
    cfg = GPTConfig.tiny()
    for model in (GPT(cfg, dtype=torch.float32), DistributedGPT(cfg, dtype=torch.float32)):
        tokens = torch.randint(0, cfg.vocab, (2, 8))
        want = model(tokens)
        own = model.pos_emb
        table = own.weight.detach().view(cfg.seq_len, cfg.hidden)
        model.pos_emb = torch.nn.Embedding.from_pretrained(table)
        assert torch.equal(model(tokens), want)
        with torch.no_grad():
            assert torch.equal(model(tokens), want)
    return True


def test_replaced_position_embedding():
    """A GPT runs with any module in the place of its position embedding."""
    assert run_distributed(_other_position_embedding, 1) == [True]


def test_feed_forward_result_in_place():
    """What the fused feed-forward block returns may be modified in place (a residual added to it), in any number of
    dimensions."""
    from axonn_b200.ops.mlp import _MLPFn

    torch.manual_seed(0)
    w1, w2 = (torch.randn(128 * 64, requires_grad=True) for _ in range(2))
    for shape in ((6, 64), (2, 3, 64)):
        x = torch.randn(shape, requires_grad=True)
        y = _MLPFn.apply(x, w1, None, w2, None, 64, "gelu")
        z = _MLPFn.apply(x, w1, None, w2, None, 64, "gelu") + x
        y += x
        assert torch.equal(y, z) and y.shape == shape and y.grad_fn is not None


def test_operands_are_copied_only_where_a_kernel_needs_it():
    """Weights inside a flat buffer lie on 16 bytes, which is enough for an operand."""
    from axonn_b200.ops.gemm import as_written

    flat = torch.arange(128, dtype=torch.float32)
    flat = flat[(-flat.data_ptr() // 4) % 8:]                          # starts on 32 bytes
    t = flat[4:68].view(8, 8)
    assert t.data_ptr() % 32 == 16 and as_written(t) is t
    for got in (as_written(t, 32), as_written(t.t().contiguous().t()), as_written(flat[1:65].view(8, 8))):
        assert got.is_contiguous() and got.data_ptr() % 16 == 0 and got.data_ptr() not in (t.data_ptr(), flat[1:].data_ptr())
    assert torch.equal(as_written(t, 32), t) and torch.equal(as_written(t.t()), t.t())
