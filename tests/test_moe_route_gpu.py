"""The routing kernel of the local mixture-of-experts layer against torch's softmax and top-k."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _route(logits, k, C, rows):
    from axonn_b200.parallel import moe

    return moe._LocalRoute.apply(logits, k, C, rows)


@pytest.mark.parametrize("T,E,k,C", [(1, 1, 1, 8), (5, 3, 2, 8), (127, 4, 4, 40), (128, 8, 2, 40), (129, 8, 1, 24), (4097, 9, 2, 1000),
                                     (3000, 16, 3, 704), (8192, 8, 2, 2560), (600, 17, 2, 96), (600, 32, 8, 200)])
def test_route(T, E, k, C):
    """One block and many, every register width, ties (bf16 logits on a coarse grid: equal probabilities are taken in the
    order of the experts), experts past their capacity.  The same experts as torch.topk; gates and balance loss are fp32
    (2e-6 relative), gradients are rounded to bf16 once (2^-9)."""
    torch.manual_seed(T + E)
    z = ((torch.randn(T, E, device=DEV) * 4).round() / 4 + 0.5 * torch.arange(E, device=DEV) / E).bfloat16().requires_grad_(True)
    rows = (C + 63) // 64 * 64
    gate, aux, dest, inverse, counts, stats = _route(z, k, C, rows)
    idx = F.softmax(z.detach().float(), -1).topk(k, -1)[1]
    # a token's experts as a set: which of two equal ones comes first does not matter
    chosen = torch.full((T, E), False, device=DEV).scatter(1, idx, True)
    z64 = z.detach().double().requires_grad_(True)
    q = z64.softmax(-1)
    per = chosen.sum(0).float()
    assert torch.equal(stats[:E], per) and torch.equal(stats[E:2 * E], (per - C).clamp_min(0))
    assert torch.equal(counts.float(), per.clamp_max(C))
    assert abs(float(stats[2 * E]) - float((per - C).clamp_min(0).sum()) / (T * k)) < 1e-6
    aux64 = E * (per.double() / (T * k) * q.mean(0)).sum()
    assert abs(float(aux.detach()) - float(aux64)) < 2e-6 * float(aux64)
    dense64 = q * chosen / (q * chosen).sum(-1, keepdim=True)
    assert float((gate.detach().double().sort(-1)[0] - dense64.detach().topk(k, -1)[0].sort(-1)[0]).abs().max()) < 1e-6
    # every kept assignment lies where the inverse map says, in the buffer of an expert that the token has chosen
    d = dest.view(T, k).long()
    kept = d >= 0
    assert bool(chosen.gather(1, torch.where(kept, d // rows, 0))[kept].all()) and bool((d % rows < C)[kept].all())
    assert torch.equal(inverse.long()[d[kept]], torch.arange(T * k, device=DEV).view(T, k)[kept])
    assert int((inverse >= 0).sum()) == int(kept.sum()) == int(counts.sum())
    # gradients; the gates' upstream gradient is a function of the gate, so that the order among equal ones does not matter
    da = torch.full((), 0.7, device=DEV)
    for use_gate, use_aux in ((True, True), (True, False), (False, True)):
        outs = [(gate, gate.detach() * 3 + 1, dense64, dense64.detach() * 3 + 1)] * use_gate + [(aux, da, aux64, da.double())] * use_aux
        got = torch.autograd.grad([o[0] for o in outs], z, [o[1] for o in outs], retain_graph=True)[0]
        want = torch.autograd.grad([o[2] for o in outs], z64, [o[3] for o in outs], retain_graph=True)[0]
        # with one expert, or all of them chosen, gradients vanish but for fp32 cancellation of terms of order one per token
        noise = 1e-6 * T ** 0.5 if use_gate else 1e-6
        assert float((got.double() - want).norm()) <= 2.0 ** -8 * float(want.norm()) + noise, (use_gate, use_aux)


def test_route_nan_and_infinities():
    """A NaN (or +inf) makes a row's probabilities NaN: the first k experts; -inf experts are not chosen while others are
    left."""
    inf, nan = float("inf"), float("nan")
    z = torch.tensor([[1.0, nan, 0.0, 2.0], [1.0, inf, 0.0, 2.0], [-inf, 1.0, 2.0, -inf], [0.0] * 4], device=DEV).bfloat16()
    gate, aux, dest, inverse, counts, stats = _route(z, 2, 8, 64)
    experts = (dest.view(4, 2) // 64).sort(-1)[0].tolist()
    assert experts == [[0, 1], [0, 1], [1, 2], [0, 1]]
    assert bool(gate[:2].isnan().all()) and bool(torch.isfinite(gate[2:]).all())
    assert stats[:4].tolist() == [3.0, 4.0, 1.0, 0.0]


@pytest.fixture
def _grid():
    import torch.distributed as dist

    from axonn_b200 import axonn as ax

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    if not ax.is_initialized:
        ax.init(G_inter=1, G_data=1, G_intra_r=1, G_intra_c=1, G_intra_d=1)


@pytest.mark.parametrize("E", [4, 8])
@pytest.mark.parametrize("cast", [torch.float16, torch.float32])
def test_router_under_autocast(_grid, E, cast):
    """With 4 experts the router's product has autocast's type and the routing takes it as it is; with 8 it is bf16.  The
    same experts and balance loss as softmax and top-k of those logits, and its gradient by the router (2^-7)."""
    from axonn_b200 import ops
    from axonn_b200.parallel.moe import ExpertParallelMoE, route_top_k

    torch.manual_seed(E)
    layer = ExpertParallelMoE(64, 64, n_experts=E, top_k=2, dtype=torch.bfloat16, init_std=0.3)
    x = torch.randn(300, 64, device=DEV, dtype=torch.bfloat16)
    with torch.autocast("cuda", dtype=cast):
        logits = ops.linear(x, layer.router)
        idx, aux = (route_top_k(logits, 2, 10 ** 6)[i] for i in (0, 4))
        layer(x)
    assert logits.dtype == (cast if E == 4 else torch.bfloat16)
    assert torch.equal(layer.last_assignments_per_expert, torch.bincount(idx.reshape(-1), minlength=E).float())
    assert abs(float(layer.last_aux_loss.detach()) - float(aux.detach())) <= 1e-5 * float(aux.detach())
    if E == 8:                                       # with 4 the backward of the product refuses two types
        (got,), (want,) = (torch.autograd.grad(v, layer.router) for v in (layer.last_aux_loss, aux))
        assert float((got - want).float().norm()) <= 2.0 ** -7 * float(want.float().norm())


def test_statistics_belong_to_the_caller(_grid):
    """Sums over ranks or steps are made in place, before the backward too, and do not reach the gradient."""
    from axonn_b200.parallel.moe import ExpertParallelMoE

    torch.manual_seed(0)
    layer = ExpertParallelMoE(64, 64, n_experts=8, top_k=2, dtype=torch.bfloat16, init_std=0.3)
    x = torch.randn(300, 64, device=DEV, dtype=torch.bfloat16)
    grads = []
    for add in (0, 1000):
        loss = layer(x).float().square().sum() + layer.last_aux_loss
        for t in (layer.last_assignments_per_expert, layer.last_dropped_per_expert, layer.last_drop_fraction):
            t += add
        grads.append(torch.autograd.grad(loss, layer.router)[0])
    assert torch.equal(*grads)
