"""Gradient clipping whose norm and factor come from the norm kernel, against 64-bit arithmetic."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module", autouse=True)
def _grid():
    import torch.distributed as dist

    from axonn_b200 import axonn as ax

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    if not ax.is_initialized:
        ax.init(G_inter=1, G_data=1, G_intra_r=1, G_intra_c=1, G_intra_d=1)


@pytest.mark.parametrize("sizes", [(1,), (7, 0, 65536, 65537), (3_000_001, 12, 900_000), (17,) * 1100])
@pytest.mark.parametrize("max_norm", [1e-3, 1e9, float("inf"), 0.0])
@pytest.mark.parametrize("grouped", [False, True])
def test_clip_factor(sizes, max_norm, grouped):
    """One block and many, tensors without elements, a limit above and below the norm, parameters in groups of one rank
    and without a group.  fp32 sums of n squares: relative error of the norm below 1e-5; scaled gradients are rounded
    once to their type (2^-9 for bf16)."""
    from axonn_b200 import axonn as ax
    from axonn_b200.intra_layer import clip_grad_norm_

    torch.manual_seed(len(sizes))
    dts = [torch.bfloat16, torch.float32, torch.float16]
    ps = []
    for i, n in enumerate(sizes):
        p = torch.nn.Parameter(torch.zeros(n, device=DEV, dtype=dts[i % 3]))
        p.grad = torch.randn(n, device=DEV).to(dts[i % 3])
        if grouped and i % 2:
            p.is_tensor_parallel = True
            p.process_group_for_norm_reduction = ax.comm_handle.inner_intra_layer_parallel_group
        ps.append(p)
    before = [p.grad.double() for p in ps]
    norm = torch.stack([g.pow(2).sum() for g in before]).sum().sqrt()
    got = clip_grad_norm_(ps, max_norm)
    assert got.shape == () and got.dtype == torch.float32
    assert abs(float(got) - float(norm)) <= 1e-5 * float(norm)
    f = min(1.0, max_norm / (float(norm) + 1e-6))
    for p, g in zip(ps, before):
        if g.numel():
            tol = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10, torch.float32: 2e-5}[p.dtype]
            # fp16 gradients scaled into the subnormal range keep an absolute spacing of 2^-24
            assert float((p.grad.double() - g * f).abs().max()) <= tol * float((g * f).abs().max()) + 2.0 ** -24


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_clip_factor_nonfinite(bad):
    """A NaN reaches every gradient, an infinite norm makes the factor zero: what the tensor operations gave."""
    from axonn_b200.intra_layer import clip_grad_norm_

    p = torch.nn.Parameter(torch.zeros(5, device=DEV))
    p.grad = torch.tensor([1.0, 2.0, bad, 4.0, 5.0], device=DEV)
    want = p.grad * torch.clamp(1.0 / (p.grad.norm() + 1e-6), max=1.0)
    total = clip_grad_norm_([p], 1.0)
    assert torch.equal(p.grad.isnan(), want.isnan()) and torch.equal(p.grad.nan_to_num(), want.nan_to_num())
    assert not bool(torch.isfinite(total))
    p.grad = torch.full((5,), bad, device=DEV)
    with pytest.raises(RuntimeError, match="non-finite"):
        clip_grad_norm_([p], 1.0, error_if_nonfinite=True)
