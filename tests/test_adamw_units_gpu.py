"""AdamW over lists whose work is cut into quarters, eighths and sixteenths of a chunk of 65536 elements."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("sizes", [
    [1, 7, 4095, 4096, 4097, 65535, 65536, 65537, 200003],            # few tensors: sixteenths
    [8191, 8192, 8193, 65536] * 12,                                   # many of a chunk at most: quarters
    [140001] * 600,                                                   # 1800 chunks: eighths
], ids=["sixteenths", "quarters", "eighths"])
def test_every_element_once(sizes):
    from axonn_b200.optim import FusedAdamW
    from axonn_b200.ops import _lib

    torch.manual_seed(len(sizes))
    ps = [torch.nn.Parameter(torch.randn(n, device=DEV).bfloat16()) for n in sizes]
    for p in ps:
        p.grad = torch.randn(p.shape, device=DEV).bfloat16()
    before = [p.detach().double() for p in ps]
    opt = FusedAdamW(ps, lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    opt.step()
    for p, w in zip(ps, before):
        g, st = p.grad.double(), opt.state[p]
        m, v = 0.1 * g, 0.05 * g * g
        want = w * (1 - 1e-2 * 0.1) - 1e-2 * (m / 0.1) / ((v / 0.05).sqrt() + 1e-8)
        # fp32 arithmetic of half a dozen roundings, the update at most 1e-2
        assert float((st["master"].double() - want).abs().max()) < 4e-6
        assert float((st["exp_avg"].double() - m).abs().max()) < 1e-6 and float((st["exp_avg_sq"].double() - v).abs().max()) < 4e-6
        assert torch.equal(p.detach(), st["master"].bfloat16())
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
