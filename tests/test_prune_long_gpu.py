"""Gradient pruning of long tensors, whose passes run from either end."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
N = 1 << 25                       # the shortest 16-bit tensor that counts as long; fp32 from half of it


def _make(kind, n, dtype):
    g = torch.randn(n, device=DEV)
    if kind == "rows":            # scales that differ from row to row and repeat with a period
        g *= torch.logspace(-6, 2, 4096, device=DEV).repeat(n // 4096 + 1)[:n]
    elif kind == "spike":         # a few large values
        g *= 1e-3
        g[5234567:5234567 + 2000] = 50.0
    elif kind == "ties":
        g = g.round()
    elif kind == "zeros":
        g[: n - n // 3] = 0
    elif kind == "heavy":         # tails over many octaves
        g = g * torch.randn(n, device=DEV).mul_(3).exp()
    elif kind == "nan":
        g[::1003] = float("nan")
        g[5] = float("inf")
    elif kind == "large":         # a threshold among the largest finite values
        g = g.abs().clamp_max(1).mul_(60000.0)
    return g.to(dtype)


def _check(g, keep):
    from axonn_b200 import ops

    bits = (g.view(torch.int32) & 0x7FFFFFFF) if g.dtype == torch.float32 else (g.view(torch.int16).int() & 0x7FFF)
    k = max(1, int(round(g.numel() * keep)))
    limit = bits.sort(descending=True)[0][k - 1]
    as_int = torch.int32 if g.dtype == torch.float32 else torch.int16
    want = torch.where(bits >= limit, g.view(as_int), torch.zeros_like(g.view(as_int)))
    assert torch.equal(ops.prune_topk_(g, keep).view(as_int), want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("kind,keep", [("normal", 0.1), ("normal", 0.999), ("normal", 1e-7), ("rows", 0.01), ("spike", 3e-4),
                                       ("ties", 0.3), ("zeros", 0.5), ("heavy", 0.001), ("nan", 0.1), ("large", 0.01)])
def test_prune_long(dtype, kind, keep):
    """Exactly the entries whose magnitude bits reach those of the k-th largest, for every distribution."""
    torch.manual_seed(1)
    _check(_make(kind, N + 13, dtype), keep)


@pytest.mark.parametrize("n,at", [(N - 1, 0), (N, 0), (N + 1, 0), (N + 7, 4), (2 * N + 1, 8), (148 * 1024 * 8 * 32, 0)])
def test_prune_lengths_and_offsets(n, at):
    """Lengths around the rule, a tensor 8 bytes off the alignment that the vector loads need, one 16 bytes into its buffer."""
    buf = torch.empty(n + 16, device=DEV, dtype=torch.bfloat16)
    g = buf[at:at + n].copy_(torch.randn(n, device=DEV))
    _check(g, 0.2)


@pytest.mark.parametrize("n", [100 << 20, (100 << 20) + 4])
def test_prune_fp32_around_the_upper_length(n):
    """fp32 tensors go through the passes from either end up to a length, and from the beginning past it."""
    torch.manual_seed(1)
    _check(torch.randn(n, device=DEV), 0.1)
