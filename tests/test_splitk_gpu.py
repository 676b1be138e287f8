"""Split-K products: rows around the sizes of a ring stage, every epilogue, and launches that overlap their predecessors."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF16 = torch.bfloat16


def _close(got, want, bound):
    assert float((got.double() - want).norm()) <= bound * float(want.norm())


@pytest.mark.parametrize("M", [1, 8, 31, 32, 33, 64, 65, 96, 97, 128, 129, 300])
@pytest.mark.parametrize("N,K", [(136, 1024), (1024, 4096), (264, 520), (4104, 2048), (16384, 512)])
def test_rows(M, N, K):
    from axonn_b200 import ops
    from axonn_b200.ops import _lib, gemm

    torch.manual_seed(M + N + K)
    eps = 2.0 ** -8                                # one rounding of an fp32 sum to bf16
    a, b = torch.randn(M, K, device=DEV).to(BF16), torch.randn(N, K, device=DEV).to(BF16)
    bias = torch.randn(N + 1, device=DEV).to(BF16)[1:]             # off 4 bytes
    want = a.double() @ b.double().t()
    buf = torch.full((M + 2, N), float("nan"), dtype=BF16, device=DEV)
    buf[0], buf[-1] = 3.0, 3.0
    out, aux = buf[1:-1], torch.full((M, N), float("nan"), dtype=BF16, device=DEV)
    _close(gemm.matmul_nt(a, b, out=out), want, eps)
    _close(gemm.matmul_nt(a, b, out=out, bias=bias, epilogue=ops.EPI_BIAS), want + bias.double(), eps)
    gemm.matmul_nt(a, b, out=out, bias=bias, epilogue=ops.EPI_BIAS_GELU, aux=aux)
    _close(aux, want + bias.double(), eps)
    _close(out, torch.nn.functional.gelu(want + bias.double(), approximate="tanh"), 2 * eps)
    assert bool((buf[[0, -1]] == 3).all())
    _close(gemm.matmul_nn(a, b.t().contiguous()), want, eps)
    acc = torch.ones(M, N, device=DEV)
    _close(gemm.matmul_nt(a, b, out=acc, accumulate=True), want + 1, 1e-5)
    acc = out.copy_(torch.ones_like(out))
    _close(gemm.matmul_nt(a, b, out=acc, accumulate=True), want + 1, eps)
    if M % 8 == 0:
        _close(gemm.matmul_tn(a.t().contiguous(), b.t().contiguous()), want, eps)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0


def test_overlapping_launches():
    """Each product needs what the kernel just before it in the stream has written - as its rows, as its weights, as its
    bias, or in the place of its output - and a replay in a graph does the same."""
    from axonn_b200 import ops
    from axonn_b200.ops import gemm

    torch.manual_seed(0)
    M, H = 24, 1024
    x = torch.randn(M, H, device=DEV).to(BF16)
    w = [(torch.randn(H, H, device=DEV) / 32).to(BF16) for _ in range(3)]
    bias = torch.randn(H, device=DEV).to(BF16)
    gathered = torch.empty(H, H, device=DEV, dtype=BF16)

    def chain(sync):
        y, b = x.clone(), bias.clone()
        ws = [t.clone() for t in w]
        outs = []
        for i in range(6):
            y = gemm.matmul_nt(y, ws[i % 3], bias=b, epilogue=ops.EPI_BIAS_GELU)         # rows from the last product
            sync()
            gemm.matmul_nt(ws[0], ws[1], out=gathered)                                  # weights from a product
            sync()
            y = gemm.matmul_nt(y, gathered)
            sync()
            ws[i % 3].mul_(0.5)                                                         # weights written by another library's kernel
            sync()
            y = gemm.matmul_nt(y, ws[i % 3])
            sync()
            b.copy_(y[0])
            sync()
            z = gemm.matmul_nt(y, ws[2], bias=b, epilogue=ops.EPI_BIAS)
            sync()
            gemm.matmul_nt(x, ws[2], out=y)                                             # over the last product's operand
            sync()
            y = gemm.matmul_nt(z, ws[1])
            y = (y.float() / y.float().std()).to(BF16)
            outs.append(torch.cat([y, z]))
        return torch.stack(outs)
    want = chain(torch.cuda.synchronize)
    for _ in range(20):
        assert torch.equal(chain(lambda: None), want)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = chain(lambda: None)
    for _ in range(5):
        got.zero_()
        g.replay()
        assert torch.equal(got, want)


def test_deadline_starts_after_the_predecessor():
    """A product that is launched while its predecessor still runs does not count that one's time against its own waits: 15 ms of
    a product held to two SMs, before one with a deadline of 3 ms."""
    from axonn_b200.ops import _lib, gemm

    torch.manual_seed(1)
    long_a, long_b = (torch.randn(4096, 8192, device=DEV).to(BF16) for _ in range(2))
    a, b = torch.randn(24, 1024, device=DEV).to(BF16), torch.randn(1024, 1024, device=DEV).to(BF16)
    want = gemm.matmul_nt(a, b)
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    L = _lib.lib()
    torch.cuda.synchronize()
    start.record()
    try:
        L.axb_gemm_set_max_ctas(2)
        gemm.matmul_nt(long_a, long_b)
        L.axb_gemm_set_max_ctas(0)
        _lib.set_wait_timeout_ms(3)
        got = gemm.matmul_nt(a, b)
    finally:
        L.axb_gemm_set_max_ctas(0)
        _lib.set_wait_timeout_ms(120000)
    end.record()
    torch.cuda.synchronize()
    assert start.elapsed_time(end) > 6
    assert _lib.device_status() == 0 and torch.equal(got, want)
