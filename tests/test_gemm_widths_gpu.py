"""Products on CTA pairs whose tiles are not 256 columns wide, and those whose operands change roles."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# M, N, K: ragged tokens and odd ends on both sides of the rule for the width, one and several waves, halved last waves, output
# rows off 32 bytes (N % 16 == 8), tiles of 64 and 128 columns for the small ones
SHAPES = [(777, 6144, 256), (777, 3072, 1024), (769, 4104, 264), (1300, 2056, 328), (300, 8200, 136), (2500, 1032, 512), (513, 14344, 72),
          (3000, 1024, 200), (1024, 3080, 128), (1, 264, 64), (65, 8, 1024), (308, 1000, 256), (1000, 1024, 1024), (129, 4096, 520),
          (1531, 1032, 264), (640, 1000, 8),
          # long enough along K for exchanged roles to pay
          (777, 6144, 1032), (769, 4104, 1032), (300, 8200, 1032), (2500, 1032, 1032), (1300, 2056, 2056)]


def _check(got, want, bound):
    assert float((got.double() - want).norm()) <= bound * float(want.norm())
    # every element: K products of unit variance, one rounding each of sum and (GELU) argument
    assert float((got.double() - want).abs().max()) <= 4 * bound * float(want.abs().max())


def _guarded(M, N, dtype):
    """An M x N tensor of NaN between two rows of a mark."""
    buf = torch.full((M + 2, N), float("nan"), dtype=dtype, device=DEV)
    buf[0], buf[-1] = 3.0, 3.0
    return buf, buf[1:-1]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_widths(M, N, K, dtype):
    from axonn_b200 import ops
    from axonn_b200.ops import _lib, gemm

    torch.manual_seed(M + N + K)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    a, b, bias = (torch.randn(s, device=DEV).to(dtype) for s in ((M, K), (N, K), (N,)))
    bt = b.t().contiguous()
    want = a.double() @ b.double().t()
    for fn, x, kw, ref in (
            (gemm.matmul_nt, b, {}, want),
            (gemm.matmul_nt, b, dict(bias=bias, epilogue=ops.EPI_BIAS), want + bias.double()),
            (gemm.matmul_nn, bt, {}, want)):
        buf, out = _guarded(M, N, dtype)
        fn(a, x, out=out, **kw)
        _check(out, ref, eps)
        assert bool((buf[0] == 3).all()) and bool((buf[-1] == 3).all())
    (buf, out), (abuf, aux) = _guarded(M, N, dtype), _guarded(M, N, dtype)
    gemm.matmul_nt(a, b, out=out, bias=bias, epilogue=ops.EPI_BIAS_GELU, aux=aux)
    _check(aux, want + bias.double(), eps)
    _check(out, torch.nn.functional.gelu(want + bias.double(), approximate="tanh"), 2 * eps)
    assert bool((buf[[0, -1]] == 3).all()) and bool((abuf[[0, -1]] == 3).all())
    # an activation in layout 1, which the launcher takes too
    buf, out = _guarded(M, N, dtype)
    gemm._launch(1, a, bt, M, N, K, out, bias, ops.EPI_BIAS_GELU)
    _check(out, torch.nn.functional.gelu(want + bias.double(), approximate="tanh"), 2 * eps)
    # fp32 results and accumulation keep the roles of the operands
    _check(gemm.matmul_nt(a, b, out_dtype=torch.float32), want, 1e-5)
    acc = torch.ones(M, N, dtype=torch.float32, device=DEV)
    gemm.matmul_nt(a, b, out=acc, accumulate=True)
    _check(acc, want + 1, 1e-5)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
