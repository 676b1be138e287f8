"""Batched products with one segment per problem: only the tile rows with data are dealt out to the CTA pairs."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EDGES = [0, 1, 255, 256, 257, 512, 513, 800]


@pytest.mark.parametrize("counts", [
    EDGES * 2,                              # several waves, the last one in halves of tiles
    [0, 0, 0],                              # nothing but zeros to store
    [800],
    [3] * 127 + [800],                      # the longest list
    [3] * 128 + [800],                      # one more: tiles without data are skipped one by one
], ids=["edges", "empty", "full", "list128", "skip129"])
def test_rows_without_data(counts):
    from axonn_b200.ops import _lib, gemm

    E, rows, N, K = len(counts), 800, 520, 192
    torch.manual_seed(E)
    seg = torch.tensor(counts, dtype=torch.int32, device=DEV).view(E, 1)
    live = torch.arange(rows, device=DEV)[None, :] < seg.long()
    a = torch.randn(E, rows, K, device=DEV).bfloat16() * live[:, :, None]
    b = torch.randn(E, N, K, device=DEV).bfloat16()
    bt = b.transpose(1, 2).contiguous()
    for _ in range(2):                      # results land in memory full of NaN: what no tile writes shows
        junk = torch.full((E, rows, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        del junk
        y = gemm.bmm_nt(a, b, seg=seg, seg_rows=rows)
        junk = torch.full((E, rows, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        del junk
        z = gemm.bmm_nn(a, bt, seg=seg, seg_rows=rows)
        for e in {0, 1, 2, 3, E // 2, E - 2, E - 1} & set(range(E)):
            want = a[e].double() @ b[e].double().t()
            # one rounding to bf16 of an fp32 sum
            assert float((y[e].double() - want).norm()) <= 2.0 ** -8 * float(want.norm())
            assert float((z[e].double() - want).norm()) <= 2.0 ** -8 * float(want.norm())
        assert bool((y[~live] == 0).all()) and bool((z[~live] == 0).all())
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
