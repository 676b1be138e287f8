"""Kernels that are launched while their predecessor still runs: the same bits as with a synchronisation after every layer."""

import os
import shutil
import subprocess

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


@pytest.mark.parametrize("llama", [False, True])
@pytest.mark.parametrize("batch,seq,hidden", [(1, 24, 256), (2, 300, 512), (3, 512, 1024)])
def test_blocks(batch, seq, hidden, llama, monkeypatch):
    """Forward and backward of blocks in a row - norms, products, rotary embedding, attention, column sums -, each layer's
    parameters written just before it is called."""
    from axonn_b200.models.blocks import TransformerBlock
    from axonn_b200.ops import _lib

    torch.manual_seed(seq)
    blk = TransformerBlock(hidden, hidden // 64, 2 * hidden, n_kv_heads=hidden // 128 if llama else None, activation="swiglu" if llama else "gelu",
                           rms=llama, bias=not llama, rope_theta=1e4 if llama else None, max_seq=512, dtype=BF16)
    with torch.no_grad():
        for p in blk.parameters():
            p.copy_(torch.randn_like(p) * (0.5 if p.dim() == 1 and p.numel() <= 3 * hidden else 0.05))
    base = [p.detach().clone() for p in blk.parameters()]
    x0, dy = (torch.randn(batch, seq, hidden, device=DEV).to(BF16) for _ in range(2))

    def run():
        outs = []
        x = x0.clone()
        for i in range(4):
            with torch.no_grad():
                for p, b in zip(blk.parameters(), base):
                    torch.mul(b, 1 - i / 8, out=p)
                x = blk(x)
                x = (x.float() / x.float().std()).to(BF16)
            outs.append(x)
        a = x0.clone().requires_grad_(True)
        y = blk(a)
        return outs + [y.detach(), *torch.autograd.grad(y, [a, *blk.parameters()], dy)]

    def waiting(status, what, check=_lib.check):
        check(status, what)
        torch.cuda.synchronize()
    with monkeypatch.context() as m:                 # every launch from Python, and waited for
        m.setattr(_lib, "_HOST", None)
        m.setattr(_lib, "check", waiting)
        want = run()
    for _ in range(10):
        for a, b in zip(run(), want):
            assert torch.equal(a, b)


_REFUSED_LAUNCH = """
#include "axonn_b200.h"
#include "common.cuh"
__global__ void kernel(int) {}
static int launch() { AXB_CUDA(axb::pdl_launch(kernel, dim3(0), dim3(32), 0, nullptr, 1)); return 0; }
int main() { return launch() == -1 && axb_last_error()[0] != 0 && cudaPeekAtLastError() == cudaSuccess ? 0 : 1; }
"""


@pytest.mark.skipif(not shutil.which("nvcc"), reason="needs nvcc")
def test_a_refused_launch_is_reported_once(tmp_path):
    """The runtime refuses an empty grid: the launcher returns that, and the runtime has nothing left for the next launch to find."""
    import axonn_b200

    csrc = os.path.join(os.path.dirname(axonn_b200.__file__), "csrc")
    (tmp_path / "launch.cu").write_text(_REFUSED_LAUNCH)
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", csrc, str(tmp_path / "launch.cu"),
                    os.path.join(csrc, "common.cu"), "-o", str(tmp_path / "launch")], check=True)
    subprocess.run([str(tmp_path / "launch")], check=True)


def test_a_cap_leaves_its_sms_to_the_other_stream():
    """A column sum behind a product that is held to a few SMs does not wait on the others: what another stream launches has them."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib, gemm

    a, b = (torch.randn(4096, 8192, device=DEV).to(BF16) for _ in range(2))
    x, y = torch.randn(65536, 4096, device=DEV).to(BF16), torch.randn(1 << 24, device=DEV)
    want = ops.column_sum(x)
    y.mul_(1.0)
    side, behind = torch.cuda.Stream(), torch.cuda.Event()
    L = _lib.lib()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        try:
            L.axb_gemm_set_max_ctas(2)
            gemm.matmul_nt(a, b)                       # 15 ms
            got = ops.column_sum(x)
        finally:
            L.axb_gemm_set_max_ctas(0)
        behind.record()
    done = torch.cuda.Event()
    for _ in range(20):
        y.mul_(1.0)
    done.record()
    done.synchronize()
    assert not behind.query()                            # the product is still at work
    torch.cuda.synchronize()
    assert torch.equal(got, want)
