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


def _synchronised(monkeypatch, run):
    """``run()`` with every launch made from Python, and waited for."""
    from axonn_b200.ops import _lib

    def waiting(status, what, check=_lib.check):
        check(status, what)
        torch.cuda.synchronize()
    with monkeypatch.context() as m:
        m.setattr(_lib, "_HOST", None)
        m.setattr(_lib, "check", waiting)
        return run()


@pytest.mark.parametrize("llama", [False, True])
@pytest.mark.parametrize("batch,seq,hidden", [(1, 24, 256), (2, 300, 512), (3, 512, 1024)])
def test_blocks(batch, seq, hidden, llama, monkeypatch):
    """Forward and backward of blocks in a row - norms, products, rotary embedding, attention, column sums -, each layer's
    parameters written just before it is called."""
    from axonn_b200.models.blocks import TransformerBlock

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

    want = _synchronised(monkeypatch, run)
    for _ in range(10):
        for a, b in zip(run(), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, BF16, torch.float16])
@pytest.mark.parametrize("n", [1001, 1 << 20, (1 << 24) + 8, (1 << 25) + 4096])
def test_pruning_what_an_overlapped_launch_has_written(n, dtype, monkeypatch):
    """The later passes load the gradient before they wait: it comes from a kernel that lets the next launch begin early, directly
    in front of the first pass."""
    from axonn_b200 import ops

    torch.manual_seed(n)
    base, scale = torch.randn(n, device=DEV).to(dtype), torch.full((), 0.5, device=DEV)
    g = torch.empty_like(base)

    def run():
        outs = []
        for keep in (0.1, 0.5):
            g.copy_(base)
            ops.multi_tensor_scale_([g], scale)
            ops.prune_topk_(g, keep)
            ops.multi_tensor_scale_([g], scale)
            ops.prune_topk_(g, keep / 2)
            outs.append(g.clone())
        return outs
    want = _synchronised(monkeypatch, run)
    assert all(0 < int((w != 0).sum()) < n for w in want)
    for _ in range(5):
        for a, b in zip(run(), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("sizes", [[70000, 300001, 9], [4096] * 200, [1 << 20] * 9], ids=["few", "many small", "long"])
def test_optimizer_steps(sizes, monkeypatch):
    """Gradients scaled by a kernel of the same kind, norm and clipping factor, scale, status copy and AdamW, four times in a row.  The
    gradients are small powers of two times integers: their squares add up exactly, in any order."""
    from axonn_b200 import ops
    from axonn_b200.intra_layer import clip_grad_norm_
    from axonn_b200.optim import FusedAdamW

    torch.manual_seed(len(sizes))
    start = [torch.randn(n, device=DEV).to(BF16) for n in sizes]
    grads = [torch.randint(-1, 2, (n,), device=DEV).to(BF16) for n in sizes]
    half = torch.full((), 0.5, device=DEV)

    def run():
        ps = [torch.nn.Parameter(p.clone()) for p in start]
        opt = FusedAdamW(ps, lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
        totals = []
        for p in ps:
            p.grad = torch.empty_like(p)
        for i in range(4):
            for p, g in zip(ps, grads):
                p.grad.copy_(g.roll(i))
            ops.multi_tensor_scale_([p.grad for p in ps], half)
            totals.append(clip_grad_norm_(ps, 1.0))
            opt.step()
        return totals + [t for p in ps for t in (p.detach(), p.grad, *(opt.state[p][k] for k in ("master", "exp_avg", "exp_avg_sq")))]
    want = _synchronised(monkeypatch, run)
    assert float(want[0]) == pytest.approx(0.5 * sum(float(g.float().pow(2).sum()) for g in grads) ** 0.5, rel=1e-6)
    for _ in range(5):
        for a, b in zip(run(), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("tokens,hidden,ffn,experts", [(77, 256, 512, 4), (1500, 512, 1024, 8)])
def test_expert_layer(tokens, hidden, ffn, experts, monkeypatch):
    """Forward and backward of an expert layer, twice in a row: routing, permutations, products over the tile rows with data."""
    from axonn_b200.parallel.moe import ExpertParallelMoE

    torch.manual_seed(tokens)
    layer = ExpertParallelMoE(hidden, ffn, n_experts=experts, top_k=2, dtype=BF16)
    with torch.no_grad():
        for p in layer.parameters():
            p.copy_(torch.randn_like(p) * 0.05)
    x0, dy = (torch.randn(1, tokens, hidden, device=DEV).to(BF16) for _ in range(2))

    def run():
        x = x0.clone().requires_grad_(True)
        y = layer(x)
        z = layer((y.float() / y.float().std()).to(BF16))
        return [y.detach(), z.detach(), *torch.autograd.grad([z, layer.last_aux_loss], [x, *layer.parameters()], [dy, torch.ones((), device=DEV)])]
    want = _synchronised(monkeypatch, run)
    for _ in range(5):
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
    y.mul_(1.0)
    side, (start, done, behind) = torch.cuda.Stream(), (torch.cuda.Event(enable_timing=True) for _ in range(3))
    L = _lib.lib()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):                      # kernels loaded, the stream's memory allocated: neither waits for the GPU below
        gemm.matmul_nt(a, b)
        want = ops.column_sum(x)
    torch.cuda.synchronize()
    torch.cuda._sleep(2 * 10 ** 8)                     # 0.1 s: everything is launched before anything runs
    start.record()
    side.wait_event(start)
    with torch.cuda.stream(side):
        try:
            L.axb_gemm_set_max_ctas(2)
            gemm.matmul_nt(a, b)                       # 15 ms
            got = ops.column_sum(x)
        finally:
            L.axb_gemm_set_max_ctas(0)
        behind.record()
    for _ in range(20):
        y.mul_(1.0)
    done.record()
    torch.cuda.synchronize()
    assert start.elapsed_time(behind) > 6 and start.elapsed_time(done) < start.elapsed_time(behind) / 2
    assert torch.equal(got, want)
