"""The native host paths (csrc/host_ops.cpp) against the Python code that launches the same kernels: same bits over all forms
that either takes, refused where it was refused, seen by everything that looks at an operation."""

import gc
import threading
import time

import pytest
import torch
import torch.distributed as dist

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16 = torch.bfloat16


@pytest.fixture(scope="module", autouse=True)
def _grid():
    from axonn_b200 import axonn as ax
    from axonn_b200.ops import _lib

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    if not ax.is_initialized:
        ax.init(G_inter=1, G_data=1, G_intra_r=1, G_intra_c=1, G_intra_d=1)
    assert _lib.host() is not None


def _python(monkeypatch, fn):
    from axonn_b200.ops import _lib

    with monkeypatch.context() as m:
        m.setattr(_lib, "_HOST", None)
        return fn()


def _forms(shape, dtype):
    base = torch.randn(torch.Size(shape).numel() + 8, device=DEV).to(dtype)
    wide = torch.randn(*shape[:-1], 2 * shape[-1], device=DEV).to(dtype)
    yield base[:-8].view(shape)
    yield base[8:].view(shape)                                    # 16 bytes (fp32: 32) into a buffer
    yield wide[..., :shape[-1]]                                   # rows with gaps
    yield base[:1].expand(shape)


@pytest.mark.parametrize("dtype", [BF16, torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(8,), (1, 16), (3, 5, 264), (300, 128), (0, 16)])
@pytest.mark.parametrize("rms,residual,bias", [(True, False, False), (False, True, True), (False, False, True), (True, True, False),
                                               (False, False, False)])
def test_norms(shape, dtype, rms, residual, bias, monkeypatch):
    from axonn_b200 import ops

    torch.manual_seed(1)
    gamma, beta = ((torch.randn(shape[-1], device=DEV) + 1).to(dtype) for _ in range(2))
    for form in range(4):
        x0, d0, dy, dh = (list(_forms(shape, dtype))[f] for f in (form, (form + 1) % 4, (form + 2) % 4, (form + 3) % 4))

        def both(grads):
            x, d, g, b = (t.detach().requires_grad_(r) for t, r in zip((x0, d0, gamma, beta), grads))
            b = b if bias else None
            if residual:
                out = ops.add_rms_norm(x, d, g) if rms else ops.add_layer_norm(x, d, g, b)
            else:
                out = (ops.rms_norm(x, g) if rms else ops.layer_norm(x, g, b),)
            leaves = [t for t in (x, d if residual else None, g, b) if t is not None and t.requires_grad]
            res = [o.detach() for o in out]
            assert all(o.requires_grad == bool(leaves) for o in out)
            if leaves and x.numel():
                res += torch.autograd.grad(out, leaves, [dh, dy][-len(out):], retain_graph=True)
                res += torch.autograd.grad(out[-1], leaves, dy)      # the residual's gradient missing
            return res
        for grads in ([True] * 4, [False] * 4, [False, True, False, True], [True, False, True, False]):
            got, want = both(grads), _python(monkeypatch, lambda: both(grads))
            assert len(got) == len(want)
            for a, w in zip(got, want):
                assert a.shape == w.shape and a.dtype == w.dtype and torch.equal(a, w)


def test_norms_are_seen(monkeypatch):
    """Saved-tensor hooks in another layout, a second backward, in-place writes, function transforms, streams and threads."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib

    x = torch.randn(40, 256, device=DEV, dtype=BF16, requires_grad=True)
    d, g = torch.randn_like(x), torch.ones(256, device=DEV, dtype=BF16, requires_grad=True)
    dy = torch.randn_like(x)
    (want,) = torch.autograd.grad(ops.add_rms_norm(x, d, g)[1], x, dy)
    turned = lambda t: t.t().contiguous().t() if t.dim() == 2 else t  # noqa: E731
    with torch.autograd.graph.saved_tensors_hooks(lambda t: turned(t.detach()), lambda t: t):
        y = ops.add_rms_norm(x, d, g)[1]
    assert torch.equal(torch.autograd.grad(y, x, dy)[0], want)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: 1 / 0, lambda t: t), pytest.raises(ZeroDivisionError):
        ops.add_rms_norm(x, d, g)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: 1 / 0):
        y = ops.add_rms_norm(x, d, g)[1]
    with pytest.raises(ZeroDivisionError):
        torch.autograd.grad(y, x, dy)
    with torch.autograd.detect_anomaly(check_nan=False):
        assert torch.equal(torch.autograd.grad(ops.add_rms_norm(x, d, g)[1], x, dy)[0], want)
    y = ops.rms_norm(x, g)
    torch.autograd.grad(y, x, dy)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(y, x, dy)
    h, y = ops.add_rms_norm(x, d, g)
    h.add_(1)                                                         # saved for the backward
    with pytest.raises(RuntimeError):
        torch.autograd.grad(y, x, dy)
    y = ops.rms_norm(x, g)
    y.add_(1)                                                         # not saved
    torch.autograd.grad(y, x, dy)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: ops.rms_norm(t, g).sum())(x.detach())
    with torch.inference_mode():
        z = ops.rms_norm(x, g)
    assert z.is_inference() and torch.equal(z, ops.rms_norm(x, g).detach())
    with pytest.raises(RuntimeError):
        ops.rms_norm(z, g)                                            # an inference tensor cannot be saved
    before = _lib.launch_count
    torch.autograd.grad(ops.rms_norm(x, g), x, dy)
    counted = _lib.launch_count - before
    before = _lib.launch_count
    _python(monkeypatch, lambda: None)
    got = []

    def work():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            a = x.detach().clone().requires_grad_(True)
            got.append(torch.autograd.grad(ops.add_rms_norm(a, d, g)[1], a, dy)[0])
        s.synchronize()
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work) for _ in range(4)]
    [t.start() for t in threads], [t.join() for t in threads]
    assert counted == 3 and _lib.launch_count - before == 12 and len(got) == 4 and all(torch.equal(a, want) for a in got)
    _lib.reset_launch_count()
    assert _lib.launch_count == 0


@pytest.mark.parametrize("dtype", [BF16, torch.float16, torch.float32])
@pytest.mark.parametrize("native", [False, True])
@pytest.mark.parametrize("residual", [False, True])
def test_norms_of_views_at_any_offset(residual, native, dtype, monkeypatch):
    """Dense views that do not begin on 16 bytes - input, residual, gain, bias, incoming gradients - are what their copies are; the
    launchers themselves refuse such addresses."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib

    if not native:
        monkeypatch.setattr(_lib, "_HOST", None)
    shapes = [(6, 264), (6, 264), (264,), (264,), (6, 264), (6, 264)]
    off = [torch.randn(1 + torch.Size(s).numel(), device=DEV).to(dtype)[1:].view(s) for s in shapes]
    assert all(t.data_ptr() % 16 for t in off)

    def run(tensors, grad):
        x, d, g, b = (t.detach().requires_grad_(grad) for t in tensors[:4])
        out = ops.add_layer_norm(x, d, g, b) if residual else (ops.layer_norm(x, g, b),)
        leaves = (x, d, g, b) if residual else (x, g, b)
        return [o.detach() for o in out] + list(torch.autograd.grad(out, leaves, tensors[4:4 + len(out)]) if grad else ())
    for grad in (False, True):
        for i in range(7):                                                # all, or one at a time
            mixed = [t if i in (j, 6) else t.clone() for j, t in enumerate(off)]
            for a, w in zip(run(mixed, grad), run([t.clone() for t in off], grad)):
                assert torch.equal(a, w)
    # sums of six values in another order: 6 roundings of 2^-24
    assert float((ops.column_sum(off[0]) - ops.column_sum(off[0].clone())).abs().max()) <= 6 * 2 ** -24 * float(off[0].float().abs().sum(0).max())


@pytest.mark.parametrize("form", ["dense", "strided", "other type"])
@pytest.mark.parametrize("native", [False, True])
@pytest.mark.parametrize("residual", [False, True])
def test_second_derivatives_are_refused(native, residual, form, monkeypatch):
    """First derivatives with ``create_graph`` are what they are without; one of them, also beside terms that do have a second
    derivative, is not taken for a constant."""
    from axonn_b200 import ops
    from axonn_b200.ops import _lib

    if not native:
        monkeypatch.setattr(_lib, "_HOST", None)
    x, d = (torch.randn(3, 5, 64, device=DEV, requires_grad=True) for _ in range(2))
    g = torch.ones(64, device=DEV, dtype=BF16 if form == "other type" else torch.float32, requires_grad=True)
    leaves = (x, d, g) if residual else (x, g)

    def loss():
        a, b = (t.transpose(0, 1) if form == "strided" else t for t in (x, d))
        y = sum(ops.add_layer_norm(a, b, g, None)) if residual else ops.rms_norm(a, g)
        return y.sum() + sum((t ** 3).sum() for t in leaves)
    want = torch.autograd.grad(loss(), leaves)
    got = torch.autograd.grad(loss(), leaves, create_graph=True)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    for a in got:
        for leaf in leaves:
            with pytest.raises(RuntimeError, match="second derivatives"):
                torch.autograd.grad(a.pow(2).sum(), leaf, allow_unused=True, retain_graph=True)


@pytest.mark.parametrize("dtype", [BF16, torch.float16, torch.float32])
def test_linear_and_attention(dtype, monkeypatch):
    from axonn_b200 import ops
    from axonn_b200.intra_layer import Linear

    for n, k, bias, act in ((64, 24, True, "gelu"), (264, 512, False, None), (20, 24, True, None), (8, 8, False, "gelu")):
        layer = Linear(k, n, bias=bias, expert_mode=True, dtype=dtype)
        for x in _forms((2, 33, k), dtype):
            def call():
                with torch.no_grad():
                    return layer(x, activation=act)
            try:
                want = _python(monkeypatch, call)
            except Exception as e:
                with pytest.raises(type(e)):
                    call()
                continue
            assert torch.equal(call(), want)
    for shape in ((2, 100, 2, 4, 64), (1, 256, 1, 3, 128), (1, 9, 2, 3, 32)):
        for qkv in _forms(shape, dtype):
            with torch.no_grad():
                assert torch.equal(ops.flash_attention_packed(qkv), _python(monkeypatch, lambda: ops.flash_attention_packed(qkv)))


def test_launch_errors_keep_their_type(monkeypatch):
    """A launcher that refuses a call: the error and its text are those of the Python paths.  What is not for the native paths is left
    to the general ones."""
    from axonn_b200 import ops
    from axonn_b200.intra_layer import Linear
    from axonn_b200.ops import _lib

    assert issubclass(_lib.KernelError, RuntimeError)
    layer = Linear(64, 64, bias=False, expert_mode=True, dtype=BF16)
    flat, narrow = torch.randn(65, device=DEV, dtype=BF16), torch.randn(2, 12, device=DEV, dtype=BF16)
    gain = torch.ones(12, device=DEV, dtype=BF16)

    def refused(call):
        before = _lib.launch_count
        with torch.no_grad(), pytest.raises(_lib.KernelError) as e:
            call()
        assert _lib.launch_count == before
        return str(e.value)
    for call, text in ((lambda: layer(flat[1:].view(1, 64)), "axb_gemm failed (status -1): TMA base address must be 16-byte aligned"),
                       (lambda: ops.rms_norm(narrow, gain), "axb_norm_fwd failed (status -1): norm: hidden 12 unsupported"),
                       (lambda: ops.add_rms_norm(narrow, narrow, gain), "axb_add_norm_fwd failed (status -1): norm: hidden 12 unsupported")):
        assert refused(call) == text == _python(monkeypatch, lambda: refused(call))
    x = narrow.clone().requires_grad_(True)
    with pytest.raises(_lib.KernelError):
        ops.rms_norm(x, gain)
    host = _lib.host()
    x, w = torch.randn(8, device=DEV, dtype=BF16), torch.ones(8, device=DEV, dtype=BF16)
    assert host.norm(x.cpu(), None, w, None, 1e-5, True) is None and host.norm(x, None, w.cpu(), None, 1e-5, True) is None
    assert host.norm(x, None, w[:4], None, 1e-5, True) is None and host.norm(x, None, w.float(), None, 1e-5, True) is None
    assert host.linear(x, w, None, 8, 8, False) is None and host.attention(x, 1.0) is None
    with pytest.raises(TypeError):
        host.norm(x, None, w, None, "eps", True)


@pytest.mark.parametrize("path,grad", [("norm", False), ("norm", True), ("linear", False), ("attention", False)])
def test_other_threads_run_while_a_launch_waits(path, grad):
    """A launch that finds the queue full (more of them than it holds, behind half a second of work) holds up its own thread only."""
    from axonn_b200.ops import _lib

    host = _lib.host()
    x, w = torch.randn(16, 64, device=DEV, dtype=BF16, requires_grad=grad), torch.ones(64, device=DEV, dtype=BF16)
    weight, qkv = torch.randn(64 * 64, device=DEV, dtype=BF16), torch.randn(1, 8, 1, 3, 64, device=DEV, dtype=BF16)
    call = {"norm": lambda: host.norm(x, None, w, None, 1e-5, True), "linear": lambda: host.linear(x, weight, None, 64, 64, False),
            "attention": lambda: host.attention(qkv, 0.125)}[path]
    assert call() is not None
    torch.cuda.synchronize()
    ticks, done = [time.perf_counter()], threading.Event()

    def tick():
        while not done.wait(1e-3):
            ticks.append(time.perf_counter())
    other = threading.Thread(target=tick)
    other.start()
    longest = 0.0
    torch.cuda._sleep(10 ** 9)
    gc.disable()                                                       # a collection stops both threads
    try:
        for _ in range(3000):
            t = time.perf_counter()
            call()
            longest = max(longest, time.perf_counter() - t)
    finally:
        gc.enable()
        done.set()
        other.join()
    torch.cuda.synchronize()
    assert longest > 0.2                                               # the queue was full
    assert max(b - a for a, b in zip(ticks, ticks[1:])) < longest / 2
