"""The workloads that a program built on this package spends its GPU time on, one process, one GPU.

Every case goes through the entry points that a training or inference script calls: the tensor-parallel layers and
blocks, the attention / norm / loss operators, gradient pruning, clipping and the optimizer.  Sizes are those of the
package's own configurations (GPT-1.3B: hidden 2048, 16 heads, FFN 8192, vocabulary 50304; Llama-8B: hidden 4096,
32 query / 8 KV heads, FFN 14336), of its tests (hidden 256), and odd ones in between.  Forward-only cases are the
prompt evaluation that greedy decoding repeats for every token; the others are the layers of a training step.
"""

import math

import torch
import torch.distributed as dist
import torch.nn.functional as F

from axonn_b200 import axonn as ax
from axonn_b200 import ops
from axonn_b200.intra_layer import clip_grad_norm_
from axonn_b200.models import GPT, GPTConfig
from axonn_b200.models.blocks import ParallelAttention, ParallelLMHead, ParallelMLP, TransformerBlock, TPNorm
from axonn_b200.optim import FusedAdamW
from axonn_b200.parallel.moe import ExpertParallelMoE

BF16 = torch.bfloat16
DEV = "cuda"


def listed():
    return [
        # a short prompt (greedy decoding evaluates the whole prefix for every token): weights are read once, few rows
        dict(name="mlp_short_prompt", kind="mlp", tokens=24, hidden=2048, ffn=8192, act="gelu"),
        # attention layer of a Llama-8B model on one prompt of an odd length, no gradients
        dict(name="attention_prompt", kind="attn_layer", batch=1, seq=777, heads=32, kv_heads=8, head_dim=128),
        # the attention of a GPT-1.3B training step, forward and backward
        dict(name="attention_train", kind="attn", batch=8, seq=2048, groups=16, qpk=1, head_dim=128),
        # grouped-query attention on training sequences cut at an odd length (fine-tuning on documents)
        dict(name="attention_train_odd", kind="attn", batch=4, seq=1531, groups=8, qpk=4, head_dim=128),
        # residual add + LayerNorm between the sub-layers of a GPT-1.3B training step
        dict(name="add_layer_norm_train", kind="norm", rows=16384, hidden=2048, rms=False, residual=True),
        # RMSNorm of a Llama-8B model on an odd number of tokens
        dict(name="rms_norm_train_odd", kind="norm", rows=4099, hidden=4096, rms=True, residual=False),
        # final projection to the vocabulary with its cross-entropy, forward and backward
        dict(name="lm_head_loss", kind="lm_head", tokens=4096, hidden=2048, vocab=50304),
        # end of a training step: gradient clipping and AdamW over the parameters of one GPT-1.3B block
        dict(name="clip_and_adamw", kind="optimizer", hidden=2048, ffn=8192),
        # gradient pruning (keep the largest 10 %) of the weight gradients of one Llama-8B block
        dict(name="prune_gradients", kind="prune", hidden=4096, ffn=14336, qkv=6144, dtype="bf16", keep=0.1),
        # mixture-of-experts feed-forward layer of a training step
        dict(name="moe_train", kind="moe", tokens=8192, hidden=2048, ffn=8192, experts=8, top_k=2),
        # one whole GPT-1.3B block of a training step at the benchmark's batch: the largest call
        dict(name="gpt_block_train", kind="block", batch=8, seq=2048, hidden=2048, heads=16, kv_heads=16, ffn=8192,
             llama=False),
        # logits of a small GPT on a batch of short prompts: launches and host work
        dict(name="small_gpt_logits", kind="gpt", batch=4, seq=77, layers=2, hidden=256, heads=4, ffn=1024,
             vocab=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _seq(rng, lo, hi):
    """Sequence lengths: half of them any length, half a multiple of 128."""
    s = _log(rng, lo, hi)
    return s if rng.random() < 0.5 else max(128, s // 128 * 128)


def draw(rng):
    kind = rng.choice(["mlp", "attn_layer", "attn", "norm", "lm_head", "optimizer", "prune", "moe", "block", "gpt"])
    if kind == "mlp":
        hidden = rng.choice([256, 1024, 2048, 4096])
        return dict(kind=kind, tokens=_log(rng, 1, 4096), hidden=hidden, ffn=rng.choice([2, 3, 4]) * hidden,
                    act=rng.choice(["gelu", "swiglu"]))
    if kind == "attn_layer":
        d, qpk = rng.choice([64, 128]), rng.choice([1, 2, 4])
        kv = rng.choice([2, 4, 8])
        return dict(kind=kind, batch=rng.randint(1, 4), seq=_seq(rng, 5, 4096), heads=kv * qpk, kv_heads=kv, head_dim=d)
    if kind == "attn":
        seq = _seq(rng, 64, 4096)
        return dict(kind=kind, batch=max(1, min(16, _log(rng, 1, 16384 / seq))), seq=seq, groups=rng.choice([2, 4, 8]),
                    qpk=rng.choice([1, 2, 4]), head_dim=rng.choice([64, 128]))
    if kind == "norm":
        hidden = rng.choice([128, 256, 768, 1024, 1536, 2048, 3072, 4096, 5120, 8192])
        return dict(kind=kind, rows=_log(rng, 1, 40_000_000 / hidden), hidden=hidden, rms=rng.random() < 0.5,
                    residual=rng.random() < 0.5)
    if kind == "lm_head":
        return dict(kind=kind, tokens=_log(rng, 16, 4096), hidden=rng.choice([256, 1024, 2048]),
                    vocab=rng.choice([1024, 32000, 50304]))
    if kind == "optimizer":
        hidden = rng.choice([256, 1000, 1024, 2048])
        return dict(kind=kind, hidden=hidden, ffn=rng.choice([2, 3, 4]) * hidden)
    if kind == "prune":
        hidden = rng.choice([256, 1000, 2048, 4096])
        return dict(kind=kind, hidden=hidden, ffn=rng.choice([2, 3]) * hidden, qkv=3 * hidden,
                    dtype=rng.choice(["bf16", "bf16", "fp32", "fp16"]), keep=rng.choice([0.01, 0.1, 0.5]))
    if kind == "moe":
        hidden = rng.choice([256, 1024, 2048])
        return dict(kind=kind, tokens=_log(rng, 32, 8192), hidden=hidden, ffn=rng.choice([2, 3, 4]) * hidden,
                    experts=rng.choice([4, 8]), top_k=2)
    if kind == "block":
        seq, llama = _seq(rng, 64, 2048), rng.random() < 0.5
        heads = rng.choice([4, 8, 16])
        return dict(kind=kind, batch=max(1, min(16, _log(rng, 1, 12288 / seq))), seq=seq, hidden=128 * heads,
                    heads=heads, kv_heads=heads // 4 if llama else heads, ffn=(3 if llama else 4) * 128 * heads,
                    llama=llama)
    hidden = rng.choice([256, 512, 1024])
    return dict(kind=kind, batch=rng.randint(1, 8), seq=_seq(rng, 5, 512), layers=rng.randint(1, 4), hidden=hidden,
                heads=hidden // rng.choice([64, 128]), ffn=4 * hidden, vocab=rng.choice([1024, 8192]))


# ---------------------------------------------------------------------------------------------- inputs from the seed
class _Rand:
    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(int(seed) % (1 << 62))

    def normal(self, shape, std=1.0, dtype=BF16, mean=0.0):
        return (torch.randn(shape, device=DEV, generator=self.gen) * std + mean).to(dtype)

    def ints(self, high, shape):
        return torch.randint(0, high, shape, device=DEV, generator=self.gen)


def _named(module, r, std=0.02):
    """Fill a layer's parameters from the seed: matrices N(0, std), gains around one, biases around zero."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if "norm" in name and name.endswith("weight"):
                p.copy_(r.normal(p.shape, 0.1, p.dtype, 1.0))
            elif name.endswith("bias"):
                p.copy_(r.normal(p.shape, 0.1, p.dtype))
            else:
                p.copy_(r.normal(p.shape, std, p.dtype))
    return module


def _start():
    if not dist.is_initialized():
        torch.cuda.set_device(0)
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1)
    if not ax.is_initialized:
        ax.init(G_inter=1, G_data=1, G_intra_r=1, G_intra_c=1, G_intra_d=1)


def _optimizer_shapes(c):
    h, f = c["hidden"], c["ffn"]
    return [(h,), (h,), (3 * h * h,), (3 * h,), (h * h,), (h,), (h,), (h,), (h * f,), (f,), (h * f,), (h,)]


def prepare(case, seed):
    _start()
    c, r = case, _Rand(seed)
    kind = c["kind"]
    s = dict(c)
    if kind == "mlp":
        s["layer"] = _named(ParallelMLP(c["hidden"], c["ffn"], c["act"], bias=c["act"] == "gelu", dtype=BF16), r)
        s["x"] = r.normal((1, c["tokens"], c["hidden"]))
    elif kind == "attn_layer":
        h = c["heads"] * c["head_dim"]
        s["layer"] = _named(ParallelAttention(h, c["heads"], c["kv_heads"], bias=False, rope_theta=500000.0,
                                              max_seq=4096, dtype=BF16), r)
        s["x"] = r.normal((c["batch"], c["seq"], h))
    elif kind == "attn":
        s["qkv"] = r.normal((c["batch"], c["seq"], c["groups"], c["qpk"] + 2, c["head_dim"])).requires_grad_(True)
        s["dout"] = r.normal((c["batch"], c["seq"], c["groups"] * c["qpk"], c["head_dim"]))
    elif kind == "norm":
        s["norm"] = TPNorm(c["hidden"], eps=1e-5, rms=c["rms"], dtype=BF16)
        with torch.no_grad():
            s["norm"].weight.copy_(r.normal((c["hidden"],), 0.1, BF16, 1.0))
            if s["norm"].bias is not None:
                s["norm"].bias.copy_(r.normal((c["hidden"],), 0.1))
        for k in ("x", "delta") if c["residual"] else ("x",):
            s[k] = r.normal((c["rows"], c["hidden"])).requires_grad_(True)
        for k in ("dy", "dh") if c["residual"] else ("dy",):
            s[k] = r.normal((c["rows"], c["hidden"]))
    elif kind == "lm_head":
        s["layer"] = _named(ParallelLMHead(c["hidden"], c["vocab"], dtype=BF16), r)
        s["x"] = r.normal((1, c["tokens"], c["hidden"])).requires_grad_(True)
        s["targets"] = r.ints(c["vocab"], (1, c["tokens"]))
    elif kind == "optimizer":
        s["params"] = [torch.nn.Parameter(r.normal(n, 0.02)) for n in _optimizer_shapes(c)]
        for p in s["params"]:
            p.grad = r.normal(p.shape, 1e-3)
        s["opt"] = FusedAdamW(s["params"], lr=1e-3, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    elif kind == "prune":
        s["new"] = _prune_grads(c, r)
        s["grads"] = [torch.empty_like(g) for g in s["new"]]
    elif kind == "moe":
        s["layer"] = _named(ExpertParallelMoE(c["hidden"], c["ffn"], n_experts=c["experts"], top_k=c["top_k"],
                                              dtype=BF16), r)
        s["x"] = r.normal((1, c["tokens"], c["hidden"])).requires_grad_(True)
        s["dy"] = r.normal((1, c["tokens"], c["hidden"]))
    elif kind == "block":
        ll = c["llama"]
        s["layer"] = _named(TransformerBlock(c["hidden"], c["heads"], c["ffn"], n_kv_heads=c["kv_heads"],
                                             activation="swiglu" if ll else "gelu", rms=ll, bias=not ll,
                                             rope_theta=500000.0 if ll else None, max_seq=2048, dtype=BF16), r)
        s["x"] = r.normal((c["batch"], c["seq"], c["hidden"])).requires_grad_(True)
        s["dy"] = r.normal((c["batch"], c["seq"], c["hidden"]))
    else:
        cfg = GPTConfig(n_layers=c["layers"], hidden=c["hidden"], n_heads=c["heads"], ffn=c["ffn"], vocab=c["vocab"],
                        seq_len=512)
        s["layer"] = _named(GPT(cfg, dtype=BF16), r, std=0.05).eval()
        s["tokens_in"] = r.ints(c["vocab"], (c["batch"], c["seq"]))
    return s


def _prune_grads(c, r):
    dt = {"bf16": BF16, "fp32": torch.float32, "fp16": torch.float16}[c["dtype"]]
    h, f = c["hidden"], c["ffn"]
    return [r.normal((n,), 1e-2, dt) for n in (c["qkv"] * h, h * h, 2 * f * h, f * h)]


# ----------------------------------------------------------------------------------------------------------- one pass
def run(state):
    s = state
    kind = s["kind"]
    if kind in ("mlp", "attn_layer"):
        with torch.no_grad():
            return s["layer"](s["x"])
    if kind == "gpt":
        with torch.no_grad():
            return s["layer"](s["tokens_in"])
    if kind == "attn":
        out = ops.flash_attention_packed(s["qkv"])
        return [out.detach(), *torch.autograd.grad(out, s["qkv"], s["dout"])]
    if kind == "norm":
        leaves = [s["x"], *s["norm"].parameters()]
        if s["residual"]:
            h, y = s["norm"].add_norm(s["x"], s["delta"])
            return [h.detach(), y.detach(), *torch.autograd.grad([h, y], leaves, [s["dh"], s["dy"]])]
        y = s["norm"](s["x"])
        return [y.detach(), *torch.autograd.grad(y, leaves, s["dy"])]
    if kind == "lm_head":
        loss = s["layer"](s["x"], s["targets"])
        return [loss.detach(), *torch.autograd.grad(loss, [s["x"], *s["layer"].parameters()])]
    if kind == "optimizer":
        total = clip_grad_norm_(s["params"], 1.0)
        s["opt"].step()
        st = s["opt"].state
        return [total] + [t for p in s["params"]
                          for t in (p.detach(), p.grad, st[p]["master"], st[p]["exp_avg"], st[p]["exp_avg_sq"])]
    if kind == "prune":
        for g, new in zip(s["grads"], s["new"]):
            g.copy_(new)                       # backward has left a new gradient in the parameter's buffer
            ops.prune_topk_(g, s["keep"])
        return list(s["grads"])
    if kind == "moe":
        y = s["layer"](s["x"])
        loss_parts = [y, s["layer"].last_aux_loss]
        upstream = [s["dy"], torch.full((), 0.02, device=DEV)]
        return [y.detach(), *torch.autograd.grad(loss_parts, [s["x"], *s["layer"].parameters()], upstream)]
    y = s["layer"](s["x"])                     # a whole block
    return [y.detach(), *torch.autograd.grad(y, [s["x"], *s["layer"].parameters()], s["dy"])]


# ------------------------------------------------------------------------- bytes and operations a pass cannot do without
def _attn_flops(batch, heads, seq, d):
    return 4 * batch * heads * d * seq * (seq + 1) / 2


def work(case):
    c, kind = case, case["kind"]
    if kind == "mlp":
        w = (3 if c["act"] == "swiglu" else 2) * c["hidden"] * c["ffn"]
        return dict(bytes=2 * w + 4 * c["tokens"] * c["hidden"], flops=2 * w * c["tokens"])
    if kind == "attn_layer":
        h, t = c["heads"] * c["head_dim"], c["batch"] * c["seq"]
        w = h * (2 * h + 2 * c["kv_heads"] * c["head_dim"])
        return dict(bytes=2 * w + 4 * t * h,
                    flops=2 * w * t + _attn_flops(c["batch"], c["heads"], c["seq"], c["head_dim"]))
    if kind == "attn":
        t, d = c["batch"] * c["seq"], c["head_dim"]
        heads = c["groups"] * c["qpk"]
        return dict(bytes=2 * t * d * (2 * c["groups"] * (c["qpk"] + 2) + 2 * heads),
                    flops=3.5 * _attn_flops(c["batch"], heads, c["seq"], d))
    if kind == "norm":
        n = c["rows"] * c["hidden"]
        return dict(bytes=2 * n * (7 if c["residual"] else 4), flops=20 * n)
    if kind == "lm_head":
        w = c["hidden"] * c["vocab"]
        return dict(bytes=4 * w + 4 * c["tokens"] * c["hidden"], flops=6 * w * c["tokens"])
    if kind == "optimizer":
        n = sum(s[0] for s in _optimizer_shapes(c))
        return dict(bytes=n * (2 + 2 + 4 * 3 * 2 + 2), flops=20 * n)
    if kind == "prune":
        n = c["hidden"] * (c["qkv"] + c["hidden"] + 3 * c["ffn"])
        return dict(bytes=n * (4 if c["dtype"] == "fp32" else 2) * 2, flops=2 * n)
    if kind == "moe":
        h, f, t = c["hidden"], c["ffn"], c["tokens"]
        w = 3 * h * f * c["experts"]
        return dict(bytes=4 * w + 8 * t * h, flops=6 * 3 * h * f * t * c["top_k"])
    if kind == "block":
        h, t = c["hidden"], c["batch"] * c["seq"]
        d = h // c["heads"]
        w = h * (2 * h + 2 * c["kv_heads"] * d) + (3 if c["llama"] else 2) * h * c["ffn"]
        return dict(bytes=4 * w + 8 * t * h,
                    flops=6 * w * t + 3.5 * _attn_flops(c["batch"], c["heads"], c["seq"], d))
    h, t = c["hidden"], c["batch"] * c["seq"]
    w = c["layers"] * (4 * h * h + 2 * h * c["ffn"]) + h * c["vocab"]
    return dict(bytes=2 * w + 2 * t * c["vocab"],
                flops=2 * w * t + c["layers"] * _attn_flops(c["batch"], c["heads"], c["seq"], h // c["heads"]))


def tolerance(case):
    """About four times what the path differs by from its 64-bit value: bf16 storage of the results and of the
    intermediate activations (2^-9 per rounding)."""
    kind = case["kind"]
    if kind == "prune":
        return "exact"
    if kind == "optimizer":
        return {"rel": 2e-4}      # fp32 arithmetic; a gradient at a bf16 rounding boundary may go the other way
    return {"rel": {"norm": 8e-3,       # one rounding: measured 1.7e-3
                    "lm_head": 1e-2,    # 2.9e-3
                    "attn": 1.2e-2,     # bf16 probabilities and score gradients: 2.8e-3
                    "mlp": 2e-2, "attn_layer": 2e-2, "moe": 2e-2,      # a layer's rounded intermediates: 5e-3
                    "block": 2.4e-2, "gpt": 3e-2}[kind]}               # several layers: 6e-3, 7e-3


# ------------------------------------------------------------------------------------------- the same path in 64 bits
def _rope(x, theta):
    s, d = x.shape[1], x.shape[-1]
    inv = 1.0 / theta ** (torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    ang = torch.outer(torch.arange(s, dtype=torch.float64, device=x.device), inv)
    shape = [1, s] + [1] * (x.ndim - 3) + [d // 2]
    cos, sin = ang.cos().view(shape), ang.sin().view(shape)
    a, b = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(qkv, theta=None):
    """Causal attention of [batch, seq, groups, q_per_kv + 2, head_dim]; one batch element at a time."""
    if theta is not None:
        qkv = torch.cat([_rope(qkv[:, :, :, :-1], theta), qkv[:, :, :, -1:]], 3)
    b, s, g, n, d = qkv.shape
    hidden = torch.ones(s, s, dtype=torch.bool, device=qkv.device).triu(1)
    outs = []
    for i in range(b):
        q, k, v = qkv[i, :, :, :n - 2], qkv[i, :, :, n - 2], qkv[i, :, :, n - 1]
        z = torch.einsum("sgqd,tgd->gqst", q, k) / math.sqrt(d)
        p = z.masked_fill(hidden, -math.inf).softmax(-1)
        outs.append(torch.einsum("gqst,tgd->sgqd", p, v).reshape(s, g * (n - 2), d))
    return torch.stack(outs)


def _swiglu(z):
    v = z.reshape(*z.shape[:-1], z.shape[-1] // 16, 2, 8)
    gate, up = (v[..., i, :].reshape(*z.shape[:-1], z.shape[-1] // 2) for i in (0, 1))
    return F.silu(gate) * up


def _norm64(x, w, b, rms):
    if rms:
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * w
    return F.layer_norm(x, x.shape[-1:], w, b, 1e-5)


def _mlp64(x, p, prefix, hidden, act):
    z = F.linear(x, p[prefix + "fc1.weight"].reshape(-1, hidden), p.get(prefix + "fc1.bias"))
    z = _swiglu(z) if act == "swiglu" else F.gelu(z, approximate="tanh")
    return F.linear(z, p[prefix + "fc2.weight"].reshape(hidden, -1), p.get(prefix + "fc2.bias"))


def _attention64(x, p, prefix, kv_heads, head_dim, theta):
    b, s, h = x.shape
    qkv = F.linear(x, p[prefix + "qkv.weight"].reshape(-1, h), p.get(prefix + "qkv.bias"))
    o = _attend(qkv.reshape(b, s, kv_heads, -1, head_dim), theta).reshape(b, s, -1)
    return F.linear(o, p[prefix + "proj.weight"].reshape(h, -1), p.get(prefix + "proj.bias"))


def _block64(x, p, prefix, hidden, kv_heads, head_dim, llama):
    theta, act = (500000.0, "swiglu") if llama else (None, "gelu")
    y = _norm64(x, p[prefix + "norm1.weight"], p.get(prefix + "norm1.bias"), llama)
    x = x + _attention64(y, p, prefix + "attn.", kv_heads, head_dim, theta)
    y = _norm64(x, p[prefix + "norm2.weight"], p.get(prefix + "norm2.bias"), llama)
    return x + _mlp64(y, p, prefix + "mlp.", hidden, act)


def _moe64(s, x, router, w1, w2):
    """Routing as the layer defines it (bf16 logits, fp32 softmax, top-k, capacity in token order); 64 bits after it."""
    c = s
    t, e, k = x.shape[0], c["experts"], c["top_k"]
    z = x @ router.t()
    z = z + (z.to(BF16).double() - z).detach()               # the router's logits are bf16 values
    idx = z.detach().float().softmax(-1).topk(k, -1)[1]
    probs = z.softmax(-1)
    gate = probs.gather(1, idx)
    gate = gate / gate.sum(-1, keepdim=True)
    onehot = F.one_hot(idx.reshape(-1), e)
    slot = ((onehot.cumsum(0) * onehot).sum(-1) - 1).reshape(t, k)
    capacity = max(8, (math.ceil(1.25 * t * k / e) + 7) // 8 * 8)
    y = torch.zeros_like(x)
    for i in range(e):
        tok, which = ((idx == i) & (slot < capacity)).nonzero(as_tuple=True)
        out = _swiglu(x[tok] @ w1[i].t()) @ w2[i].t()
        y = y.index_add(0, tok, out * gate[tok, which][:, None])
    aux = e * (onehot.double().mean(0) * probs.mean(0)).sum()
    return y, aux


def exact(case, seed):
    s = prepare(case, seed)
    kind = s["kind"]
    if kind == "prune":
        out = []
        for g in s["new"]:
            keep = max(1, int(round(g.numel() * s["keep"])))
            limit = g.abs().float().sort(descending=True)[0][keep - 1]
            out.append(torch.where(g.abs().float() >= limit, g, torch.zeros_like(g)))
        return out
    if kind == "optimizer":
        total = torch.stack([p.grad.double().pow(2).sum() for p in s["params"]]).sum().sqrt()
        clip = (1.0 / (total + 1e-6)).clamp(max=1.0)
        out = [total]
        for p in s["params"]:
            g = (p.grad.double() * clip).to(BF16)            # gradients stay bf16 tensors
            m, v = 0.1 * g.double(), 0.05 * g.double() ** 2
            w = p.detach().double() * (1 - 1e-3 * 0.1) - 1e-3 * (m / 0.1) / ((v / 0.05).sqrt() + 1e-8)
            out += [w, g.double(), w, m, v]
        return out
    if kind == "attn":
        qkv = s["qkv"].detach().double().requires_grad_(True)
        out = _attend(qkv)
        return [out.detach(), *torch.autograd.grad(out, qkv, s["dout"].double())]
    if kind == "norm":
        p = [q.detach().double().requires_grad_(True) for q in s["norm"].parameters()]
        x = s["x"].detach().double().requires_grad_(True)
        if s["residual"]:
            h = x + s["delta"].detach().double()
            h = h + (h.to(BF16).double() - h).detach()       # the residual stream is a bf16 tensor
            y = _norm64(h, p[0], p[1] if len(p) > 1 else None, s["rms"])
            return [h.detach(), y.detach(),
                    *torch.autograd.grad([h, y], [x, *p], [s["dh"].double(), s["dy"].double()])]
        y = _norm64(x, p[0], p[1] if len(p) > 1 else None, s["rms"])
        return [y.detach(), *torch.autograd.grad(y, [x, *p], s["dy"].double())]
    p = {n: q.detach().double().requires_grad_(True) for n, q in s["layer"].named_parameters()}
    if kind == "gpt":
        with torch.no_grad():
            h, tok = s["hidden"], s["tokens_in"]
            x = p["tok_emb.weight"].reshape(-1, h)[tok] + p["pos_emb.weight"].reshape(-1, h)[:tok.shape[1]]
            for i in range(s["layers"]):
                x = _block64(x, p, "blocks.%d." % i, h, s["heads"], h // s["heads"], False)
            return _norm64(x, p["norm_f.weight"], p["norm_f.bias"], False) @ p["head.proj.weight"].reshape(-1, h).t()
    x = s["x"].detach().double().requires_grad_(True)
    if kind == "mlp":
        with torch.no_grad():
            return _mlp64(x, p, "", s["hidden"], s["act"])
    if kind == "attn_layer":
        with torch.no_grad():
            return _attention64(x, p, "", s["kv_heads"], s["head_dim"], 500000.0)
    if kind == "lm_head":
        z = x.reshape(-1, s["hidden"]) @ p["proj.weight"].reshape(-1, s["hidden"]).t()
        loss = F.cross_entropy(z, s["targets"].reshape(-1))
        return [loss.detach(), *torch.autograd.grad(loss, [x, *p.values()])]
    if kind == "moe":
        y, aux = _moe64(s, x.reshape(-1, s["hidden"]), p["router"], p["w1"], p["w2"])
        y = y.reshape(x.shape)
        return [y.detach(), *torch.autograd.grad([y, aux], [x, *p.values()],
                                                 [s["dy"].double(), torch.full((), 0.02, dtype=torch.float64,
                                                                               device=DEV)])]
    y = _block64(x, p, "", s["hidden"], s["kv_heads"], s["hidden"] // s["heads"], s["llama"])
    return [y.detach(), *torch.autograd.grad(y, [x, *p.values()], s["dy"].double())]
