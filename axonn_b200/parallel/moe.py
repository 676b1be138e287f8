"""Expert-parallel mixture-of-experts layer (top-k softmax router, SwiGLU experts).

Experts are partitioned over an expert-parallel group (by default the
data-parallel group: every data-parallel rank owns ``n_experts / G_data``
experts and routes its own tokens).  Tokens travel to the owners of their
experts and back with an all-to-all in each direction:

* on GPUs with peer memory the exchange is done by this package's dispatch and
  combine kernels (``csrc/moe.cu``): a token row is stored straight into the
  owning rank's expert buffer over NVLink while it is being gathered, and the
  expert outputs are pulled back, scaled by the gate and summed in one pass;
* otherwise ``all_to_all_single`` moves fixed-capacity buffers.

Fixed expert capacity keeps all shapes static (no host synchronisation):
``capacity = ceil(capacity_factor * tokens * top_k / n_experts)`` slots per
expert and source rank; assignments beyond it are dropped, as in
GShard/Switch routing.

The reference has no expert parallelism — its Mixtral patch only
tensor-parallelises every expert
(``axonn/models/transformers/modify_mixtral.py:86-97``); this layer is an
extension required for the Mixtral-style configuration.
"""

import ctypes
import math

import torch
import torch.distributed as dist
import torch.nn as nn
import torch.nn.functional as F
from torch.autograd.function import once_differentiable

from .. import axonn as ax
from .. import ops
from ..ops import _lib


class _AllToAll(torch.autograd.Function):
    """Equal-split all-to-all along dim 0; backward is the same exchange."""

    @staticmethod
    def forward(ctx, x, group):
        ctx.group = group
        if dist.get_world_size(group) == 1:
            return x
        x = x.contiguous()
        out = torch.empty_like(x)
        dist.all_to_all_single(out, x, group=group)
        return out

    @staticmethod
    def backward(ctx, g):
        if dist.get_world_size(ctx.group) == 1:
            return g, None
        g = g.contiguous()
        out = torch.empty_like(g)
        dist.all_to_all_single(out, g, group=ctx.group)
        return out, None


class _LocalRoute(torch.autograd.Function):
    """Top-``k`` softmax routing of ``logits [T, E]`` (bf16) into capacity buffers of ``rows`` rows per expert, ``C`` of them in
    use: ``(gate [T, k], balance loss, dest, inverse, counts, statistics)``; two launches forward and one backward
    (``csrc/moe_local.cu``).  Statistics: ``[assignments per expert | dropped per expert | dropped fraction]``."""

    @staticmethod
    def forward(ctx, logits, k, C, rows):
        logits = logits.contiguous()
        T, E = logits.shape
        dev = logits.device
        idx, dest, inverse, counts = (torch.empty(n, dtype=torch.int32, device=dev) for n in (T * k, T * k, E * rows, E))
        gate, aux, stats, assigned, scratch = (torch.empty(n, dtype=torch.float32, device=dev)
                                               for n in ((T, k), (), 2 * E + 1, E, ((T + 127) // 128 + 1) * E + 1))
        word = stats.data_ptr()
        _lib.check(_lib.lib().axb_moe_route(_lib.addr(logits), T, E, k, C, rows, _lib.addr(idx), _lib.addr(gate),
                                            _lib.addr(dest), _lib.addr(inverse), _lib.addr(counts), _lib.addr(assigned), word,
                                            word + 4 * E, _lib.addr(aux), word + 8 * E, _lib.addr(scratch), _lib.stream()), "axb_moe_route")
        _lib.add_launches(1)
        ctx.save_for_backward(logits, idx, gate, assigned)      # the statistics are the caller's, who may sum them in place
        ctx.mark_non_differentiable(dest, inverse, counts, stats)
        ctx.set_materialize_grads(False)
        ctx.k = k
        return gate, aux, dest, inverse, counts, stats

    @staticmethod
    @once_differentiable
    def backward(ctx, dgate, daux, *_):
        logits, idx, gate, assigned = (t.contiguous() for t in ctx.saved_tensors)
        if dgate is None and daux is None:
            return None, None, None, None
        T, E = logits.shape
        dgate = None if dgate is None else dgate.float().contiguous()
        daux = None if daux is None else daux.float()
        dlogits = torch.empty_like(logits)
        _lib.check(_lib.lib().axb_moe_route_bwd(_lib.addr(logits), T, E, ctx.k, _lib.addr(idx), _lib.addr(gate), _lib.addr(dgate),
                                                _lib.addr(daux), _lib.addr(assigned), _lib.addr(dlogits), _lib.stream()),
                   "axb_moe_route_bwd")
        return dlogits, None, None, None


_ROUTE_MAX_EXPERTS = 32       # AXB_MOE_MAX_EXPERTS: the routing kernel holds a token's logits in registers


class _LocalDispatch(torch.autograd.Function):
    """Token rows ``[T, H]`` into the experts' capacity buffers ``[E, rows, H]`` (zeros where no token is), and the
    adjoint: the sum of a token's rows (``csrc/moe_local.cu``)."""

    @staticmethod
    def forward(ctx, x2, dest, inverse, E, rows, k):
        x2 = _dense(x2)
        ctx.save_for_backward(dest)
        ctx.T, ctx.k = x2.shape[0], k
        out = torch.empty((E, rows, x2.shape[1]), dtype=x2.dtype, device=x2.device)
        _rows_kernel(x2, inverse, out, None, None, None, k)
        return out

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        (dest,) = ctx.saved_tensors
        return _tokens_kernel(_dense(g), dest, None, ctx.T, ctx.k), None, None, None, None, None


class _LocalCombine(torch.autograd.Function):
    """``y[t] = sum_j gate[t, j] * out[dest[t, j]]`` over the kept assignments, fp32 sums; the adjoint gives the
    experts' output gradient and the gate's in one pass."""

    @staticmethod
    def forward(ctx, out, gate, dest, inverse, T, k):
        ctx.save_for_backward(out, gate, dest, inverse)
        ctx.k = k
        return _tokens_kernel(out, dest, gate, T, k)

    @staticmethod
    @once_differentiable
    def backward(ctx, g):
        out, gate, dest, inverse = ctx.saved_tensors
        dout = torch.empty_like(out)
        dgate = torch.zeros_like(gate)                   # dropped assignments keep zero
        _rows_kernel(_dense(g), inverse, dout, gate, out, dgate, ctx.k)
        return dout, dgate, None, None, None, None


def _dense(t):
    """Contiguous and 16-byte aligned (the kernels use 16-byte accesses)."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _rows_kernel(x, inverse, out, gate, other, dgate, k):
    _lib.check(_lib.lib().axb_moe_rows(_lib.ptr(x), _lib.ptr(inverse), _lib.ptr(out), _lib.ptr(gate), _lib.ptr(other),
                                       _lib.ptr(dgate), ctypes.c_int(inverse.numel()), ctypes.c_int(k),
                                       ctypes.c_int(x.shape[1]), _lib.stream_ptr()), "axb_moe_rows")


def _tokens_kernel(buf, dest, gate, T, k):
    H = buf.shape[-1]
    y = torch.empty((T, H), dtype=buf.dtype, device=buf.device)
    _lib.check(_lib.lib().axb_moe_tokens(_lib.ptr(buf), _lib.ptr(dest), _lib.ptr(gate), _lib.ptr(y), ctypes.c_int(T),
                                         ctypes.c_int(k), ctypes.c_int(H), _lib.stream_ptr()), "axb_moe_tokens")
    return y


def route_top_k(logits, top_k, capacity):
    """Router decisions for ``logits`` [T, E].

    Returns (expert index [T, k], gate [T, k] renormalised over the chosen
    experts, slot [T, k] position inside the expert's capacity buffer, keep
    mask [T, k], auxiliary load-balancing loss)."""
    T, E = logits.shape
    probs = F.softmax(logits.float(), dim=-1)
    gate, idx = probs.topk(top_k, dim=-1)
    gate = gate / gate.sum(-1, keepdim=True)
    onehot = F.one_hot(idx.reshape(-1), E)                       # [T*k, E], token-major order
    slot = (onehot.cumsum(0) * onehot).sum(-1).reshape(T, top_k) - 1
    keep = slot < capacity
    # Switch-style balance loss: E * sum_e (fraction of assignments to e) * (mean router prob of e)
    frac = onehot.float().mean(0) * 1.0
    aux = E * (frac * probs.mean(0)).sum()
    return idx, gate, slot, keep, aux


class ExpertParallelMoE(nn.Module):
    """Mixture-of-experts feed-forward layer with whole experts placed on the ranks of ``ep_group`` (default: the
    data-parallel group): top-``top_k`` routing with a per-expert capacity of ``capacity_factor * tokens * top_k /
    n_experts`` rows, dispatch of the routed rows to the experts' ranks, SwiGLU experts as two batched GEMMs over
    all local experts, combine weighted by the gate values.  After a forward, ``last_aux_loss`` (load-balancing
    loss), ``last_drop_fraction``, ``last_assignments_per_expert`` and ``last_dropped_per_expert`` describe the
    routing (device tensors, no host synchronisation)."""

    def __init__(self, hidden, ffn, n_experts=8, top_k=2, capacity_factor=1.25, ep_group=None, dtype=None,
                 init_std=0.02, out_init_std=None):
        super().__init__()
        assert ax.is_initialized
        self.group = ep_group if ep_group is not None else ax.comm_handle.data_parallel_group
        self.ep = dist.get_world_size(self.group)
        self.ep_rank = dist.get_rank(self.group)
        assert n_experts % self.ep == 0, "n_experts must be divisible by the expert-parallel group size"
        self.hidden, self.ffn, self.n_experts, self.top_k = hidden, ffn, n_experts, top_k
        self.n_local = n_experts // self.ep
        self.capacity_factor = capacity_factor
        dev = ax.config.device
        self.router = nn.Parameter(torch.empty(n_experts, hidden, dtype=dtype, device=dev))
        nn.init.normal_(self.router, std=init_std)
        # materialise all experts with the shared RNG stream, keep mine (same weights for any ep size)
        w1 = torch.empty(n_experts, 2 * ffn, hidden, dtype=dtype, device=dev)
        w2 = torch.empty(n_experts, hidden, ffn, dtype=dtype, device=dev)
        nn.init.normal_(w1, std=init_std)
        nn.init.normal_(w2, std=out_init_std or init_std)
        lo, hi = self.ep_rank * self.n_local, (self.ep_rank + 1) * self.n_local
        self.w1 = nn.Parameter(w1[lo:hi].clone())   # [gate|up] interleaved in blocks of 8 rows (ops.swiglu layout)
        self.w2 = nn.Parameter(w2[lo:hi].clone())
        del w1, w2
        for p in (self.w1, self.w2):
            p.is_expert_parallel = self.ep > 1
        self.last_aux_loss = None
        self.last_drop_fraction = None
        self.last_assignments_per_expert = None
        self.last_dropped_per_expert = None

    @torch.no_grad()
    def full_tensor(self, name, t=None):
        """All experts' ``w1`` / ``w2`` (``[n_experts, ...]``; or an optimizer state tensor laid out like them),
        gathered over the expert-parallel group; the router is replicated and returned as it is."""
        t = getattr(self, name).detach() if t is None else t
        if name == "router" or self.ep == 1:
            return t
        out = torch.empty((self.n_experts,) + tuple(t.shape[1:]), dtype=t.dtype, device=t.device)
        dist.all_gather_into_tensor(out, t.contiguous(), group=self.group)
        return out

    @torch.no_grad()
    def shard_tensor(self, name, full):
        if name == "router" or self.ep == 1:
            return full
        return full[self.ep_rank * self.n_local:(self.ep_rank + 1) * self.n_local].clone()

    def _load_from_state_dict(self, state_dict, prefix, *args, **kwargs):
        """Accept ``w1`` / ``w2`` holding all experts (a checkpoint of another grid) as well as the local ones."""
        if self.ep > 1:
            for name in ("w1", "w2"):
                v = state_dict.get(prefix + name)
                if v is not None and v.shape[0] == self.n_experts:
                    state_dict[prefix + name] = self.shard_tensor(name, v)
        super()._load_from_state_dict(state_dict, prefix, *args, **kwargs)

    def capacity(self, tokens):
        c = math.ceil(self.capacity_factor * tokens * self.top_k / self.n_experts)
        return max(8, (c + 7) // 8 * 8)

    def _experts(self, x, seg=None, seg_rows=0):
        """x: [n_local, rows, H] -> [n_local, rows, H].  One launch per GEMM over the tiles of all local experts
        (capacity buffers make the shapes uniform).  ``seg`` (int32 [n_local, rows / seg_rows]): how many rows of
        each ``seg_rows``-row capacity segment hold tokens - the others are zero, and the GEMMs skip the tiles
        (weight gradient: the K blocks) that contain none."""
        return ops.swiglu_experts(x, self.w1, self.w2, seg, seg_rows)

    def _forward_local(self, x2, logits, C):
        """The layer when every expert is on this GPU: same routing, capacity and statistics as the general path; the
        permutations are one kernel each, the expert GEMMs skip the rows of the buffers that hold no token, and
        nothing waits for the host.  The buffers are padded to 64 rows per expert, which the weight-gradient GEMM
        needs of its reduction dimension."""
        T, E, k = x2.shape[0], self.n_experts, self.top_k
        rows = (C + 63) // 64 * 64
        # the kernel reads bf16; under autocast a router whose product is torch's (8 does not divide E) gives autocast's type
        if E <= _ROUTE_MAX_EXPERTS and logits.dtype == torch.bfloat16:
            gate, self.last_aux_loss, dest, inverse, counts, stats = _LocalRoute.apply(logits, k, C, rows)
            self.last_assignments_per_expert, self.last_dropped_per_expert = stats[:E], stats[E:2 * E]
            self.last_drop_fraction = stats[2 * E]
        else:
            probs = F.softmax(logits.float(), dim=-1)
            gate, idx = probs.topk(k, dim=-1)
            gate = gate / gate.sum(-1, keepdim=True)
            idx = idx.contiguous()
            dest, inverse, counts = (torch.empty(n, dtype=torch.int32, device=x2.device) for n in (T * k, E * rows, E))
            assigned = torch.empty(E, dtype=torch.float32, device=x2.device)
            _lib.check(_lib.lib().axb_moe_slots(_lib.ptr(idx), ctypes.c_longlong(T * k), ctypes.c_int(E), ctypes.c_int(C),
                                                ctypes.c_int(rows), _lib.ptr(dest), _lib.ptr(inverse), _lib.ptr(counts),
                                                _lib.ptr(assigned), _lib.stream_ptr()), "axb_moe_slots")
            self.last_aux_loss = E * (assigned / (T * k) * probs.mean(0)).sum()
            kept = counts.float()
            self.last_drop_fraction = 1.0 - kept.sum() / (T * k)
            self.last_assignments_per_expert = assigned
            self.last_dropped_per_expert = assigned - kept
        xin = _LocalDispatch.apply(x2, dest, inverse, E, rows, k)
        out = self._experts(xin, counts.view(E, 1), rows)
        return _LocalCombine.apply(out, gate.contiguous(), dest, inverse, T, k)

    def forward(self, x):
        shape = x.shape
        x2 = x.reshape(-1, self.hidden)
        T = x2.shape[0]
        C = self.capacity(T)
        E, k = self.n_experts, self.top_k
        logits = ops.linear(x2, self.router)
        if (self.ep == 1 and T > 0 and x2.is_cuda and x2.dtype == torch.bfloat16 and self.w1.dtype == x2.dtype
                and self.hidden % 8 == 0):
            return self._forward_local(x2, logits, C).reshape(shape)
        idx, gate, slot, keep, aux = route_top_k(logits, k, C)
        self.last_aux_loss = aux
        self.last_drop_fraction = 1.0 - keep.float().mean().detach()
        # routing statistics of this rank's tokens (device tensors, no host synchronisation): assignments per
        # expert before the capacity cut, and how many of them were dropped per expert
        with torch.no_grad():
            flat_idx = idx.reshape(-1)
            ones = torch.ones(flat_idx.shape, dtype=torch.float32, device=flat_idx.device)
            zeros = torch.zeros(E, dtype=torch.float32, device=flat_idx.device)
            self.last_assignments_per_expert = zeros.index_add(0, flat_idx, ones)
            self.last_dropped_per_expert = zeros.index_add(0, flat_idx, (~keep).reshape(-1).float())
        dest = (idx * C + slot.clamp(max=C - 1)).reshape(-1)           # row in the [E*C, H] send buffer
        keep_f = keep.reshape(-1)
        from . import moe_kernels

        if moe_kernels.usable(self.group, x2):
            y = moe_kernels.dispatch_experts_combine(self, x2, dest, keep_f, gate.reshape(-1), C)
            return y.reshape(shape)
        src_tok = torch.arange(T, device=x.device).repeat_interleave(k)
        send = x2.new_zeros(E * C, self.hidden)
        send = send.index_copy(0, dest[keep_f], x2.index_select(0, src_tok[keep_f]))
        # [E, C, H] = [ep, n_local, C, H]: chunk j goes to rank j; received [ep(src), n_local, C, H]
        recv = _AllToAll.apply(send.reshape(self.ep, self.n_local * C, self.hidden), self.group)
        recv = recv.reshape(self.ep, self.n_local, C, self.hidden).transpose(0, 1)
        out = self._experts(recv.reshape(self.n_local, self.ep * C, self.hidden))
        out = out.reshape(self.n_local, self.ep, C, self.hidden).transpose(0, 1)
        back = _AllToAll.apply(out.reshape(self.ep, self.n_local * C, self.hidden), self.group)
        back = back.reshape(E * C, self.hidden)
        picked = back.index_select(0, dest) * (gate.reshape(-1) * keep_f).to(back.dtype)[:, None]
        y = picked.reshape(T, k, self.hidden).sum(1)
        return y.reshape(shape)
