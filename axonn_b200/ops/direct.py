"""When a kernel may stand in for a call: for an autograd function (``no_graph``), for the call of a layer (``plain_layer``).

An autograd function costs more host time than the launch (4 us against 5 us, and as much again in reshapes and saved tensors),
and evaluating a model without gradients is bound by host time for short prompts."""

import functools

import torch
from torch.autograd import forward_ad

from . import _lib

_PLAIN = (torch.Tensor, torch.nn.Parameter)
_module = torch.nn.modules.module
_CALL = torch.nn.Module.__call__
_own_forward = {}


def no_graph(*tensors) -> bool:
    """No gradient can be asked of an operation on ``tensors`` (``None`` entries are skipped) and nothing looks at it from
    outside: grad mode is off or none of them requires a gradient, and they are ``plain_tensors`` (written out here: a call
    costs 0.4 us, in each of the twenty operations of a small model)."""
    grad = torch.is_grad_enabled()
    for t in tensors:
        if t is not None and (type(t) not in _PLAIN or not t.is_cuda or (grad and t.requires_grad)):
            return False
    return (not torch._C._are_functorch_transforms_active() and torch._C._get_tracing_state() is None
            and forward_ad._current_level < 0 and not torch.compiler.is_compiling())


def plain_tensors(*tensors) -> bool:
    """Ordinary CUDA tensors (``None`` entries are skipped) while no tracer, compiler, function transform or forward-mode level
    is active."""
    for t in tensors:
        if t is not None and (type(t) not in _PLAIN or not t.is_cuda):
            return False
    return (not torch._C._are_functorch_transforms_active() and torch._C._get_tracing_state() is None
            and forward_ad._current_level < 0 and not torch.compiler.is_compiling())


def host_paths():
    """The native host paths (``_lib.host``) while neither a compiler nor a forward-mode level is active - they ask everything else
    themselves -, otherwise ``None``."""
    return None if forward_ad._current_level >= 0 or torch.compiler.is_compiling() else _lib.host()


def own_forward(cls):
    """Class decorator: calls of such layers may be replaced (see ``plain_layer``) while ``cls.forward`` is what it is now."""
    _own_forward[cls] = cls.forward
    return cls


def plain_layer(layer) -> bool:
    """Is calling ``layer`` nothing but the forward that its class was defined with?  Of a class marked with ``own_forward`` and no
    other, its forward replaced neither on the instance nor on the class, neither hooks nor a compiled call in its way."""
    cls = type(layer)
    return (cls in _own_forward and cls.forward is _own_forward[cls] and cls.__call__ is _CALL and "forward" not in layer.__dict__
            and layer._compiled_call_impl is None
            and not (layer._forward_hooks or layer._forward_pre_hooks or layer._backward_hooks or layer._backward_pre_hooks
                     or _module._has_any_global_hook()))


class _SecondDerivative(torch.autograd.Function):
    """``outs`` as they are, as functions of ``inputs`` without a derivative."""

    @staticmethod
    def forward(ctx, what, n, *tensors):
        ctx.what = what
        return tuple(t if t is None else t.detach() for t in tensors[:n])

    @staticmethod
    def backward(ctx, *_):
        raise RuntimeError(f"{ctx.what}: second derivatives are not implemented")


def first_derivative_only(backward):
    """Decorator of a ``Function.backward`` whose gradients come from kernels that leave no graph: differentiating them by what the
    function was called with is an error, whatever they are added to.  (After ``once_differentiable`` they count as constants when the
    incoming gradient needs none, which is how a loss that is a sum begins, and for ``torch.autograd.grad``, which walks only the part
    of the graph that leads to the tensors it is given.)  The saved tensors stand for the inputs."""
    @functools.wraps(backward)
    def wrapper(ctx, *grads):
        with torch.no_grad():
            out = backward(ctx, *grads)
        if not torch.is_grad_enabled():
            return out
        outs = out if isinstance(out, tuple) else (out,)
        return _SecondDerivative.apply(type(ctx).__name__, len(outs), *outs, *grads, *ctx.saved_tensors)
    return wrapper
