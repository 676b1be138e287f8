"""When an operation may launch its kernel without an autograd function around it.

The function costs more host time than the launch (4 us against 5 us, and as much again in reshapes and saved tensors), and
evaluating a model without gradients is bound by host time for short prompts."""

import torch
from torch.autograd import forward_ad

_PLAIN = (torch.Tensor, torch.nn.Parameter)


def no_graph(*tensors) -> bool:
    """No gradient can be asked of an operation on ``tensors`` (``None`` entries are skipped) and nothing looks at it from
    outside: grad mode is off or none of them requires a gradient, they are ordinary CUDA tensors, and no tracer, compiler,
    function transform or forward-mode level is active."""
    grad = torch.is_grad_enabled()
    for t in tensors:
        if t is not None and (type(t) not in _PLAIN or not t.is_cuda or (grad and t.requires_grad)):
            return False
    return (not torch._C._are_functorch_transforms_active() and torch._C._get_tracing_state() is None
            and forward_ad._current_level < 0 and not torch.compiler.is_compiling())
