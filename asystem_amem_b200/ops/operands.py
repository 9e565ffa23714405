"""How the kernels want their operands: rows without gaps that start on a 16-byte boundary, and the
device that holds them current."""
from __future__ import annotations

from functools import wraps

import torch
from torch.autograd import forward_ad


def on_operands_device(launch):
    """``launch`` with the device of its first tensor current: a launch goes to the current device, wherever
    its operands lie."""
    @wraps(launch)
    def call(*args, **kw):
        t = args[0] if args else next((v for v in kw.values() if isinstance(v, torch.Tensor)), None)
        if t is not None and t.is_cuda and t.get_device() != torch.cuda.current_device():
            with torch.cuda.device(t.get_device()):
                return launch(*args, **kw)
        return launch(*args, **kw)
    return call


def current_stream() -> int:
    """Handle of the current stream: without the Stream object, whose making takes 3 us of a launch's 12."""
    if torch.cuda.is_initialized():
        return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())
    return torch.cuda.current_stream().cuda_stream


def tangents_about() -> bool:
    """Whether a tensor may carry a forward-mode tangent, which the kernels know nothing of."""
    return forward_ad._current_level >= 0


def concrete(*values) -> bool:
    """Whether ``values`` are tensors: a symbolic tracer hands stand-ins through, of which no branch can be asked."""
    for v in values:
        if not isinstance(v, torch.Tensor):
            return False
    return True


def plain_cuda(*tensors: torch.Tensor) -> bool:
    """Whether ``tensors`` are ordinary tensors of one GPU in a program that runs eagerly: what a kernel that
    autograd knows only as a :class:`torch.autograd.Function` can take.  Subclasses, tracing, dispatch modes
    and function transforms (vmap, forward mode) need torch's own operators."""
    if torch.compiler.is_compiling():       # (first: a compiler follows no further)
        return False
    device = tensors[0].device
    return (device.type == "cuda" and all(type(t) in (torch.Tensor, torch.nn.Parameter) and t.device == device for t in tensors)
            and not tangents_about() and torch._C._functorch.peek_interpreter_stack() is None and torch._C._len_torch_dispatch_stack() == 0
            and not torch.jit.is_tracing())


def apart(*tensors: torch.Tensor) -> list[torch.Tensor]:
    """A view of each of ``tensors``, which autograd tells apart even where they are one tensor or one is computed from another:
    derivatives with respect to the views are the partial ones that a backward function owes."""
    return [t.view_as(t) for t in tensors]


def dense(t: torch.Tensor) -> torch.Tensor:
    """``t`` where it is contiguous and starts on 16 bytes (the kernels move 16-byte vectors), a copy of
    it otherwise: a contiguous view may start at any element."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()
