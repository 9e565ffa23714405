"""How the kernels want their operands: rows without gaps that start on a 16-byte boundary, and the
device that holds them current."""
from __future__ import annotations

from functools import wraps

import torch
from torch.autograd import forward_ad


def on_operands_device(launch):
    """``launch(t, ...)`` with the device of ``t`` current: a launch goes to the current device, wherever its
    operands lie."""
    @wraps(launch)
    def call(t, *args, **kw):
        if t.is_cuda and t.get_device() != torch.cuda.current_device():
            with torch.cuda.device(t.get_device()):
                return launch(t, *args, **kw)
        return launch(t, *args, **kw)
    return call


def tangents_about() -> bool:
    """Whether a tensor may carry a forward-mode tangent, which the kernels know nothing of."""
    return forward_ad._current_level >= 0


def dense(t: torch.Tensor) -> torch.Tensor:
    """``t`` where it is contiguous and starts on 16 bytes (the kernels move 16-byte vectors), a copy of
    it otherwise: a contiguous view may start at any element."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()
