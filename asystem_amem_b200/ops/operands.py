"""How the kernels want their operands: rows without gaps that start on a 16-byte boundary, and the
device that holds them current."""
from __future__ import annotations

from contextlib import nullcontext

import torch


def on_device_of(t: torch.Tensor):
    """Context in which the device of ``t`` is current: a launch goes to the current device, wherever
    its operands lie."""
    return nullcontext() if t.get_device() == torch.cuda.current_device() else torch.cuda.device(t.get_device())


def dense(t: torch.Tensor) -> torch.Tensor:
    """``t`` where it is contiguous and starts on 16 bytes (the kernels move 16-byte vectors), a copy of
    it otherwise: a contiguous view may start at any element."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()
