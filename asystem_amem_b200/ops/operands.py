"""How the kernels want their operands: rows without gaps that start on a 16-byte boundary."""
from __future__ import annotations

import torch


def dense(t: torch.Tensor) -> torch.Tensor:
    """``t`` where it is contiguous and starts on 16 bytes (the kernels move 16-byte vectors), a copy of
    it otherwise: a contiguous view may start at any element."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()
