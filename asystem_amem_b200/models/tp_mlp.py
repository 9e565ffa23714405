"""Tensor-parallel SwiGLU MLP block (Llama-3-70B shape by default: d=8192, ffn=28672) with
sequence-parallel activations: all-gather -> GEMM for the gate/up projection, GEMM ->
reduce-scatter for the down projection, both single fused kernels.

Reference parity: none -- the reference ships no model and no GEMM; baseline for these layers
is cuBLAS + NCCL.
"""
from __future__ import annotations

import torch
import torch.nn as nn
from torch.nn.modules.module import _has_any_global_hook

from ..ops.gemm import gemm_swiglu
from ..ops.elementwise import swiglu
from ..ops.operands import tangents_about
from ..parallel.tp import ColumnParallelLinear, RowParallelLinear


def _calls_its_product_alone(m: nn.Module) -> bool:
    """Whether m(x) is a projection's product on one rank and nothing else: neither wrapped, hooked nor replaced."""
    return (type(m) is ColumnParallelLinear and "forward" not in m.__dict__ and not m._forward_hooks and not m._forward_pre_hooks
            and m.comm.nranks == 1 and not _has_any_global_hook())


class TPMLP(nn.Module):
    def __init__(self, comm, dim: int = 8192, ffn_dim: int = 28672, device="cuda"):
        super().__init__()
        self.comm, self.ffn_local = comm, ffn_dim // comm.nranks
        # gate and up projections share one column-parallel GEMM: rows [0, ffn_local) = gate
        self.w13 = ColumnParallelLinear(dim, 2 * ffn_dim, comm, device=device)
        self.w2 = RowParallelLinear(ffn_dim, dim, comm, device=device)

    def forward(self, x_shard: torch.Tensor) -> torch.Tensor:
        """x_shard: bf16 [tokens / tp, dim] -> bf16 [tokens / tp, dim]"""
        if x_shard.is_cuda and self.ffn_local % 8 == 0:
            w13 = self.w13
            if _calls_its_product_alone(w13) and not tangents_about():
                w = w13.weight
                if not (torch.is_grad_enabled() and (x_shard.requires_grad or w.requires_grad)):
                    # one rank, no gradients: the activation rides in the projection's epilogue
                    return self.w2(gemm_swiglu(x_shard.contiguous(), w.contiguous(), comm=w13.comm))
        return self.w2(swiglu(self.w13(x_shard)).to(torch.bfloat16))
