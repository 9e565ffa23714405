"""Tensor-parallel SwiGLU MLP block (Llama-3-70B shape by default: d=8192, ffn=28672) with
sequence-parallel activations: all-gather -> GEMM for the gate/up projection, GEMM ->
reduce-scatter for the down projection, both single fused kernels.

Reference parity: none -- the reference ships no model and no GEMM; baseline for these layers
is cuBLAS + NCCL.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from ..ops.gemm import gemm_swiglu
from ..ops.elementwise import swiglu
from ..parallel.tp import ColumnParallelLinear, RowParallelLinear


class TPMLP(nn.Module):
    def __init__(self, comm, dim: int = 8192, ffn_dim: int = 28672, device="cuda"):
        super().__init__()
        self.comm, self.ffn_local = comm, ffn_dim // comm.nranks
        # gate and up projections share one column-parallel GEMM: rows [0, ffn_local) = gate
        self.w13 = ColumnParallelLinear(dim, 2 * ffn_dim, comm, device=device)
        self.w2 = RowParallelLinear(ffn_dim, dim, comm, device=device)

    def forward(self, x_shard: torch.Tensor) -> torch.Tensor:
        """x_shard: bf16 [tokens / tp, dim] -> bf16 [tokens / tp, dim]"""
        plain = type(self.w13) is ColumnParallelLinear and "forward" not in self.w13.__dict__ and not self.w13._forward_hooks and not self.w13._forward_pre_hooks
        w = self.w13.weight if plain else None
        if (plain and self.comm.nranks == 1 and x_shard.is_cuda and self.ffn_local % 8 == 0
                and not (torch.is_grad_enabled() and (x_shard.requires_grad or w.requires_grad))):
            # one rank, no gradients: the activation rides in the projection's epilogue (a projection that a
            # program wrapped, hooked or replaced is called as the module that it is)
            return self.w2(gemm_swiglu(x_shard.contiguous(), w.contiguous()))
        return self.w2(swiglu(self.w13(x_shard)).to(torch.bfloat16))
