"""Tensor-parallel SwiGLU MLP block (Llama-3-70B shape by default: d=8192, ffn=28672) with
sequence-parallel activations: all-gather -> GEMM for the gate/up projection, GEMM ->
reduce-scatter for the down projection, both single fused kernels.

Reference parity: none -- the reference ships no model and no GEMM; baseline for these layers
is cuBLAS + NCCL.
"""
from __future__ import annotations

import torch
import torch.nn as nn
from torch.autograd import forward_ad
from torch.nn.modules.module import _has_any_global_hook

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

    def _calls_nothing_else(self, x_shard: torch.Tensor) -> bool:
        """Whether w13(x_shard) is the projection's product alone: no gradient of either mode asks for it, and it is
        neither wrapped, hooked nor replaced."""
        m = self.w13
        if type(m) is not ColumnParallelLinear or "forward" in m.__dict__ or m._forward_hooks or m._forward_pre_hooks or _has_any_global_hook():
            return False
        if torch.is_grad_enabled() and (x_shard.requires_grad or m.weight.requires_grad):
            return False
        return all(forward_ad.unpack_dual(t).tangent is None for t in (x_shard, m.weight))

    def forward(self, x_shard: torch.Tensor) -> torch.Tensor:
        """x_shard: bf16 [tokens / tp, dim] -> bf16 [tokens / tp, dim]"""
        if self.comm.nranks == 1 and x_shard.is_cuda and self.ffn_local % 8 == 0 and self._calls_nothing_else(x_shard):
            # one rank: the activation rides in the projection's epilogue
            self.w13.comm.begin(x_shard)
            return self.w2(gemm_swiglu(x_shard.contiguous(), self.w13.weight.contiguous()))
        return self.w2(swiglu(self.w13(x_shard)).to(torch.bfloat16))
