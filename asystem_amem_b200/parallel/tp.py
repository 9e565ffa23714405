"""Tensor parallelism with sequence parallelism (Megatron style) on the fused GEMM kernels.

Activations between the two linears of a block are sharded by rows (tokens).  The
column-parallel linear all-gathers them inside its GEMM kernel; the row-parallel linear
reduce-scatters its output from the GEMM epilogue.  Backward uses the mirrored fused kernels
for the activation gradients and the library's own tcgen05 GEMM for the weight gradients.

Reference parity: none to match -- tensor parallelism appears in the reference only as
integration text (README.md:279-293, SGLang's tensor-model-parallel group); its users run
cuBLAS and NCCL back to back.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from ..ops.gemm import all_gather_gemm, gemm_input_grad, gemm_reduce_scatter, gemm_weight_grad


def _wgrad(gy: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    """gw[N, K] = gy[M, N].T @ x[M, K] on the library's tcgen05 GEMM, which reads both operands as they lie."""
    if gy.is_cuda and gy.dtype == torch.bfloat16 and x.dtype == torch.bfloat16:
        return gemm_weight_grad(gy.contiguous(), x.contiguous())
    return gy.t() @ x


def _gathered(comm, shard: torch.Tensor) -> torch.Tensor:
    """The rows of every rank (the shard itself on one rank)."""
    shard = shard.contiguous()
    if comm.nranks == 1:
        return shard
    full = torch.empty(shard.shape[0] * comm.nranks, shard.shape[1], dtype=shard.dtype, device=shard.device)
    comm.all_gather(shard, full)
    return full


class _ColumnFn(torch.autograd.Function):
    """y[M, N_local] = all_gather_rows(x_shard)[M, K] @ w[N_local, K].T"""

    @staticmethod
    def forward(ctx, x_shard, w, comm):
        ctx.comm = comm
        ctx.save_for_backward(x_shard, w)
        return all_gather_gemm(comm, x_shard.contiguous(), w.contiguous())

    @staticmethod
    def backward(ctx, gy):
        comm = ctx.comm
        x_shard, w = ctx.saved_tensors
        gy = gy.contiguous()
        # dx_shard = reduce_scatter_rows(gy @ w): the mirrored fused kernel, B = w.T [K, N_local]; one
        # rank has nothing to scatter and its GEMM reads w as it lies
        gx = gemm_input_grad(gy, w.contiguous(), comm=comm) if comm.nranks == 1 else gemm_reduce_scatter(comm, gy, w.t().contiguous())
        gw = _wgrad(gy, _gathered(comm, x_shard))
        return gx, gw, None


class _RowFn(torch.autograd.Function):
    """y_shard[M / n, N] = reduce_scatter_rows(x[M, K_local] @ w[N, K_local].T)"""

    @staticmethod
    def forward(ctx, x, w, comm):
        ctx.comm = comm
        ctx.save_for_backward(x, w)
        return gemm_reduce_scatter(comm, x.contiguous(), w.contiguous())

    @staticmethod
    def backward(ctx, gy_shard):
        comm = ctx.comm
        x, w = ctx.saved_tensors
        gy_shard = gy_shard.contiguous()
        # dx = all_gather_rows(gy_shard) @ w  -> fused all-gather GEMM with B = w.T [K_local, N]
        gx = gemm_input_grad(gy_shard, w.contiguous(), comm=comm) if comm.nranks == 1 else all_gather_gemm(comm, gy_shard, w.t().contiguous())
        gw = _wgrad(_gathered(comm, gy_shard), x)
        return gx, gw, None


class ColumnParallelLinear(nn.Module):
    """Weight [out_features / tp, in_features]; input rows sharded over the TP group."""

    def __init__(self, in_features: int, out_features: int, comm, device="cuda", std: float = 0.02):
        super().__init__()
        assert out_features % comm.nranks == 0
        self.comm = comm
        self.weight = nn.Parameter(torch.randn(out_features // comm.nranks, in_features, device=device, dtype=torch.bfloat16) * std)

    def forward(self, x_shard):
        return _ColumnFn.apply(x_shard, self.weight, self.comm)


class RowParallelLinear(nn.Module):
    """Weight [out_features, in_features / tp]; output rows sharded over the TP group."""

    def __init__(self, in_features: int, out_features: int, comm, device="cuda", std: float = 0.02):
        super().__init__()
        assert in_features % comm.nranks == 0
        self.comm = comm
        self.weight = nn.Parameter(torch.randn(out_features, in_features // comm.nranks, device=device, dtype=torch.bfloat16) * std)

    def forward(self, x):
        return _RowFn.apply(x, self.weight, self.comm)
