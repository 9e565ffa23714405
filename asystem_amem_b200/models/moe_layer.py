"""Expert-parallel MoE layer: top-k softmax routing, fused dispatch (permute inside the
all-to-all), the experts' SwiGLU FFN as two grouped tcgen05 GEMMs over all local experts at once
(group boundaries read on the device from the dispatch's ``expert_offsets``), fused combine
(un-permute + weighted sum while pulling the rows back).

Without gradients nothing of a layer's forward returns to the host: dispatch -> grouped GEMM with
the SwiGLU epilogue -> grouped GEMM straight into the combine buffer -> combine.  With gradients
the two communication steps run as autograd functions whose backward passes reuse the same kernels
(parallel/ep.py) and the expert GEMMs are :class:`GroupedLinear` (output, input gradient and weight
gradient each one grouped launch that reads the group boundaries on the device).

Reference parity: none -- the reference keeps NCCL's all-to-all buffers alive across
ncclPause / ncclResume (README.md:132) and leaves the layer to the framework above it."""
from __future__ import annotations

import torch
import torch.nn as nn

from ..ops.gemm import grouped_gemm_bf16, grouped_gemm_input_grad, grouped_gemm_weight_grad, interleave_gate_up
from ..ops.elementwise import swiglu
from ..ops.moe import MoeDispatcher, route
from ..ops.operands import dense
from ..parallel.ep import ep_combine, ep_route_dispatch


class GroupedLinear(torch.autograd.Function):
    """out[rows of group e] = rows @ w[e].T for every group, differentiable.  ``covered``: every row belongs to a group, so
    that the gradient of the rows needs no zeros underneath."""

    @staticmethod
    def forward(ctx, rows, w, offsets, covered=False):
        ctx.save_for_backward(rows, w, offsets)
        ctx.covered = covered
        return grouped_gemm_bf16(rows.contiguous(), w.contiguous(), offsets, rows_hint=rows.shape[0])

    @staticmethod
    def backward(ctx, g_out):
        rows, w, offsets = ctx.saved_tensors
        g_out = dense(g_out)
        g_rows = g_w = None
        if ctx.needs_input_grad[0]:
            g_rows = torch.empty_like(rows) if ctx.covered else torch.zeros_like(rows)
            grouped_gemm_input_grad(g_out, w.contiguous(), offsets, out=g_rows, rows_hint=rows.shape[0])
        if ctx.needs_input_grad[1]:
            g_w = grouped_gemm_weight_grad(g_out, rows.contiguous(), offsets)
        return g_rows, g_w, None, None


class MoELayer(nn.Module):
    def __init__(self, ep_comm, dim: int = 4096, ffn_dim: int = 1536, num_experts: int = 64, top_k: int = 8,
                 tokens_per_rank: int = 16384, capacity_factor: float = 2.0, device="cuda", seed: int = 0):
        super().__init__()
        self.comm, self.E, self.k, self.dim = ep_comm, num_experts, top_k, dim
        self.El = num_experts // ep_comm.nranks
        g = torch.Generator(device="cpu").manual_seed(seed)
        self.router = nn.Parameter((torch.randn(num_experts, dim, generator=g) * 0.02).to(device=device, dtype=torch.bfloat16))
        base = ep_comm.rank * self.El
        ge = torch.Generator(device="cpu").manual_seed(seed + 1 + base)
        self.w13 = nn.Parameter((torch.randn(self.El, 2 * ffn_dim, dim, generator=ge) * 0.02).to(device=device, dtype=torch.bfloat16))
        self.w2 = nn.Parameter((torch.randn(self.El, dim, ffn_dim, generator=ge) * 0.02).to(device=device, dtype=torch.bfloat16))
        cap = int(capacity_factor * tokens_per_rank * top_k)
        self.dispatcher = MoeDispatcher(ep_comm, num_experts, dim, cap)
        self.ffn_dim = ffn_dim
        self.tokens_hint = tokens_per_rank * top_k
        self._w13_fused = None          # (version of w13, gate / up rows interleaved for the SwiGLU epilogue)
        self.last_dropped = None        # int32 [1] on the device: rows this rank could not take in the last forward

    def _fused_w13(self) -> torch.Tensor:
        v = self.w13._version
        if self._w13_fused is None or self._w13_fused[0] != v:
            self._w13_fused = (v, interleave_gate_up(self.w13.detach(), self.ffn_dim))
        return self._w13_fused[1]

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        fusable = self.ffn_dim % 32 == 0 and x.is_cuda
        if torch.is_grad_enabled() and (x.requires_grad or self.w2.requires_grad):
            rows, offsets, send_pos, idx, w = ep_route_dispatch(self.dispatcher, x, self.router, self.k)
            h = GroupedLinear.apply(rows, self.w13, offsets, True)      # `rows` are the rows of the groups and no more
            y = GroupedLinear.apply(swiglu(h).to(torch.bfloat16), self.w2, offsets, True)
            return ep_combine(self.dispatcher, y, w, idx, send_pos)
        idx, w = route(x, self.router, self.k)
        res = self.dispatcher.dispatch(x.contiguous(), idx)
        self.last_dropped = res.dropped
        if fusable:
            a = grouped_gemm_bf16(res.recv_x, self._fused_w13(), res.expert_offsets, rows_hint=self.tokens_hint, swiglu=True)
        else:
            h = grouped_gemm_bf16(res.recv_x, self.w13.detach(), res.expert_offsets, rows_hint=self.tokens_hint)
            a = swiglu(h).to(torch.bfloat16)
        # the second GEMM writes the experts' outputs where the combine reads them
        grouped_gemm_bf16(a, self.w2.detach(), res.expert_offsets, out=self.dispatcher.y, rows_hint=self.tokens_hint)
        return self.dispatcher.combine(idx, w, res.send_pos)
