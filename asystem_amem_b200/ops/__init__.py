"""Fused operations: tcgen05 GEMM and its tensor-parallel forms, MoE dispatch/combine."""
from .gemm import (all_gather_gemm, gemm_bf16, gemm_input_grad, gemm_reduce_scatter, gemm_swiglu, gemm_weight_grad, grouped_gemm_bf16,  # noqa: F401
                   grouped_gemm_input_grad, grouped_gemm_weight_grad, interleave_gate_up)
from .elementwise import adamw_step, embedding, gated, rms_norm, rotate, swiglu  # noqa: F401
from .moe import DispatchResult, MoeDispatcher, route  # noqa: F401,E402
