"""Expert parallelism with gradients, on the fused dispatch / combine kernels.

Forward of one MoE layer on every rank of the expert-parallel communicator::

    rows[pos(t, c)] = x[t]                      dispatch  (permute inside the all-to-all)
    y               = experts(rows)             local, grouped by expert
    out[t]          = sum_c w[t, c] * y[pos(t, c)]   combine (un-permute + weighted sum)

Both communication steps are linear maps whose transposes are each other, so the backward pass
runs on the same two kernels and needs no new device code:

* d out / d y  : ``g_y[pos(t, c)] = w[t, c] * g_out[t]`` is a dispatch of the ``T * k`` scaled
  rows with one choice per row.  The kernels place rows by (expert, source rank, pair order), and
  the flattened pair order of the ``[T * k, 1]`` problem is the pair order of the ``[T, k]`` one,
  so every row lands exactly where its forward row was.
* d out / d w  : ``g_w[t, c] = <g_out[t], y[pos(t, c)]>`` needs the expert outputs back at their
  tokens: a combine of the ``[T * k, 1]`` problem with unit weights is that gather.
* d rows / d x : ``g_x[t] = sum_c g_rows[pos(t, c)]`` is a combine with unit weights.

On one rank nothing has to travel: the steps then run between the caller's tensors, and the backward of
the combine is one kernel (``MoeDispatcher.combine_grad_local``).

The four steps are plain functions (``dispatch_forward`` ... ``combine_backward``) so that a
caller which schedules its own backward pass -- or a test that runs several ranks as threads of
one process, where the autograd engine's single per-device thread could not run the ranks'
collectives side by side -- can call them directly; ``ep_dispatch`` / ``ep_combine`` wrap them
as autograd functions for everybody else.  Every rank must run the same sequence of steps.

The reference library stops at the communication layer (its all-to-all is NCCL's grouped
send/recv kept alive across ncclPause/ncclResume); routing, permutation and their gradients are
left to the training framework above it.
"""
from __future__ import annotations

import torch

from ..ops.moe import (DispatchResult, MoeDispatcher, _kernel_routes, _route_grads_torch, _route_launch, _route_logits_grad,  # noqa: F401
                       route)
from ..ops.operands import dense


def _between_tensors(disp: MoeDispatcher, rows: torch.Tensor) -> bool:
    """Whether a one-rank step reads ``rows`` where they are; more of them than the dispatcher's buffers
    hold are left to the general form, which refuses them."""
    return disp.local(rows) and rows.shape[0] <= disp.capacity


def dispatch_forward(disp: MoeDispatcher, x: torch.Tensor, idx: torch.Tensor, all_routed: bool = False):
    """Returns (rows, expert_offsets, send_pos, total): ``rows`` is a private copy of the
    received rows (the receive buffer is reused by the next dispatch).  ``all_routed``: every entry of ``idx`` names an
    expert, so that one rank knows the total without reading it back."""
    local = disp.local(x) and x.shape[0] == idx.shape[0]
    res = disp.dispatch_local(x.contiguous(), idx) if local else disp.dispatch(x.contiguous(), idx)
    if local and all_routed:
        return res.recv_x, res.expert_offsets, res.send_pos, res.recv_x.shape[0]
    total = int(res.expert_offsets[-1].item())  # host sync: `rows` has exactly the rows that arrived
    # (shrunk, not sliced: a view made inside an autograd function could not be changed in place)
    rows = res.recv_x.resize_(total, disp.d) if local else res.recv_x[:total].clone()
    return rows, res.expert_offsets, res.send_pos, total


def dispatch_backward(disp: MoeDispatcher, g_rows: torch.Tensor, idx: torch.Tensor, send_pos: torch.Tensor) -> torch.Tensor:
    T, k = idx.shape
    ones = torch.ones(T, k, dtype=torch.float32, device=g_rows.device)
    if _between_tensors(disp, g_rows):
        return disp.combine_local(g_rows, idx, ones, send_pos)
    disp.y[: g_rows.shape[0]] = g_rows.to(torch.bfloat16)
    return disp.combine(idx, ones, send_pos)


def combine_forward(disp: MoeDispatcher, y_rows: torch.Tensor, idx: torch.Tensor, w: torch.Tensor, send_pos: torch.Tensor) -> torch.Tensor:
    if _between_tensors(disp, y_rows):
        return disp.combine_local(y_rows, idx, w, send_pos)
    disp.y[: y_rows.shape[0]] = y_rows.to(torch.bfloat16)
    return disp.combine(idx, w, send_pos)


def combine_backward(disp: MoeDispatcher, g_out: torch.Tensor, y_rows: torch.Tensor, idx: torch.Tensor, w: torch.Tensor,
                     send_pos: torch.Tensor):
    """Returns (g_y_rows, g_w)."""
    if disp.local(g_out) and _between_tensors(disp, y_rows) and w.shape == idx.shape and g_out.shape[0] == idx.shape[0]:
        return disp.combine_grad_local(g_out, y_rows, w, send_pos)
    T, k = idx.shape
    d = g_out.shape[1]
    flat_idx = idx.reshape(T * k, 1)
    # expert outputs back at their (token, choice): the gather for the routing-weight gradient
    disp.y[: y_rows.shape[0]] = y_rows.to(torch.bfloat16)
    ones = torch.ones(T * k, 1, dtype=torch.float32, device=g_out.device)
    y_at = disp.combine(flat_idx, ones, send_pos.reshape(T * k))
    g_w = (y_at.view(T, k, d).float() * g_out.float().unsqueeze(1)).sum(-1)
    # scaled output gradients to the experts, landing row for row where the forward rows were
    scaled = (g_out.float().unsqueeze(1) * w.float().unsqueeze(2)).to(torch.bfloat16).view(T * k, d)
    res = disp.dispatch(scaled, flat_idx)
    return res.recv_x[: y_rows.shape[0]].clone(), g_w


class _Dispatch(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, idx, disp, all_routed):
        rows, offsets, send_pos, _ = dispatch_forward(disp, x, idx, all_routed)
        ctx.disp = disp
        ctx.save_for_backward(idx, send_pos)
        ctx.mark_non_differentiable(offsets, send_pos)
        return rows, offsets, send_pos

    @staticmethod
    def backward(ctx, g_rows, _g_off, _g_pos):
        idx, send_pos = ctx.saved_tensors
        return dispatch_backward(ctx.disp, g_rows.contiguous(), idx, send_pos), None, None, None


class _RouteDispatch(torch.autograd.Function):
    """Routing and dispatch of one rank as one step, so that the tokens' gradient, which comes through both, is one sum."""

    @staticmethod
    def forward(ctx, x, router, disp, k):
        idx, w = _route_launch(x, router, k)
        rows, offsets, send_pos, _ = dispatch_forward(disp, x, idx, all_routed=True)
        ctx.disp = disp
        ctx.save_for_backward(x, router, idx, w, send_pos)
        ctx.mark_non_differentiable(offsets, send_pos, idx)
        return rows, offsets, send_pos, idx, w

    @staticmethod
    def backward(ctx, g_rows, _g_off, _g_pos, _g_idx, g_w):
        x, router, idx, w, send_pos = ctx.saved_tensors
        of_x, of_router = ctx.needs_input_grad[:2]
        g_x = g_router = None
        if torch.is_grad_enabled():     # a graph of the routing's gradient is wanted: torch's operators make one
            if of_x or of_router:
                g_x, g_router = _route_grads_torch(x, router, idx, g_w, of_x, of_router)
            return (g_x + dispatch_backward(ctx.disp, g_rows.contiguous(), idx, send_pos) if of_x else None), g_router, None, None
        w, idx, send_pos, router = map(dense, (w, idx, send_pos, router))
        g_logits = _route_logits_grad(g_w.contiguous(), w, idx, router.shape[0])
        if of_x:
            g_x = ctx.disp.input_grad_local(dense(g_rows), send_pos, idx, g_logits, router)
        if of_router:
            g_router = g_logits.t() @ x
        return g_x, g_router, None, None


class _Combine(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y_rows, w, idx, send_pos, disp):
        ctx.disp = disp
        ctx.save_for_backward(y_rows, w, idx, send_pos)
        return combine_forward(disp, y_rows, idx, w, send_pos)

    @staticmethod
    def backward(ctx, g_out):
        y_rows, w, idx, send_pos = ctx.saved_tensors
        g_y, g_w = combine_backward(ctx.disp, g_out.contiguous(), y_rows, idx, w, send_pos)
        return g_y, g_w.to(w.dtype), None, None, None


def ep_dispatch(disp: MoeDispatcher, x: torch.Tensor, idx: torch.Tensor, all_routed: bool = False):
    """Differentiable dispatch: (rows grouped by local expert, expert_offsets, send_pos).  ``all_routed``: the caller knows
    that every entry of ``idx`` names an expert (see :func:`dispatch_forward`)."""
    return _Dispatch.apply(x, idx.to(torch.int32).contiguous(), disp, all_routed)


def ep_route_dispatch(disp: MoeDispatcher, x: torch.Tensor, router: torch.Tensor, k: int):
    """Differentiable routing (:func:`ops.moe.route`) and dispatch: (rows grouped by local expert, expert_offsets, send_pos, idx,
    w).  One step where one rank's kernels take ``x`` and ``router`` and ``x`` wants a gradient, the two otherwise (as outputs of one
    step the rows would want a gradient for the router's sake, and the experts would compute it)."""
    if x.requires_grad and disp.local(x) and router.shape[0] == disp.E and _kernel_routes(x, router, k):
        return _RouteDispatch.apply(x, router, disp, k)
    idx, w = route(x, router, k)
    return *ep_dispatch(disp, x, idx, all_routed=router.shape[0] == disp.E), idx, w


def ep_combine(disp: MoeDispatcher, y_rows: torch.Tensor, w: torch.Tensor, idx: torch.Tensor, send_pos: torch.Tensor) -> torch.Tensor:
    """Differentiable combine of the experts' outputs (rows in dispatch order) with weights ``w``."""
    return _Combine.apply(y_rows, w, idx.to(torch.int32).contiguous(), send_pos, disp)
