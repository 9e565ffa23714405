"""Passes over rows as single kernels: SwiGLU, the root-mean-square norm and the rotary embedding with their
gradients, an embedding's gradient, the sum of gradients into a shard and its AdamW update.

Reference parity: none -- the reference contains no arithmetic on user data.
"""
from __future__ import annotations

import ctypes

import torch
import torch.nn.functional as F

from .. import bindings as B
from .operands import apart, concrete, current_stream, dense, on_operands_device, plain_cuda, tangents_about


def _fused(h: torch.Tensor) -> bool:
    return not tangents_about() and h.is_cuda and h.dtype == torch.bfloat16 and h.dim() == 2 and h.shape[1] % 16 == 0 and h.data_ptr() % 16 == 0


class _SwiGLU(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h):
        ctx.save_for_backward(h)
        return _forward(h)

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, g):
        (h,) = ctx.saved_tensors
        return _gradient(dense(h), dense(g))     # (dense: a hook on saved tensors may give them back in any strides)


@on_operands_device
def _gradient(h: torch.Tensor, g: torch.Tensor) -> torch.Tensor:
    out = torch.empty_like(h)
    f, p, o = h.shape[1] // 2, h.data_ptr(), out.data_ptr()
    B.check(B.load_library().amemSwiGLUGrad(p, p + 2 * f, 2 * f, g.data_ptr(), o, o + 2 * f, h.shape[0], f, current_stream()), "amemSwiGLUGrad")
    return out


@on_operands_device
def _forward(h: torch.Tensor) -> torch.Tensor:
    f, p = h.shape[1] // 2, h.data_ptr()
    out = torch.empty(h.shape[0], f, dtype=h.dtype, device=h.device)
    B.check(B.load_library().amemSwiGLU(p, p + 2 * f, 2 * f, out.data_ptr(), h.shape[0], f, current_stream()), "amemSwiGLU")
    return out


def swiglu(h: torch.Tensor) -> torch.Tensor:
    """silu(h[:, :f]) * h[:, f:] of a [rows, 2 f] tensor in fp32, rounded once to h's type."""
    if _fused(h):
        h = h.contiguous()
        return _SwiGLU.apply(h) if torch.is_grad_enabled() and h.requires_grad else _forward(h)
    f = h.shape[1] // 2
    return (F.silu(h[:, :f].float()) * h[:, f:].float()).to(h.dtype)


def _rms_norm(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    v = x.float()
    v = v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + eps)
    return (v * weight.float()).to(x.dtype)


@on_operands_device
def _rms_forward(x: torch.Tensor, weight: torch.Tensor, eps: float, keep: bool):
    rows, dim = x.numel() // x.shape[-1], x.shape[-1]
    out = torch.empty_like(x)
    rstd = torch.empty(rows, dtype=torch.float32, device=x.device) if keep else None
    B.check(B.load_library().amemRmsNorm(x.data_ptr(), weight.data_ptr(), out.data_ptr(), rstd.data_ptr() if keep else None, rows, dim, float(eps), current_stream()),
            "amemRmsNorm")
    return out, rstd


@on_operands_device
def _rms_gradient(g: torch.Tensor, x: torch.Tensor, weight: torch.Tensor, rstd: torch.Tensor, of_x: bool, of_weight: bool):
    lib, rows, dim = B.load_library(), rstd.numel(), x.shape[-1]
    g_x, g_w = torch.empty_like(x) if of_x else None, torch.empty_like(weight) if of_weight else None
    part = torch.empty(lib.amemRmsNormGradBlocks(rows), dim, dtype=torch.float32, device=x.device) if of_weight else None
    p = [t if t is None else t.data_ptr() for t in (g_x, part, g_w)]
    B.check(lib.amemRmsNormGrad(g.data_ptr(), x.data_ptr(), weight.data_ptr(), rstd.data_ptr(), *p, rows, dim, current_stream()), "amemRmsNormGrad")
    return g_x, g_w


class _RMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, eps):
        out, rstd = _rms_forward(x, weight, eps, True)
        ctx.save_for_backward(x, weight, rstd)
        ctx.eps = eps
        return out

    @staticmethod
    def backward(ctx, g):
        x, weight, rstd = ctx.saved_tensors
        wanted = ctx.needs_input_grad[:2]
        if torch.is_grad_enabled():     # a graph of the gradient is wanted: torch's operators make one
            x, weight = apart(x, weight)
            at = [t for t, w in zip((x, weight), wanted) if w]
            grads = iter(torch.autograd.grad(_rms_norm(x, weight, ctx.eps), at, g, create_graph=True))
            return *(next(grads) if w else None for w in wanted), None
        return *_rms_gradient(dense(g), dense(x), dense(weight), dense(rstd), *wanted), None


def _norm_pays(rows: int, dim: int, gradients: bool) -> bool:
    """Whether one kernel is sooner done than seven passes of torch's: it takes a block per row, so of many short rows it makes
    the same time as of longer ones.  Forward, kernel / torch, us: 65536 rows of 8 74 / 29, of 72 74 / 72, of 128 74 / 100, 1 M of 72
    1036 / 946, of 96 1036 / 1190, 8192 of 8 14 / 25; with gradients 65536 of 8 162 / 80, of 64 162 / 199, 1 M of 64 2568 / 2548."""
    return rows <= 8192 or dim >= (64 if gradients else 80)


def rms_norm(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """``x / sqrt(mean(x^2) + eps) * weight`` over the last dimension in fp32, rounded once to x's type.  One
    kernel for bf16 rows that lie densely on one GPU."""
    if (concrete(x, weight) and x.dtype == weight.dtype == torch.bfloat16 and x.dim() > 0 and x.numel() > 0 and weight.shape == x.shape[-1:] and x.shape[-1] % 8 == 0
            and x.shape[-1] <= 16384 and x.numel() // x.shape[-1] < 2 ** 31 and plain_cuda(x, weight) and x.is_contiguous() and weight.is_contiguous()
            and (x.data_ptr() | weight.data_ptr()) % 16 == 0):
        gradients = torch.is_grad_enabled() and (x.requires_grad or weight.requires_grad)
        if _norm_pays(x.numel() // x.shape[-1], x.shape[-1], gradients):
            return _RMSNorm.apply(x, weight, eps) if gradients else _rms_forward(x, weight, eps, False)[0]
    return _rms_norm(x, weight, eps)


def _as_rows(t: torch.Tensor) -> tuple[int, int]:
    """Rows and their length for the element-wise kernels over a dense tensor: one row, since a row of its own for each of many short
    ones leaves most of a block's threads without a vector (65536 rows of 64: 26.7 us, torch's two passes 16.4)."""
    return (1, t.numel()) if t.numel() < 2 ** 31 else (t.numel() // t.shape[-1], t.shape[-1])


@on_operands_device
def _gated_forward(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    out, (rows, f) = torch.empty_like(gate), _as_rows(gate)
    B.check(B.load_library().amemSwiGLU(gate.data_ptr(), up.data_ptr(), f, out.data_ptr(), rows, f, current_stream()), "amemSwiGLU")
    return out


@on_operands_device
def _gated_gradient(gate: torch.Tensor, up: torch.Tensor, g: torch.Tensor):
    g_gate, g_up, (rows, f) = torch.empty_like(gate), torch.empty_like(up), _as_rows(gate)
    B.check(B.load_library().amemSwiGLUGrad(gate.data_ptr(), up.data_ptr(), f, g.data_ptr(), g_gate.data_ptr(), g_up.data_ptr(), rows, f, current_stream()),
            "amemSwiGLUGrad")
    return g_gate, g_up


class _Gated(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate, up):
        ctx.save_for_backward(gate, up)
        return _gated_forward(gate, up)

    @staticmethod
    def backward(ctx, g):
        gate, up = ctx.saved_tensors
        if torch.is_grad_enabled():
            gate, up = apart(gate, up)
            at = [t for t, w in zip((gate, up), ctx.needs_input_grad) if w]
            grads = iter(torch.autograd.grad(F.silu(gate) * up, at, g, create_graph=True))
            return tuple(next(grads) if w else None for w in ctx.needs_input_grad)
        return tuple(t if w else None for t, w in zip(_gated_gradient(dense(gate), dense(up), dense(g)), ctx.needs_input_grad))


def gated(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """silu(gate) * up of two tensors of one shape.  One kernel, in fp32 and rounded once, for bf16 that lies densely on
    one GPU."""
    if (concrete(gate, up) and gate.dtype == up.dtype == torch.bfloat16 and gate.shape == up.shape and gate.dim() > 0 and gate.numel() > 0 and gate.shape[-1] % 8 == 0
            and plain_cuda(gate, up) and gate.is_contiguous() and up.is_contiguous() and (gate.data_ptr() | up.data_ptr()) % 16 == 0):
        return _Gated.apply(gate, up) if torch.is_grad_enabled() and (gate.requires_grad or up.requires_grad) else _gated_forward(gate, up)
    return F.silu(gate) * up


@on_operands_device
def _embedding_gradient(g: torch.Tensor, ids: torch.Tensor, rows: int) -> torch.Tensor:
    out = torch.empty(rows, g.shape[-1], dtype=g.dtype, device=g.device)
    n = ids.numel()
    work = torch.empty((n + 15) // 16 * 16, dtype=torch.uint8, device=g.device)
    B.check(B.load_library().amemEmbeddingGradShared(g.data_ptr(), ids.data_ptr(), out.data_ptr(), work.data_ptr(), n, g.shape[-1], rows, current_stream()),
            "amemEmbeddingGrad")
    return out


class _Embedding(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, table):
        ctx.save_for_backward(ids)
        ctx.rows = table.shape[0]
        return F.embedding(ids, table)

    @staticmethod
    def backward(ctx, g):
        (ids,) = ctx.saved_tensors
        if torch.is_grad_enabled():
            return None, torch.ops.aten.embedding_dense_backward(g, ids, ctx.rows, -1, False)
        return None, _embedding_gradient(dense(g), ids.contiguous(), ctx.rows)


def embedding(ids: torch.Tensor, table: torch.Tensor) -> torch.Tensor:
    """``table[ids]``.  The gradient of a bf16 table on one GPU sums the rows of equal ids in fp32, in an order that the ids alone
    decide, by the library's kernels (up to 16384 ids: every block looks through all of them)."""
    if (concrete(ids, table) and table.requires_grad and torch.is_grad_enabled() and table.dtype == torch.bfloat16 and table.dim() == 2 and table.shape[1] % 8 == 0 and table.shape[1] > 0
            and ids.dtype == torch.int64 and 0 < ids.numel() <= 16384 and plain_cuda(ids, table) and ids.is_contiguous()):
        return _Embedding.apply(ids, table)
    return F.embedding(ids, table)


def _rotate_plain(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> torch.Tensor:
    x1, x2 = x.float()[..., 0::2], x.float()[..., 1::2]
    o1 = x1 * cos - x2 * sin
    o2 = x1 * sin + x2 * cos
    return torch.stack((o1, o2), dim=-1).flatten(-2).to(x.dtype)


def _tokens_first(x: torch.Tensor) -> bool:
    """Whether [B, H, S, D] lies as [B, S, H, D], as a projection's output does."""
    return x.stride(1) < x.stride(2)


def _in_vectors(x: torch.Tensor) -> bool:
    b, h, s, one = x.stride()
    return one == 1 and (b | h | s) % 8 == 0 and x.data_ptr() % 16 == 0


@on_operands_device
def _rotate_launch(cos: torch.Tensor, sin: torch.Tensor, inverse: bool, tokens_first, *xs: torch.Tensor):
    n, (batch, _, seq, dim) = len(xs), xs[0].shape
    outs = []
    for x, first in zip(xs, tokens_first):
        h = x.shape[1]
        st = (seq * h * dim, dim, h * dim, 1) if first else (seq * h * dim, seq * dim, dim, 1)
        outs.append(torch.empty_strided((batch, h, seq, dim), st, dtype=x.dtype, device=x.device))
    strides = [st for x, o in zip(xs, outs) for st in (*x.stride()[:3], *o.stride()[:3])]
    B.check(B.load_library().amemRotate((ctypes.c_void_p * n)(*(x.data_ptr() for x in xs)), (ctypes.c_void_p * n)(*(o.data_ptr() for o in outs)),
                                        (ctypes.c_int * n)(*(x.shape[1] for x in xs)), (ctypes.c_longlong * (6 * n))(*strides), n, cos.data_ptr(),
                                        sin.data_ptr(), batch, seq, dim, int(inverse), current_stream()), "amemRotate")
    return tuple(outs)


class _Rotate(torch.autograd.Function):
    """A turn; its gradient is the turn back, laid out as the input was."""

    @staticmethod
    def forward(ctx, cos, sin, inverse, tokens_first, *xs):
        ctx.save_for_backward(cos, sin)
        ctx.inverse, ctx.back = inverse, [_tokens_first(x) for x in xs]
        outs = _rotate_launch(cos, sin, inverse, tokens_first, *xs)
        ctx.mark_non_differentiable(*(o for o, wanted in zip(outs, ctx.needs_input_grad[4:]) if not wanted))
        return outs

    @staticmethod
    def backward(ctx, *gs):
        cos, sin = map(dense, ctx.saved_tensors)
        wanted = ctx.needs_input_grad[4:]
        gs = [g if _in_vectors(g) else dense(g) for g, w in zip(gs, wanted) if w]
        turned = iter(_Rotate.apply(cos, sin, not ctx.inverse, [b for b, w in zip(ctx.back, wanted) if w], *gs))
        return None, None, None, None, *(next(turned) if w else None for w in wanted)


def _turn_pays(tokens: int, elements: int) -> bool:
    """Whether one kernel is sooner done than torch's operators with ``elements`` of a token in all tensors: a block per token takes
    1.1 ns whatever it has to turn (65536 tokens 74 us; torch 60 for 16 elements, 158 for 128)."""
    return elements >= 24 or tokens <= 16384


def _kernel_turns(cos: torch.Tensor, sin: torch.Tensor, *xs: torch.Tensor) -> bool:
    batch, seq, dim = xs[0].shape[0], xs[0].shape[2] if xs[0].dim() == 4 else 0, xs[0].shape[-1]
    return (all(x.dim() == 4 and x.dtype == torch.bfloat16 and x.shape[0] == batch and x.shape[2] == seq and x.shape[3] == dim and x.numel() > 0 for x in xs)
            and dim % 8 == 0 and batch * seq < 2 ** 31 and _turn_pays(batch * seq, sum(x.shape[1] for x in xs) * dim)
            and all(t.dtype == torch.float32 and t.shape == (seq, dim // 2) and t.is_contiguous() and not t.requires_grad for t in (cos, sin))
            and plain_cuda(*xs, cos, sin) and (cos.data_ptr() | sin.data_ptr()) % 16 == 0 and all(_in_vectors(x) for x in xs))


def rotate(cos: torch.Tensor, sin: torch.Tensor, *xs: torch.Tensor, as_they_lie: bool = False):
    """Rotary embedding of one or two [B, H, S, D] tensors: neighbouring elements turned by the angles of ``cos`` and
    ``sin`` [S, D / 2].  Computed in fp32 and rounded once; bf16 on one GPU in one kernel.  The results are contiguous, or
    (``as_they_lie``) laid out as the inputs, whose heads may lie inside the positions."""
    if concrete(cos, sin, *xs) and _kernel_turns(cos, sin, *xs):
        layout = [as_they_lie and _tokens_first(x) for x in xs]
        if torch.is_grad_enabled() and any(x.requires_grad for x in xs):
            return _Rotate.apply(cos, sin, False, layout, *xs)
        return _rotate_launch(cos, sin, False, layout, *xs)
    return tuple(_rotate_plain(x, cos, sin) for x in xs)


@on_operands_device
def add_pieces(dst: torch.Tensor, pieces, scale: float = 1.0, comm=None) -> None:
    """``dst[at:at + t.numel()] += scale * t`` for every (at, t) of ``pieces``, which do not overlap: contiguous bf16
    tensors on the GPU that holds ``dst``, a dense fp32 tensor.  One kernel.  ``comm``: the one-rank communicator that this is an
    operation of, if any; its bound on blocks holds."""
    n, lib = len(pieces), B.load_library()
    base, st = dst.data_ptr(), current_stream()
    args = ((ctypes.c_void_p * n)(*(t.data_ptr() for _, t in pieces)), (ctypes.c_void_p * n)(*(base + 4 * at for at, _ in pieces)),
            (ctypes.c_longlong * n)(*(t.numel() for _, t in pieces)), n, scale)
    if comm is None:
        B.check(lib.amemSumPieces(*args, st), "amemSumPieces")
    else:
        B.check(lib.amemSumPiecesLocal(*args, comm._h, st), "amemSumPiecesLocal")
    torch.autograd.graph.increment_version(dst)      # as an in-place operator does


@on_operands_device
def adamw_step(grad, m, v, master, shard, lr: float, betas, eps: float, weight_decay: float, step: int) -> None:
    """One AdamW update in place: fp32 ``m``, ``v`` and ``master`` from the fp32 ``grad``; ``shard``
    receives the new weights in bf16.  ``step`` counts from 1.  One kernel for five tensors of one shape,
    dense on one GPU; the general form takes, or refuses, what torch does."""
    flat = (grad, m, v, master, shard)
    if all(t.is_cuda and t.device == grad.device and t.shape == grad.shape and t.is_contiguous() and t.data_ptr() % 16 == 0 for t in flat) and shard.dtype == torch.bfloat16 \
            and all(t.dtype == torch.float32 for t in flat[:4]):
        B.check(B.load_library().amemAdamW(grad.data_ptr(), m.data_ptr(), v.data_ptr(), master.data_ptr(), shard.data_ptr(), grad.numel(),
                                           float(lr), float(betas[0]), float(betas[1]), float(eps), float(weight_decay), step, current_stream()), "amemAdamW")
        torch.autograd.graph.increment_version([t for t in flat[1:] if not t.is_inference()])   # as an in-place operator does
        return
    b1, b2 = betas
    c1, c2 = 1 - b1 ** step, 1 - b2 ** step
    m.mul_(b1).add_(grad, alpha=1 - b1)
    v.mul_(b2).addcmul_(grad, grad, value=1 - b2)
    if weight_decay:
        master.mul_(1 - lr * weight_decay)
    master.addcdiv_(m / c1, (v / c2).sqrt_().add_(eps), value=-lr)
    shard.copy_(master)
