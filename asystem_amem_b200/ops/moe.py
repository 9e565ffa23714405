"""Expert-parallel MoE dispatch / combine on the fused kernels.

``MoeDispatcher`` owns the symmetric receive / expert-output buffers of one communicator.
``dispatch`` returns the rows of this rank's local experts already grouped by expert (the
routing permutation happens inside the all-to-all writes); ``combine`` pulls the expert outputs
back from the expert ranks and applies the routing weights in the same pass.

On the mock backend (no GPU) the dispatcher composes the same row layout from the library's
all-gather and variable-size all-to-all on host tensors, which is how the expert-parallel
wrappers and their gradients are tested as multi-process runs on a CPU.  CUDA tensors always
go to the kernels.

Reference parity: none -- the reference names all-to-all as the largest consumer of NCCL memory
(README.md:132) but leaves routing and permutation to the framework above it.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass

import torch

from .. import bindings as B
from .operands import apart, current_stream, dense, on_operands_device, plain_cuda


def _view(ptr: int, rows: int, d: int, device) -> torch.Tensor:
    """A bf16 [rows, d] tensor over library-owned device memory (no ownership transfer)."""
    class _Holder:
        __cuda_array_interface__ = {"shape": (rows * d,), "typestr": "<i2", "data": (ptr, False), "version": 3}
    return torch.as_tensor(_Holder(), device=device).view(torch.bfloat16).view(rows, d)


def _route_torch(x: torch.Tensor, router: torch.Tensor, k: int) -> tuple[torch.Tensor, torch.Tensor]:
    top = (x @ router.t()).float().topk(k, dim=1)
    return top.indices.to(torch.int32), torch.softmax(top.values, dim=1)


@on_operands_device
def _route_launch(x: torch.Tensor, router: torch.Tensor, k: int) -> tuple[torch.Tensor, torch.Tensor]:
    T, d = x.shape
    idx, w = torch.empty(T, k, dtype=torch.int32, device=x.device), torch.empty(T, k, dtype=torch.float32, device=x.device)
    B.check(B.load_library().amemMoeRoute(x.data_ptr(), router.data_ptr(), idx.data_ptr(), w.data_ptr(), T, d, router.shape[0], k,
                                          current_stream()), "amemMoeRoute")
    return idx, w


@on_operands_device
def _route_logits_grad(g_w: torch.Tensor, w: torch.Tensor, idx: torch.Tensor, experts: int) -> torch.Tensor:
    T, k = idx.shape
    out = torch.empty(T, experts, dtype=torch.bfloat16, device=w.device)
    B.check(B.load_library().amemMoeRouteGrad(g_w.data_ptr(), w.data_ptr(), idx.data_ptr(), out.data_ptr(), T, experts, k,
                                              current_stream()), "amemMoeRouteGrad")
    return out


def _route_grads_torch(x: torch.Tensor, router: torch.Tensor, idx: torch.Tensor, g_w: torch.Tensor, of_x: bool, of_router: bool):
    """The gradients of :func:`route`'s weights with a graph of their own."""
    x, router = apart(x, router)
    again = torch.softmax((x @ router.t()).float().gather(1, idx.long()), dim=1)
    grads = iter(torch.autograd.grad(again, [t for t, n in ((x, of_x), (router, of_router)) if n], g_w, create_graph=True))
    return next(grads) if of_x else None, next(grads) if of_router else None


def _route_pays(T: int, d: int, E: int) -> bool:
    """Whether one kernel routes T tokens sooner than a library product, a cast, a top-k and a softmax do.  Every block reads the
    whole router, so a long one (experts in tiles of 16, 32, 64, 128 or 256, times d) keeps few tokens waiting, and with more than
    64 experts a block has only 8 tokens to spread that over.  Kernel / torch in us, from cold memory, under a graph:
    64 x 4096 experts (the layer's default) 14.4 / 26.7 for one token, 86 / 115 for 16384; 64 x 8192 22.6 / 32.8 and 135 / 143;
    128 x 2048 16.5 / 24.6 and 118 / 145; 256 x 2048 28.7 / 26.8 (28.7 / 30.8 for 32 tokens) and 203 / 240;
    128 x 4096 26.7 / 28.7 and, for 4096 tokens, 61.4 / 61.5, but 106 / 94 for 8192 and 197 / 160 for 16384; 72 x 4096 24.6 / 28.7,
    53 / 55, 90 / 82 and 166 / 133; and on the far side 256 x 4096 51.2 / 28.7 and 344 / 275, 64 x 16384 36.9 / 32.8 and 232 / 178."""
    if E <= 64 and d <= 8192:
        return True
    tiled = max(16, 1 << (E - 1).bit_length())
    return tiled * d <= 530_000 and (E <= 64 or d <= 2048 or T <= 4096)


class _Route(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, router, k):
        # (the gradients are the kernel's either way; with them, in us, by the kernel / torch altogether / torch's routing alone: 16384
        # tokens of 128 x 4096 experts 281 / 260 / 255; 8192 of them 153 / 176 / 182, of 256 x 4096 241 / 231 / 235; 4096, where the
        # launches of the host show, 142 / 218)
        launch = x.shape[0] <= (8192 if router.numel() <= 530_000 else 4096) or _route_pays(*x.shape, router.shape[0])
        idx, w = _route_launch(x, router, k) if launch else _route_torch(x, router, k)
        ctx.save_for_backward(x, router, idx, w)
        ctx.mark_non_differentiable(idx)
        return idx, w

    @staticmethod
    def backward(ctx, _g_idx, g_w):
        x, router, idx, w = ctx.saved_tensors
        of_x, of_router = ctx.needs_input_grad[:2]
        if torch.is_grad_enabled():     # a graph of the gradient is wanted: torch's operators make one
            return *_route_grads_torch(x, router, idx, g_w, of_x, of_router), None
        g_logits = _route_logits_grad(g_w.contiguous(), dense(w), dense(idx), router.shape[0])
        return g_logits @ router if of_x else None, g_logits.t() @ x if of_router else None, None


def _kernel_routes(x: torch.Tensor, router: torch.Tensor, k: int) -> bool:
    return (x.dtype == router.dtype == torch.bfloat16 and x.dim() == router.dim() == 2 and x.shape[0] > 0 and x.shape[1] == router.shape[1]
            and x.shape[1] > 0 and x.shape[1] % 8 == 0 and 0 < k <= router.shape[0] <= 256 and plain_cuda(x, router) and x.is_contiguous()
            and router.is_contiguous() and (x.data_ptr() | router.data_ptr()) % 16 == 0)


def route(x: torch.Tensor, router: torch.Tensor, k: int) -> tuple[torch.Tensor, torch.Tensor]:
    """The ``k`` largest of every token's logits ``x @ router.T`` and their softmax, largest first: int32 and fp32
    [T, k].  One kernel for bf16 rows that lie densely on one GPU (equal logits by the lower expert), without gradients only where
    that is the faster way.  (With them it always is for one rank's layer: its step takes the routing's gradients in with the
    dispatch's.  128 x 4096 experts of 512, top-8: 8192 tokens 3.32 ms a training step, 3.38 with torch's routing; 256 experts, 2048
    tokens 2.95 and 3.02; 8192 4.29 and 4.31.)"""
    if _kernel_routes(x, router, k):
        if torch.is_grad_enabled() and (x.requires_grad or router.requires_grad):
            return _Route.apply(x, router, k)
        if _route_pays(*x.shape, router.shape[0]):
            return _route_launch(x, router, k)
    return _route_torch(x, router, k)


@dataclass
class DispatchResult:
    recv_x: torch.Tensor          # bf16 [capacity_rows, d]; rows [0, total_rows) are valid
    expert_counts: torch.Tensor   # int32 [experts_per_rank]
    expert_offsets: torch.Tensor  # int32 [experts_per_rank + 1]
    send_pos: torch.Tensor        # int32 [T, k]: row of every (token, choice) on its expert's rank (-1: left out, no room)
    dropped: torch.Tensor | None = None   # int32 [1]: rows routed to THIS rank that did not fit its capacity


class MoeDispatcher:
    def __init__(self, comm, num_experts: int, hidden: int, capacity_rows: int):
        if num_experts % comm.nranks:
            raise ValueError("experts must divide evenly over the ranks")
        self.comm, self.E, self.d, self.capacity = comm, num_experts, hidden, capacity_rows
        self.experts_per_rank = num_experts // comm.nranks
        from ..comm import backend_usage
        self.host = backend_usage()["backend"] == "mock"   # no GPU: composed from all_gather + all_to_all_v
        if self.host:
            self.device = torch.device("cpu")
            self.recv_x = torch.zeros(capacity_rows, hidden, dtype=torch.bfloat16)
            self.y = torch.zeros(capacity_rows, hidden, dtype=torch.bfloat16)
            return
        self.device = torch.device("cuda", torch.cuda.current_device())
        self._map_buffers()

    def _map_buffers(self) -> None:
        rx, y = ctypes.c_void_p(), ctypes.c_void_p()
        B.check(self.comm.lib.amemMoeBuffers(self.comm._h, self.capacity, self.d, ctypes.byref(rx), ctypes.byref(y)), "amemMoeBuffers")
        self.recv_x = _view(rx.value, self.capacity, self.d, self.device)
        self.y = _view(y.value, self.capacity, self.d, self.device)  # experts write their outputs here

    def dispatch(self, x: torch.Tensor, topk_idx: torch.Tensor, stream=None) -> DispatchResult:
        assert x.dtype == torch.bfloat16 and x.is_contiguous() and x.shape[1] == self.d
        topk_idx = topk_idx.to(torch.int32).contiguous()
        if self.host:
            return self._host_dispatch(x, topk_idx)
        if x.data_ptr() % 16:
            with torch.cuda.stream(stream):     # (None: the current one)
                x = dense(x)
        T, k = topk_idx.shape
        counts = torch.empty(self.experts_per_rank, dtype=torch.int32, device=x.device)
        offsets = torch.empty(self.experts_per_rank + 1, dtype=torch.int32, device=x.device)
        send_pos = torch.empty(T, k, dtype=torch.int32, device=x.device)
        dropped = torch.empty(1, dtype=torch.int32, device=x.device)   # every word of the four is written by the kernels
        st = stream.cuda_stream if stream else current_stream()
        B.check(self.comm.lib.amemMoeDispatchCounted(x.data_ptr(), topk_idx.data_ptr(), T, k, self.d, self.E, self.capacity,
                                                     counts.data_ptr(), offsets.data_ptr(), send_pos.data_ptr(), dropped.data_ptr(),
                                                     self.comm._h, st), "amemMoeDispatch")
        self._last_idx = topk_idx
        return DispatchResult(self.recv_x, counts, offsets, send_pos, dropped)

    def combine(self, topk_idx: torch.Tensor, topk_w: torch.Tensor, send_pos: torch.Tensor, out: torch.Tensor | None = None,
                stream=None) -> torch.Tensor:
        """Expert outputs must have been written to ``self.y`` in the row layout of ``recv_x``."""
        topk_idx = topk_idx.to(torch.int32).contiguous()
        topk_w = topk_w.to(torch.float32).contiguous()
        if self.host:
            res = self._host_combine(topk_idx, topk_w, send_pos)
            return res if out is None else out.copy_(res)
        T, k = topk_idx.shape
        out = torch.empty(T, self.d, dtype=torch.bfloat16, device=topk_w.device) if out is None else out
        st = stream.cuda_stream if stream else current_stream()
        B.check(self.comm.lib.amemMoeCombine(topk_idx.data_ptr(), topk_w.data_ptr(), send_pos.data_ptr(), out.data_ptr(), T, k,
                                             self.d, self.E, self.capacity, self.comm._h, st), "amemMoeCombine")
        return out

    # ---- one rank: the same steps between tensors, without the communicator's buffers ----------
    def local(self, *bf16: torch.Tensor) -> bool:
        """Whether the one-rank forms below take these [rows, hidden] tensors."""
        return not self.host and self.comm.nranks == 1 and all(
            t.is_cuda and t.dtype == torch.bfloat16 and t.dim() == 2 and t.shape[0] > 0 and t.shape[1] == self.d for t in bf16)

    def dispatch_local(self, x: torch.Tensor, topk_idx: torch.Tensor) -> DispatchResult:
        """``dispatch`` whose rows land in a tensor of their own."""
        x, topk_idx = dense(x), topk_idx.to(torch.int32).contiguous()
        T, k = topk_idx.shape
        rows = min(self.capacity, T * k)
        recv = torch.empty(rows, self.d, dtype=torch.bfloat16, device=x.device)
        counts = torch.empty(self.E, dtype=torch.int32, device=x.device)
        offsets = torch.empty(self.E + 1, dtype=torch.int32, device=x.device)
        send_pos = torch.empty(T, k, dtype=torch.int32, device=x.device)
        dropped = torch.empty(1, dtype=torch.int32, device=x.device)
        B.check(self.comm.lib.amemMoeDispatchLocal(x.data_ptr(), topk_idx.data_ptr(), T, k, self.d, self.E, recv.data_ptr(), rows, counts.data_ptr(),
                                                   offsets.data_ptr(), send_pos.data_ptr(), dropped.data_ptr(), self.comm._h,
                                                   current_stream()), "amemMoeDispatchLocal")
        return DispatchResult(recv, counts, offsets, send_pos, dropped)

    def combine_local(self, y: torch.Tensor, topk_idx: torch.Tensor, topk_w: torch.Tensor, send_pos: torch.Tensor) -> torch.Tensor:
        """``combine`` of the expert outputs ``y``."""
        y, idx, w, pos = dense(y), topk_idx.to(torch.int32).contiguous(), topk_w.to(torch.float32).contiguous(), send_pos.contiguous()
        T, k = idx.shape
        out = torch.empty(T, self.d, dtype=torch.bfloat16, device=y.device)
        B.check(self.comm.lib.amemMoeCombineLocal(idx.data_ptr(), w.data_ptr(), pos.data_ptr(), y.data_ptr(), y.shape[0], out.data_ptr(), T, k, self.d, self.E,
                                                  self.comm._h, current_stream()), "amemMoeCombineLocal")
        return out

    def combine_grad_local(self, g_out: torch.Tensor, y: torch.Tensor, topk_w: torch.Tensor, send_pos: torch.Tensor):
        """Gradients of ``combine_local``: (of ``y``, bf16; of the weights, fp32)."""
        g_out, y, w, pos = dense(g_out), dense(y), topk_w.to(torch.float32).contiguous(), send_pos.contiguous()
        T, k = w.shape
        g_y, g_w = torch.empty_like(y), torch.empty(T, k, dtype=torch.float32, device=y.device)
        B.check(self.comm.lib.amemMoeCombineGradLocal(g_out.data_ptr(), y.data_ptr(), w.data_ptr(), pos.data_ptr(), g_y.data_ptr(), g_w.data_ptr(), y.shape[0],
                                                      T, k, self.d, self.comm._h, current_stream()), "amemMoeCombineGradLocal")
        return g_y, g_w

    def input_grad_local(self, g_rows: torch.Tensor, send_pos: torch.Tensor, idx: torch.Tensor, g_logits: torch.Tensor, router: torch.Tensor) -> torch.Tensor:
        """The tokens' gradient, bf16: of the rows that ``dispatch_local`` made of them and, through the logits' gradient
        [T, E], of their routing."""
        T, k = idx.shape
        g_x = torch.empty(T, self.d, dtype=torch.bfloat16, device=g_rows.device)
        B.check(self.comm.lib.amemMoeInputGradLocal(g_rows.data_ptr(), send_pos.data_ptr(), idx.data_ptr(), g_logits.data_ptr(), router.data_ptr(), g_x.data_ptr(),
                                                    g_rows.shape[0], T, k, self.d, self.E, self.comm._h, current_stream()), "amemMoeInputGradLocal")
        return g_x

    # ---- host form (mock backend): same row layout as the kernels, built from the library's
    # all-gather and variable-size all-to-all, so that the expert-parallel wrappers and their
    # gradients can be tested as real multi-process runs without a GPU ------------------------
    def _host_plan(self, topk_idx: torch.Tensor):
        """Everything both directions need, from the routing alone (every rank computes the same
        global picture): sorted pair order, destination rows, per-peer element counts."""
        n, me, El = self.comm.nranks, self.comm.rank, self.experts_per_rank
        flat = topk_idx.reshape(-1).long()                              # pair p = t * k + c
        cnt = torch.bincount(flat, minlength=self.E)                    # my pairs per expert
        all_cnt = torch.empty(n, self.E, dtype=torch.int64)
        self.comm.all_gather(cnt.contiguous(), all_cnt)                 # all_cnt[src][e]
        total = all_cnt.sum(0)
        exp_off = torch.zeros(self.E, dtype=torch.int64)                # first row of expert e at its owner
        for r in range(n):
            seg = total[r * El:(r + 1) * El]
            exp_off[r * El:(r + 1) * El] = torch.cumsum(seg, 0) - seg
        src_off = torch.cumsum(all_cnt, 0) - all_cnt                    # rows of expert e from lower source ranks
        order = torch.argsort(flat, stable=True)                        # pairs by expert, pair order inside
        starts = torch.cumsum(cnt, 0) - cnt
        within = torch.empty_like(flat)
        within[order] = torch.arange(flat.numel()) - starts[flat[order]]
        pos = exp_off[flat] + src_off[me][flat] + within
        pos = torch.where(pos < self.capacity, pos, torch.full_like(pos, -1))
        send_rows = torch.tensor([int(cnt[r * El:(r + 1) * El].sum()) for r in range(n)])
        recv_rows = torch.tensor([int(all_cnt[r][me * El:(me + 1) * El].sum()) for r in range(n)])
        return flat, order, pos, all_cnt, total, send_rows, recv_rows

    def _owner_permutation(self, all_cnt: torch.Tensor) -> torch.Tensor:
        """Rows arrive grouped [source][local expert]; the buffers hold them [local expert][source]:
        returns, for every row in arrival order, its row in the buffer."""
        n, me, El = self.comm.nranks, self.comm.rank, self.experts_per_rank
        mine = all_cnt[:, me * El:(me + 1) * El]                         # [src][el]
        per_el = mine.sum(0)
        el_off = torch.cumsum(per_el, 0) - per_el
        src_in_el = torch.cumsum(mine, 0) - mine                        # [src][el] offset inside the expert
        rows = []
        for src in range(n):
            for el in range(El):
                c = int(mine[src][el])
                rows.append(torch.arange(c) + int(el_off[el]) + int(src_in_el[src][el]))
        return torch.cat(rows) if rows else torch.zeros(0, dtype=torch.int64)

    def _host_dispatch(self, x: torch.Tensor, topk_idx: torch.Tensor) -> DispatchResult:
        T, k = topk_idx.shape
        me, El, d = self.comm.rank, self.experts_per_rank, self.d
        flat, order, pos, all_cnt, total, send_rows, recv_rows = self._host_plan(topk_idx)
        if int((pos < 0).sum()):
            raise ValueError("host form of the MoE dispatch needs a capacity that holds every routed row")
        send = x[order // k].contiguous()
        arrive = torch.empty(int(recv_rows.sum()), d, dtype=x.dtype)
        self.comm.all_to_all_v(send.view(-1), arrive.view(-1), (send_rows * d).tolist(), (recv_rows * d).tolist())
        self.recv_x[self._owner_permutation(all_cnt)] = arrive
        counts = total[me * El:(me + 1) * El].to(torch.int32)
        offsets = torch.zeros(El + 1, dtype=torch.int32)
        offsets[1:] = torch.cumsum(counts, 0)
        return DispatchResult(self.recv_x, counts, offsets, pos.to(torch.int32).view(T, k))

    def _host_combine(self, topk_idx: torch.Tensor, topk_w: torch.Tensor, send_pos: torch.Tensor) -> torch.Tensor:
        T, k = topk_idx.shape
        d = self.d
        flat, order, _pos, all_cnt, _total, send_rows, recv_rows = self._host_plan(topk_idx)
        back = self.y[self._owner_permutation(all_cnt)].contiguous()     # arrival order = what each source sent
        got = torch.empty(int(send_rows.sum()), d, dtype=self.y.dtype)
        self.comm.all_to_all_v(back.view(-1), got.view(-1), (recv_rows * d).tolist(), (send_rows * d).tolist())
        y_at = torch.empty(T * k, d, dtype=self.y.dtype)
        y_at[order] = got                                                # rows came back in sorted pair order
        out = (y_at.view(T, k, d).float() * topk_w.view(T, k, 1)).sum(1)
        return out.to(torch.bfloat16)
