"""What saved-tensor hooks give back may lie anywhere and in any strides: the kernels of the backward functions get dense copies.  No
GPU: the launches are stood in for, and look at what they are handed."""
import pytest
import torch

from asystem_amem_b200.ops import elementwise as EW
from asystem_amem_b200.ops import moe
from asystem_amem_b200.parallel import ep


def _elsewhere(t):
    """The same values, at an odd address and, where there are two dimensions, in the other order."""
    out = torch.empty(t.numel() + 1, dtype=t.dtype)[1:]
    out = out.view(t.shape[::-1]).permute(*range(t.dim() - 1, -1, -1)) if t.dim() > 1 else out.view(t.shape)
    return out.copy_(t)


def _lie_densely(*tensors):
    assert all(t.is_contiguous() and t.data_ptr() % 16 == 0 for t in tensors)


class _Dispatcher:
    E = 4

    def local(self, *_):
        return True

    def dispatch_local(self, x, idx):
        n = idx.numel()
        return moe.DispatchResult(x.repeat_interleave(idx.shape[1], 0), None, torch.tensor([0, n, n, n, n], dtype=torch.int32),
                                  torch.arange(n, dtype=torch.int32).view(idx.shape))

    def input_grad_local(self, g_rows, send_pos, idx, g_logits, router):
        _lie_densely(g_rows, send_pos, idx, g_logits, router)
        return torch.zeros(idx.shape[0], router.shape[1])


@pytest.fixture
def calls(monkeypatch):
    def rms_gradient(g, x, weight, rstd, *_):
        _lie_densely(g, x, weight, rstd)
        return torch.zeros_like(x), torch.zeros_like(weight)

    def gated_gradient(gate, up, g):
        _lie_densely(gate, up, g)
        return torch.zeros_like(gate), torch.zeros_like(up)

    def gradient(h, g):
        _lie_densely(h, g)
        return torch.zeros_like(h)

    def embedding_gradient(g, ids, rows):
        assert ids.is_contiguous()
        return torch.zeros(rows, g.shape[-1])

    def rotate_launch(cos, sin, inverse, first, *xs):
        _lie_densely(cos, sin)
        return tuple(x.clone() for x in xs)

    def logits_grad(g_w, w, idx, experts):
        _lie_densely(g_w, w, idx)
        return torch.zeros(idx.shape[0], experts)

    monkeypatch.setattr(EW, "_rms_forward", lambda x, w, eps, keep: (x.clone(), torch.ones(x.shape[0])))
    monkeypatch.setattr(EW, "_rms_gradient", rms_gradient)
    monkeypatch.setattr(EW, "_gated_forward", lambda gate, up: gate * up)
    monkeypatch.setattr(EW, "_gated_gradient", gated_gradient)
    monkeypatch.setattr(EW, "_forward", lambda h: h[:, :h.shape[1] // 2].clone())
    monkeypatch.setattr(EW, "_gradient", gradient)
    monkeypatch.setattr(EW, "_embedding_gradient", embedding_gradient)
    monkeypatch.setattr(EW, "_rotate_launch", rotate_launch)
    monkeypatch.setattr(moe, "_route_launch", moe._route_torch)
    monkeypatch.setattr(moe, "_route_logits_grad", logits_grad)
    monkeypatch.setattr(ep, "_route_launch", moe._route_torch)
    monkeypatch.setattr(ep, "_route_logits_grad", logits_grad)
    r = lambda *shape: torch.randn(*shape, requires_grad=True)
    return {"norm": lambda: EW._RMSNorm.apply(r(6, 8), r(8), 1e-5), "gated": lambda: EW._Gated.apply(r(6, 8), r(6, 8)), "swiglu": lambda: EW._SwiGLU.apply(r(6, 16)),
            "embedding": lambda: EW._Embedding.apply(torch.arange(6).view(2, 3), r(9, 8)),
            "rotate": lambda: EW._Rotate.apply(torch.ones(3, 4), torch.zeros(3, 4), False, [False], r(1, 2, 3, 8))[0],
            "route": lambda: moe._Route.apply(r(6, 8), r(4, 8), 2)[1],
            "route and dispatch": lambda: ep._RouteDispatch.apply(r(6, 8), r(4, 8), _Dispatcher(), 2)[0]}


@pytest.mark.parametrize("name", ["norm", "gated", "swiglu", "embedding", "rotate", "route", "route and dispatch"])
def test_what_a_hook_gives_back(calls, name):
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, _elsewhere):
        out = calls[name]()
    out.backward(torch.ones_like(out))
