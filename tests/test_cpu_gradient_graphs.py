"""Graphs of gradients (create_graph) through the autograd functions of the kernels.  No GPU: the launches are stood in for by
torch's operators, the backward functions are the ones that run on a GPU."""
import pytest
import torch
import torch.nn.functional as F

from asystem_amem_b200.ops import elementwise as EW
from asystem_amem_b200.ops import moe


@pytest.fixture
def functions(monkeypatch):
    monkeypatch.setattr(EW, "_rms_forward", lambda x, w, eps, keep: (EW._rms_norm(x, w, eps), x.new_empty(0)))
    monkeypatch.setattr(EW, "_gated_forward", lambda gate, up: F.silu(gate) * up)

    def route_launch(x, router, k):
        top = (x @ router.t()).topk(k, dim=1)
        return top.indices.to(torch.int32), torch.softmax(top.values, dim=1)
    monkeypatch.setattr(moe, "_route_launch", route_launch)
    return {
        "norm": (lambda a, b: EW._RMSNorm.apply(a, b, 1e-5), lambda a, b: EW._rms_norm(a, b, 1e-5)),
        "gated": (EW._Gated.apply, lambda a, b: F.silu(a) * b),
        "route": (lambda a, b: moe._Route.apply(a, b, 2)[1], lambda a, b: torch.softmax((a @ b.t()).topk(2, dim=1).values, dim=1)),
    }


# operands of one shape, so that they can be one tensor; a vector for the norm, whose weight has one dimension
SHAPES = {"norm": (8,), "gated": (3, 8), "route": (5, 8)}


@pytest.mark.parametrize("name", SHAPES)
@pytest.mark.parametrize("related", ["apart", "one tensor", "one from the other", "the first alone", "the second alone"])
def test_gradients_of_related_operands(functions, name, related):
    fn, plain = functions[name]
    g = torch.Generator().manual_seed(3)
    a, b = (torch.randn(SHAPES[name], generator=g, requires_grad=True) for _ in range(2))
    weigh = torch.randn(plain(a, b).shape, generator=g)

    def gradients(f):
        first, second = {"apart": (a, b), "one tensor": (a, a), "one from the other": (a * b.sin(), b), "the first alone": (a, b.detach()),
                         "the second alone": (a.detach(), b)}[related]
        at = [t for t in (a, b) if related != "one tensor" or t is a]
        first_order = torch.autograd.grad((f(first, second) * weigh).sum(), at, create_graph=True, allow_unused=True)
        kept = [t for t in first_order if t is not None]
        of = sum(t.square().sum() for t in kept)
        second_order = torch.autograd.grad(of, at, allow_unused=True) if of.requires_grad else ()   # (linear in the operand: none)
        return [*kept, *(t for t in second_order if t is not None)]

    got, want = gradients(fn), gradients(plain)
    assert len(got) == len(want)
    for x, y in zip(got, want):
        torch.testing.assert_close(x, y, rtol=1e-4, atol=1e-5)      # fp32, second derivatives of sums of a few terms
