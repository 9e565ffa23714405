"""Outputs that want no gradient because none of their inputs does.  No GPU: launches are stood in for."""
import pytest
import torch

from asystem_amem_b200.ops import moe
from asystem_amem_b200.parallel import ep


class _Dispatcher:
    """One rank's dispatcher, all choices kept: the rows of expert after expert."""
    E = 4

    def local(self, *_):
        return True

    def dispatch_local(self, x, idx):
        order = idx.reshape(-1).argsort(stable=True)
        pos = torch.empty(idx.numel(), dtype=torch.int32)
        pos[order] = torch.arange(idx.numel(), dtype=torch.int32)
        offsets = torch.zeros(self.E + 1, dtype=torch.int32)
        offsets[1:] = torch.bincount(idx.reshape(-1).long(), minlength=self.E).cumsum(0)
        return moe.DispatchResult(x[order // idx.shape[1]].clone(), None, offsets, pos.view(idx.shape))


@pytest.mark.parametrize("of_x", [False, True])
def test_rows_of_a_routing(monkeypatch, of_x):
    monkeypatch.setattr(ep, "_kernel_routes", lambda *_: True)
    monkeypatch.setattr(ep, "_route_launch", moe._route_torch)
    torch.manual_seed(0)
    x, router = torch.randn(6, 8, requires_grad=of_x), torch.randn(4, 8, requires_grad=True)
    rows, _, _, _, w = ep.ep_route_dispatch(_Dispatcher(), x, router, 2)
    assert rows.requires_grad == of_x and w.requires_grad


@pytest.mark.parametrize("of_q,of_k", [(True, True), (True, False), (False, True)])
def test_turned_tensors(monkeypatch, of_q, of_k):
    from asystem_amem_b200.models.llama import rope_tables
    from asystem_amem_b200.ops import elementwise as EW
    turned = []

    def launch(cos, sin, inverse, tokens_first, *xs):
        turned.append(len(xs))
        return tuple(EW._rotate_plain(x, cos, -sin if inverse else sin) for x in xs)
    monkeypatch.setattr(EW, "_rotate_launch", launch)
    cos, sin = rope_tables(3, 8, 10000.0, "cpu")
    torch.manual_seed(0)
    q, k = torch.randn(1, 2, 3, 8, requires_grad=of_q), torch.randn(1, 1, 3, 8, requires_grad=of_k)
    outs = EW._Rotate.apply(cos, sin, False, [False, False], q, k)
    assert [o.requires_grad for o in outs] == [of_q, of_k]
    g = [torch.randn_like(o) for o in outs]
    wanted = [t for t in (q, k) if t.requires_grad]
    got = torch.autograd.grad([o for o in outs if o.requires_grad], wanted, [a for a, o in zip(g, outs) if o.requires_grad], create_graph=True)
    want = torch.autograd.grad([EW._rotate_plain(t, cos, sin) for t in wanted], wanted, [a for a, o in zip(g, outs) if o.requires_grad])
    for a, b in zip(got, want):
        torch.testing.assert_close(a, b)
    assert turned == [2, len(wanted)]
