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
