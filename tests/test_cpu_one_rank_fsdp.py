"""A sharded unit of one rank, whose gradients go to its shard from where autograd left them: gradients that this form leaves to the
general one.  No GPU: the form is switched on for tensors of the host, and nothing that is tested here reaches its kernel."""
import pytest

from mp_util import run_ranks


def _gradients(rank, world, uid, kind):
    import torch
    import torch.nn as nn
    from asystem_amem_b200 import Communicator
    from asystem_amem_b200.parallel import FSDP

    class Unit(nn.Module):
        def __init__(self):
            super().__init__()
            self.tok = nn.Embedding(11, 8, sparse=kind != "dense")
            self.out = nn.Linear(8, 5, bias=False) if kind != "sparse alone" else None

        def forward(self, ids):
            x = self.tok(ids)
            return x if self.out is None else self.out(x)

    class Model(nn.Module):
        def __init__(self):
            super().__init__()
            self.units = nn.ModuleList([Unit()])

    torch.manual_seed(0)
    model = Model().to(torch.bfloat16)
    torch.manual_seed(0)
    plain = Model().to(torch.bfloat16)
    comm = Communicator(1, 0, uid)
    fsdp = FSDP(model, comm)
    fsdp.units[0].direct = kind != "dense"
    for seed in (1, 2):         # gradients of two backward passes add up
        ids = torch.randint(0, 11, (3, 4), generator=torch.Generator().manual_seed(seed))
        fsdp.forward_units(ids).float().square().sum().backward()
        plain.units[0](ids).float().square().sum().backward()
    got, want = fsdp.units[0].grad_shard, [p.grad for p in plain.parameters()]
    comm.destroy()
    want = torch.cat([(g.to_dense() if g.layout != torch.strided else g).reshape(-1) for g in want]).float()
    return float((got[:want.numel()] - want).abs().max()), float(want.abs().max())


@pytest.mark.parametrize("kind", ["dense", "sparse", "sparse alone"])
def test_sparse_gradients(kind):
    err, scale = run_ranks(_gradients, 1, args=(kind,))[0]
    assert scale > 0 and err <= 4 * 2.0 ** -8 * scale        # bf16 sums over a dozen tokens and two passes
