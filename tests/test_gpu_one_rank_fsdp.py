"""The sum of gradients into a one-rank shard: pieces of memory of every size and address, and a sharded unit that uses it."""
import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 3])
def comm(request, monkeypatch):
    """A communicator whose blocks the user does not bound, or bounds to three."""
    from asystem_amem_b200 import Communicator, get_unique_id
    if request.param:
        monkeypatch.setenv("AMEM_MAX_BLOCKS", str(request.param))
    c = Communicator(1, 0, get_unique_id())
    yield c
    torch.cuda.synchronize()
    c.destroy()


# (offset in the shard, elements, offset of the source in its memory): blocks' edges, addresses that no vector starts at, one
# launch's pieces and more, empty ones among them
ONE = [(0, 4096, 0)]
EDGES = [(0, 1, 0), (4, 7, 0), (12, 4095, 0), (4112, 4096, 0), (8212, 4097, 0), (12320, 100_003, 0)]
ODD = [(1, 9, 0), (16, 4096, 1), (4113, 5000, 3), (9123, 8192, 0)]
MANY = [(i * 300 + i % 3, 0 if i % 7 == 3 else 290 - i, i % 2) for i in range(70)]


@pytest.mark.parametrize("pieces", [ONE, EDGES, ODD, MANY, [(5, 0, 0)], []], ids=["one", "edges", "odd", "many", "empty", "none"])
@pytest.mark.parametrize("scale", [1.0, 0.37])
def test_sums_of_pieces(comm, pieces, scale):
    from asystem_amem_b200.ops.elementwise import add_pieces
    g = torch.Generator(device="cuda").manual_seed(1)
    n = max((at + k for at, k, _ in pieces), default=0) + 100
    dst = torch.randn(n, device="cuda", generator=g)
    src = [(at, torch.randn(k + shift, device="cuda", generator=g).to(torch.bfloat16)[shift:]) for at, k, shift in pieces]
    for form in ({}, {"comm": comm}):
        want, size, out = dst.double(), dst.abs().double(), dst.clone()
        factor = torch.tensor(scale, device="cuda").double()        # as the kernel has it, in fp32
        for _ in range(2):
            for at, t in src:
                want[at:at + t.numel()] += factor * t.double()
                size[at:at + t.numel()] += factor * t.double().abs()
            version = out._version
            add_pieces(out, src, scale, **form)
            assert out._version > version
        # a product and a sum in fp32, twice; what no piece covers stays as it is
        assert torch.all((out.double() - want).abs() <= size * 2.0 ** -22)
        covered = torch.zeros(n, dtype=torch.bool, device="cuda")
        for at, t in src:
            covered[at:at + t.numel()] = True
        assert torch.equal(out[~covered], dst[~covered])


class _Unit(nn.Module):
    def __init__(self, fallback):
        super().__init__()
        self.a = nn.Linear(64, 64)                                       # the bias makes the pieces behind it start at odd places
        self.odd = nn.Parameter(torch.randn(13) * 0.1)
        self.frozen = nn.Parameter(torch.randn(64) * 0.1, requires_grad=False)
        self.unused = nn.Parameter(torch.randn(100) * 0.1)
        self.b = nn.Linear(64, 64, bias=False)
        self.tok = nn.Embedding(7, 64, sparse=fallback == "sparse")

    def forward(self, x):
        h = torch.tanh(self.a(x)) * (1 + self.frozen) + self.odd.sum() + self.tok(torch.arange(x.shape[0], device=x.device) % 5)
        return self.b(h)


class _Model(nn.Module):
    def __init__(self, fallback):
        super().__init__()
        self.units = nn.ModuleList([_Unit(fallback), _Unit(fallback)])


@pytest.mark.parametrize("fallback", ["", "sparse", "layout"])
def test_sharded_gradients_are_the_dense_ones(comm, fallback):
    from asystem_amem_b200.bindings import NcclError
    from asystem_amem_b200.parallel import FSDP
    torch.manual_seed(0)
    plain = _Model(fallback).to("cuda", torch.bfloat16)
    model = _Model(fallback).to("cuda", torch.bfloat16)
    model.load_state_dict(plain.state_dict())
    fsdp = FSDP(model, comm)
    assert all(u.direct for u in fsdp.units)
    if fallback == "layout":        # a gradient that lies otherwise, as a user's hook may leave it
        for u in model.units:
            u.b.weight.register_post_accumulate_grad_hook(lambda p: setattr(p, "grad", p.grad.t().contiguous().t()))
    want = [torch.zeros_like(u.grad_shard, dtype=torch.float64) for u in fsdp.units]
    size = [w.clone() for w in want]
    for seed in (1, 2):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(33, 64, device="cuda", generator=g).to(torch.bfloat16)
        plain.zero_grad(set_to_none=True)
        h = x
        for u in plain.units:
            h = u(h)
        h.float().square().mean().backward()
        for u, w, s in zip(plain.units, want, size):
            # (a sparse gradient's rows of one id are added up here, in 64 bits)
            flat = torch.cat([(torch.zeros_like(p) if p.grad is None else p.grad if p.grad.layout == torch.strided else p.grad.double().to_dense())
                              .double().reshape(-1) for p in u.parameters()])
            w[:flat.numel()] += flat
            s[:flat.numel()] += flat.abs()
        fsdp.forward_units(x).float().square().mean().backward()
        assert all(p.grad is None for p in model.parameters())
    for u, w, s in zip(fsdp.units, want, size):
        # the same operators on the same numbers; one rounding to bf16 a pass where one of them sums in another order
        assert s.max() > 0 and torch.all((u.grad_shard.double() - w).abs() <= s * 2.0 ** -8 + s.max() * 2.0 ** -12)
    held = [u.grad_shard.clone() for u in fsdp.units]
    if not fallback:
        comm.pause()
        for u in fsdp.units:
            with pytest.raises(NcclError):
                u.reduce_grads()
        comm.resume()
        assert all(torch.equal(u.grad_shard, h) for u, h in zip(fsdp.units, held))
