"""Collectives of a communicator of one rank: copies, scales and casts at every kind of size and address."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm():
    from asystem_amem_b200 import Communicator, get_unique_id
    c = Communicator(1, 0, get_unique_id())
    yield c
    torch.cuda.synchronize()
    c.destroy()


def _data(n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dtype.is_floating_point:
        return torch.randn(n, device="cuda", generator=g).to(dtype)
    return torch.randint(-100, 100, (n,), device="cuda", generator=g).to(dtype)


@pytest.mark.parametrize("n", [1, 7, 8, 4097, 65536, 1_000_003])
@pytest.mark.parametrize("dtype", [torch.int8, torch.float16, torch.bfloat16, torch.float32, torch.int64, torch.float64])
@pytest.mark.parametrize("shift", [0, 1])       # shifted by an element: no 16-byte alignment
def test_copies(comm, n, dtype, shift):
    x = _data(n + shift, dtype, n)[shift:]
    for call in ("all_reduce", "avg", "reduce", "broadcast", "all_gather", "all_to_all", "reduce_scatter"):
        out = torch.full((n + shift + 16,), 3, device="cuda", dtype=dtype)
        y = out[shift:shift + n]
        if call == "avg":
            if not dtype.is_floating_point:
                continue
            comm.all_reduce(x, y, op="avg")
        else:
            getattr(comm, call)(x, y)
        assert torch.equal(x, y), call
        assert torch.all(out[shift + n:] == 3)
    w = x.clone()
    comm.all_reduce(x)      # in place
    assert torch.equal(x, w)


@pytest.mark.parametrize("n", [1, 9, 4096, 1_000_003])
@pytest.mark.parametrize("tin,tout", [(torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16), (torch.float16, torch.float32), (torch.float32, torch.float32),
                                      (torch.bfloat16, torch.bfloat16)])
def test_scale_and_cast(comm, n, tin, tout):
    x = _data(n, tin, 1)
    for shift in (0, 1):
        out = torch.full((n + 17,), 3, device="cuda", dtype=tout)
        y = out[shift:shift + n]
        comm.reduce_scatter(x, y, scale=0.3)
        assert torch.equal(y, (x.float() * torch.tensor(0.3, device="cuda")).to(tout))
        assert torch.all(out[shift + n:] == 3)


def test_what_is_refused_stays_refused(comm):
    from asystem_amem_b200.bindings import NcclError
    x = torch.zeros(64, device="cuda")
    f8 = x.to(torch.float8_e4m3fn)
    with pytest.raises(NcclError):
        comm.all_reduce(f8, f8.clone())
    with pytest.raises(NcclError):
        comm.reduce_scatter(x.to(torch.bfloat16), x.to(torch.float16), scale=1.0)
    comm.all_gather(f8, torch.empty_like(f8))


def test_bounded_blocks(monkeypatch):
    from asystem_amem_b200 import Communicator, get_unique_id
    monkeypatch.setenv("AMEM_MAX_BLOCKS", "3")
    c = Communicator(1, 0, get_unique_id())
    for n in (1000, 1_000_003):       # one block, and more than three
        x, wide = _data(n, torch.bfloat16, n), torch.empty(n, device="cuda")
        out = torch.empty_like(x)
        c.all_reduce(x, out)
        c.reduce_scatter(x, wide, scale=0.25)
        assert torch.equal(out, x) and torch.equal(wide, x.float() * 0.25)
    torch.cuda.synchronize()
    c.destroy()
