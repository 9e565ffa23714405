"""Dispatch and combine of a one-rank communicator against plain torch, at the sizes where the kernels
change their ways: the single-launch form's limit, tokens cut by a chunk, partial vectors, no room."""
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


@pytest.mark.parametrize("T,k,E,d", [(1, 1, 1, 8), (3, 2, 8, 2056), (341, 3, 33, 72), (1024, 8, 256, 64), (1025, 8, 64, 64), (4096, 2, 8, 264),
                                     (5000, 3, 256, 40), (130, 200, 256, 16), (2000, 33, 64, 16), (40, 1100, 7, 8)])
@pytest.mark.parametrize("room", [1.0, 0.6])
def test_dispatch_and_combine(comm, T, k, E, d, room):
    from asystem_amem_b200.ops import MoeDispatcher
    g = torch.Generator().manual_seed(T * 31 + k)
    idx = torch.randint(0, E, (T, k), generator=g, dtype=torch.int32)
    if T > 3:
        idx[1, 0], idx[2, 0] = -1, E        # no such expert: the pair goes nowhere
    x = torch.randn(T, d, generator=g).to(torch.bfloat16).cuda()
    w = torch.rand(T, k, generator=g).cuda()
    cap = max(1, int(T * k * room))
    disp = MoeDispatcher(comm, E, d, cap)
    flat = idx.reshape(-1).long()
    valid = (flat >= 0) & (flat < E)
    order = torch.argsort(torch.where(valid, flat, torch.full_like(flat, E)), stable=True)[: int(valid.sum())]
    pos = torch.full((T * k,), -1, dtype=torch.int64)
    pos[order] = torch.arange(order.numel())
    pos[pos >= cap] = -1
    counts = torch.bincount(flat[valid], minlength=E)
    offsets = torch.zeros(E + 1, dtype=torch.int64)
    offsets[1:] = counts.cumsum(0)
    for _ in range(2):
        res = disp.dispatch(x, idx.cuda())
        torch.cuda.synchronize()
        assert torch.equal(res.send_pos.cpu().reshape(-1).long(), pos)
        assert torch.equal(res.expert_offsets.cpu().long(), offsets.clamp(max=cap))
        assert torch.equal(res.expert_counts.cpu().long(), offsets.clamp(max=cap).diff())
        assert int(res.dropped) == max(0, int(valid.sum()) - cap)
        kept = order[:cap]
        assert torch.equal(res.recv_x[: kept.numel()], x[(kept // k).cuda()])
    disp.y[: kept.numel()] = torch.randn(kept.numel(), d, generator=g).to(torch.bfloat16).cuda()
    out = disp.combine(idx.cuda(), w, res.send_pos)
    ref = torch.zeros(T, d, dtype=torch.float64, device="cuda")
    size = torch.zeros_like(ref)
    for j in range(k):
        p = pos.view(T, k)[:, j].cuda()
        y = torch.where((p >= 0).unsqueeze(1), disp.y[p.clamp(min=0)].double() * w[:, j:j + 1].double(), torch.zeros((), dtype=torch.float64, device="cuda"))
        ref += y
        size += y.abs()
    # the sum's own rounding (k fp32 additions) and one rounding to bf16
    assert torch.all((out.double() - ref).abs() <= size * (k + 1) * 2.0 ** -24 + ref.abs() * 2.0 ** -8 + 1e-30)

    # the same steps between tensors, and the combine's backward
    if valid.any():
        own = disp.dispatch_local(x, idx.cuda())
        torch.cuda.synchronize()
        assert torch.equal(own.send_pos, res.send_pos) and torch.equal(own.expert_offsets, res.expert_offsets) and torch.equal(own.dropped, res.dropped)
        assert torch.equal(own.recv_x[: kept.numel()], res.recv_x[: kept.numel()])
        y = disp.y[: kept.numel()].clone()
        assert torch.equal(disp.combine_local(y, idx.cuda(), w, own.send_pos), out)
        g_out = torch.randn(T, d, generator=g).to(torch.bfloat16).cuda()
        g_y, g_w = disp.combine_grad_local(g_out, y, w, own.send_pos)
        p = pos.cuda().clamp(min=0)
        hit = (pos >= 0).cuda()
        tok = torch.arange(T * k, device="cuda") // k
        dots, sizes = torch.zeros(T * k, device="cuda", dtype=torch.float64), torch.zeros(T * k, device="cuda", dtype=torch.float64)
        for lo in range(0, T * k, 8192):
            s = slice(lo, lo + 8192)
            prod = g_out[tok[s]].double() * y[p[s]].double()
            dots[s], sizes[s] = prod.sum(1) * hit[s], prod.abs().sum(1)
        assert torch.all((g_w.reshape(-1).double() - dots).abs() <= sizes * (d / 128 + 16) * 2.0 ** -24 + 1e-30)
        assert torch.equal(g_y[p[hit]], (g_out[tok[hit]].float() * w.reshape(-1)[hit].unsqueeze(1)).to(torch.bfloat16))


# rows of at least 4 KB, more than four choices, in numbers that the bulk-copy engine gathers: five choices, eight, more
# than a stage takes (with a last pass of one), rows in uneven pieces and in three
@pytest.mark.parametrize("T,k,E,d", [(1400, 5, 5, 2056), (1000, 8, 64, 4096), (700, 16, 64, 2048), (530, 9, 256, 4104), (170, 33, 64, 12288)])
@pytest.mark.parametrize("room", [1.0, 0.6])
def test_combine_by_bulk_copies(comm, T, k, E, d, room):
    test_dispatch_and_combine(comm, T, k, E, d, room)


# rows in two uneven pieces, long enough to be gathered so
@pytest.mark.parametrize("T,k,E,d", [(530, 9, 256, 7000)])
@pytest.mark.parametrize("room", [1.0, 0.6])
def test_combine_of_rows_in_uneven_pieces(comm, T, k, E, d, room):
    test_dispatch_and_combine(comm, T, k, E, d, room)
