"""Layers and their gradients on tensors as a program leaves them: gradients that start at any element,
rows changed in place, results given at any address."""
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


def _rand(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


def _shifted(t):
    """The same values, contiguous, one element behind a 16-byte boundary."""
    flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
    view = flat[1:].view(t.shape)
    view.copy_(t)
    assert view.is_contiguous() and view.data_ptr() % 16
    return view


def test_moe_layer_with_a_gradient_that_starts_at_an_odd_address(comm):
    from asystem_amem_b200.models import MoELayer
    layer = MoELayer(comm, 64, 96, 4, 2, tokens_per_rank=33, capacity_factor=1.0)
    x, g = _rand((33, 64), 1), _rand((33, 64), 2)
    got = []
    for grad in (g, _shifted(g)):
        a = x.clone().requires_grad_(True)
        layer.zero_grad(set_to_none=True)
        layer(a).backward(grad)
        got.append([a.grad] + [p.grad for p in layer.parameters()])
    assert all(torch.equal(s, t) for s, t in zip(*got))


def test_moe_steps_on_rows_at_odd_addresses(comm):
    from asystem_amem_b200.ops import MoeDispatcher
    from asystem_amem_b200.parallel import ep
    T, k, E, d = 21, 3, 5, 72
    disp = MoeDispatcher(comm, E, d, T * k)
    idx = torch.randint(0, E, (T, k), generator=torch.Generator().manual_seed(3), dtype=torch.int32).cuda()
    w, x, y, g = torch.rand(T, k, device="cuda"), _rand((T, d), 4), _rand((T * k, d), 5), _rand((T, d), 6)
    rows, _, pos, _ = ep.dispatch_forward(disp, x, idx)
    assert torch.equal(ep.dispatch_forward(disp, _shifted(x), idx)[0], rows)
    assert torch.equal(disp.dispatch(_shifted(x), idx).recv_x[:T * k], rows)
    assert torch.equal(ep.combine_forward(disp, _shifted(y), idx, w, pos), ep.combine_forward(disp, y, idx, w, pos))
    assert torch.equal(ep.dispatch_backward(disp, _shifted(y), idx, pos), ep.dispatch_backward(disp, y, idx, pos))
    for a, b in zip(ep.combine_backward(disp, _shifted(g), _shifted(y), idx, w, pos), ep.combine_backward(disp, g, y, idx, w, pos)):
        assert torch.equal(a, b)


def test_dispatched_rows_changed_in_place(comm):
    from asystem_amem_b200.ops import MoeDispatcher
    from asystem_amem_b200.parallel.ep import ep_combine, ep_dispatch
    T, k, E, d = 21, 2, 4, 64
    disp = MoeDispatcher(comm, E, d, T * k - 5)      # a few rows find no room
    idx = torch.randint(0, E, (T, k), generator=torch.Generator().manual_seed(11), dtype=torch.int32).cuda()
    got = []
    for in_place in (False, True):
        x, w = _rand((T, d), 12).requires_grad_(True), torch.full((T, k), 0.5, device="cuda")
        rows, _, pos = ep_dispatch(disp, x, idx)
        assert rows.shape == (T * k - 5, d)
        rows = rows.mul_(2) if in_place else rows * 2
        out = ep_combine(disp, rows, w, idx, pos)
        out.backward(_rand((T, d), 13))
        got.append((out.detach(), x.grad))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_swiglu_with_a_gradient_that_starts_at_an_odd_address():
    from asystem_amem_b200.ops import swiglu
    h, g = _rand((33, 48), 7), _rand((33, 24), 8)
    got = []
    for grad in (g, _shifted(g)):
        a = h.clone().requires_grad_(True)
        swiglu(a).backward(grad)
        got.append(a.grad)
    assert torch.equal(*got)


@pytest.mark.parametrize("M,N,K", [(16, 72, 64), (64, 136, 1000), (65, 72, 64), (300, 264, 520), (1000, 1000, 256)])
@pytest.mark.parametrize("shift", [1, 4])
def test_gemm_into_a_result_at_an_odd_address(comm, M, N, K, shift):
    from asystem_amem_b200.ops import all_gather_gemm, gemm_bf16, gemm_reduce_scatter
    a, b = _rand((M, K), 9), _rand((N, K), 10)
    ref = a.float() @ b.float().t()
    for call in (gemm_bf16, lambda *x, **k: all_gather_gemm(comm, *x, **k), lambda *x, **k: gemm_reduce_scatter(comm, *x, **k)):
        buf = torch.full((M * N + 16,), 3.0, device="cuda", dtype=torch.bfloat16)
        out = buf[shift:shift + M * N].view(M, N)
        call(a, b, out=out)
        # one rounding to bf16 of fp32 sums: at most 2^-8 of the largest
        assert (out.float() - ref).abs().max().item() <= 2.0 ** -8 * ref.abs().max().item() + 1e-6
        assert torch.all(buf[:shift] == 3) and torch.all(buf[shift + M * N:] == 3)
