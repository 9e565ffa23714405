"""Routing of a mixture-of-experts layer as one kernel: the order of its choices, their weights, the gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# one, two and four tiles of tokens a block and of experts; experts, tokens and K that end inside a tile; k = E; the
# most experts
SIZES = [(1, 8, 2, 64), (7, 8, 8, 72), (33, 16, 4, 4096), (1200, 8, 2, 256), (5000, 8, 1, 136), (1300, 32, 8, 520), (5000, 24, 3, 64),
         (100, 40, 4, 1000), (1300, 64, 8, 4096), (40, 128, 6, 200), (20, 256, 256, 64), (9, 100, 5, 4104), (3, 1, 1, 8)]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _small_integers(T, E, d):
    """Operands whose logits are whole numbers up to 64, exact in every type, with many ties."""
    g = _gen(T + E)
    x = torch.randint(-1, 2, (T, d), device="cuda", generator=g) * (torch.rand(T, d, device="cuda", generator=g) < 48 / d)
    keep = x.abs().cumsum(1) <= 64
    return (x * keep).to(torch.bfloat16), torch.randint(-1, 2, (E, d), device="cuda", generator=g).to(torch.bfloat16)


@pytest.mark.parametrize("T,E,k,d", SIZES)
def test_choices_and_weights(T, E, k, d):
    from asystem_amem_b200.ops import route
    x, router = _small_integers(T, E, d)
    idx, w = route(x, router, k)
    top = (x.double() @ router.double().t()).sort(dim=1, descending=True, stable=True)     # equal values: lower index first
    assert idx.dtype == torch.int32 and torch.equal(idx.long(), top.indices[:, :k])
    ref = torch.softmax(top.values[:, :k], dim=1)
    # fp32: the exponential and the quotient to a few roundings, a sum of k terms
    assert torch.all((w.double() - ref).abs() <= ref * (k + 8) * 2.0 ** -23 + 1e-37)


@pytest.mark.parametrize("T,E,k,d", SIZES)
def test_gradients(T, E, k, d):
    from asystem_amem_b200.ops import route
    x = torch.randn(T, d, device="cuda", generator=_gen(1)).to(torch.bfloat16).requires_grad_(True)
    router = (torch.randn(E, d, device="cuda", generator=_gen(2)) * d ** -0.5).to(torch.bfloat16).requires_grad_(True)
    g = torch.randn(T, k, device="cuda", generator=_gen(3))
    idx, w = route(x, router, k)
    w.backward(g)
    logits = x.detach().double() @ router.detach().double().t()
    chosen = logits.gather(1, idx.long())
    # a choice may differ from the exact order by a rounding of two logits to bf16
    kth = logits.topk(k, dim=1).values[:, -1:]
    assert torch.all(chosen >= kth - 2 * 2.0 ** -8 * kth.abs() - 1e-6) and all(len(set(r)) == k for r in idx.tolist())
    # a rounding to bf16 (8 significant bits) is at most 2^-8 of the logit: as much twice over in every exponent
    off = 2 * 2.0 ** -8 * logits.abs().max(dim=1, keepdim=True).values + 2.0 ** -20
    ref = torch.softmax(chosen, dim=1)
    assert torch.all((w.detach().double() - ref).abs() <= ref * (off.exp() - 1) + 1e-37)
    # the logits' gradient from the weights as they came out, rounded to bf16; then sums of bf16 products, rounded
    wd, gd = w.detach().double(), g.double()
    gl = torch.zeros(T, E, device="cuda", dtype=torch.float64).scatter_(1, idx.long(), wd * (gd - (wd * gd).sum(1, keepdim=True)))
    spread = torch.zeros_like(gl).scatter_(1, idx.long(), wd * (gd.abs() + (wd * gd).abs().sum(1, keepdim=True)))
    for got, want, terms in ((x.grad, gl @ router.detach().double(), spread @ router.detach().double().abs()),
                             (router.grad, gl.t() @ x.detach().double(), spread.t() @ x.detach().double().abs())):
        assert torch.all((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + terms * (2.0 ** -8 + (T + E) * 2.0 ** -23) + 1e-30)


def test_every_form_that_torch_takes():
    from asystem_amem_b200.ops import route
    x = torch.randn(6, 64, device="cuda", generator=_gen(4)).to(torch.bfloat16)
    router = torch.randn(8, 64, device="cuda", generator=_gen(5)).to(torch.bfloat16)
    idx, w = route(x, router, 3)
    off = torch.empty(6 * 64 + 1, device="cuda", dtype=torch.bfloat16)[1:].view(6, 64).copy_(x)
    for a, b in ((x.t().contiguous().t(), router), (off, router), (x, router.t().contiguous().t())):
        i, v = route(a, b, 3)
        assert torch.equal(i, idx) and torch.allclose(v, w, rtol=2.0 ** -5)      # logits that round to bf16 apart
    assert route(x[:0], router, 3)[0].shape == (0, 3)
    with pytest.raises(RuntimeError):
        route(x, router, 9)
    # not-a-number sorts above everything, infinities as values; the softmax of either is torch's
    x[1, 0], x[2], router[3] = float("nan"), 1.0, float("inf")
    i, v = route(x, router, 3)
    top = (x @ router.t()).float().topk(3, dim=1)
    assert torch.equal(torch.softmax(top.values, dim=1).isnan(), v.isnan()) and i[1].tolist() == [0, 1, 2] and int(i[2, 0]) == 3
    # a gradient of the gradient
    a = torch.randn(6, 64, device="cuda", generator=_gen(6)).to(torch.bfloat16).requires_grad_(True)
    (ga,) = torch.autograd.grad(route(a, torch.ones_like(router), 3)[1].sum(), a, create_graph=True)
    assert ga.requires_grad


@pytest.fixture(scope="module")
def comm():
    from asystem_amem_b200 import Communicator, get_unique_id
    c = Communicator(1, 0, get_unique_id())
    yield c
    torch.cuda.synchronize()
    c.destroy()


# columns that end inside a warp's piece and in a second one, an odd number of choices, more than a warp looks up at once, no room
# for some rows
@pytest.mark.parametrize("T,E,k,d,room", [(1, 8, 1, 8, 1.0), (37, 8, 3, 1032, 1.0), (700, 16, 2, 4096, 1.0), (20, 64, 40, 264, 1.0), (300, 8, 2, 72, 0.5)])
def test_routing_and_dispatch_as_one_step(comm, T, E, k, d, room):
    from asystem_amem_b200.ops import MoeDispatcher, route
    from asystem_amem_b200.parallel import ep
    x0 = torch.randn(T, d, device="cuda", generator=_gen(7)).to(torch.bfloat16)
    router0 = (torch.randn(E, d, device="cuda", generator=_gen(8)) * d ** -0.5).to(torch.bfloat16)
    disp = MoeDispatcher(comm, E, d, max(1, int(T * k * room)))
    got = []
    for fused in (True, False):
        x, router = x0.clone().requires_grad_(True), router0.clone().requires_grad_(True)
        if fused:
            rows, offsets, pos, idx, w = ep.ep_route_dispatch(disp, x, router, k)
            assert type(rows.grad_fn).__name__ == "_RouteDispatchBackward"
        else:
            idx, w = route(x, router, k)
            rows, offsets, pos = ep.ep_dispatch(disp, x, idx)
        g_rows = torch.randn(rows.shape, device="cuda", generator=_gen(9)).to(torch.bfloat16)
        g_w = torch.randn(w.shape, device="cuda", generator=_gen(10))
        torch.autograd.backward([rows, w], [g_rows, g_w])
        got.append([rows.detach(), offsets, pos, idx, w.detach(), router.grad, x.grad])
    assert all(torch.equal(a, b) for a, b in zip(got[0][:6], got[1][:6]))
    # in 64 bits from the weights as they came out
    pos, idx, w, gd = got[0][2].long(), got[0][3].long(), got[0][4].double(), g_w.double()
    gl = torch.zeros(T, E, device="cuda", dtype=torch.float64).scatter_(1, idx, w * (gd - (w * gd).sum(1, keepdim=True)))
    spread = torch.zeros_like(gl).scatter_(1, idx, w * (gd.abs() + (w * gd).abs().sum(1, keepdim=True)))
    picked = torch.where((pos >= 0).unsqueeze(2), g_rows.double()[pos.clamp(min=0)], torch.zeros((), device="cuda", dtype=torch.float64))
    want, terms = picked.sum(1) + gl @ router0.double(), spread @ router0.double().abs()
    # one rounding of the sum to bf16, one of each logit's gradient, k + k additions and the softmax's gradient in fp32
    small = (3 * k + 16) * 2.0 ** -23
    assert torch.all((got[0][6].double() - want).abs() <= want.abs() * 2.0 ** -8 + terms * (2.0 ** -8 + small) + picked.abs().sum(1) * small + 1e-30)


def test_a_graph_through_routing_and_dispatch(comm):
    from asystem_amem_b200.ops import MoeDispatcher
    from asystem_amem_b200.parallel import ep
    x = torch.randn(6, 64, device="cuda", generator=_gen(11)).to(torch.bfloat16).requires_grad_(True)
    router = torch.randn(8, 64, device="cuda", generator=_gen(12)).to(torch.bfloat16).requires_grad_(True)
    out = ep.ep_route_dispatch(MoeDispatcher(comm, 8, 64, 12), x, router, 2)
    (gx,) = torch.autograd.grad(out[4].square().sum() + out[0].float().sum(), x, create_graph=True)
    assert gx.requires_grad and torch.autograd.grad(gx.float().sum(), router)[0].shape == router.shape


# more experts than one kernel routes in time: torch's operators without gradients and, for many tokens, with them
@pytest.mark.parametrize("T,E,k,d", [(40, 256, 8, 4096), (8200, 96, 2, 2056)])
def test_routing_over_many_experts(T, E, k, d):
    from asystem_amem_b200.ops import route
    from asystem_amem_b200.ops.moe import _route_pays
    assert not _route_pays(T, d, E)
    test_gradients(T, E, k, d)
    x = torch.randn(T, d, device="cuda", generator=_gen(1)).to(torch.bfloat16)
    router = (torch.randn(E, d, device="cuda", generator=_gen(2)) * d ** -0.5).to(torch.bfloat16)
    idx, w = route(x, router, k)
    logits = x.double() @ router.double().t()
    chosen = logits.gather(1, idx.long())
    # as in the test of the gradients: roundings of the logits to bf16
    kth, off = logits.topk(k, dim=1).values[:, -1:], 2 * 2.0 ** -8 * logits.abs().max(dim=1, keepdim=True).values + 2.0 ** -20
    assert idx.dtype == torch.int32 and torch.all(chosen >= kth - 2 * 2.0 ** -8 * kth.abs() - 1e-6)
    ref = torch.softmax(chosen, dim=1)
    assert torch.all((w.double() - ref).abs() <= ref * (off.exp() - 1) + 1e-37)
