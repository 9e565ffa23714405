"""The element-wise kernels and the fused gate / up projection against plain torch in fp32 / fp64."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _rand(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("rows,f", [(1, 8), (3, 24), (257, 1000), (70, 14336), (0, 64)])
def test_swiglu_and_its_gradient(rows, f):
    from asystem_amem_b200.ops import swiglu
    h = _rand((rows, 2 * f), 1, 3.0)
    if rows > 2:
        h[1, 0], h[1, f], h[2, 1] = 80.0, -80.0, -80.0
    g = _rand((rows, f), 2)
    a = h.clone().requires_grad_(True)
    out = swiglu(a)
    out.backward(g)
    b = h.double().requires_grad_(True)
    ref = F.silu(b[:, :f]) * b[:, f:]
    ref.backward(g.double())
    # one rounding to bf16 (8 significant bits: at most 2^-8 of the value) of a value computed in fp32, where
    # 1 + gate * (1 - sigmoid) loses at most 9 of 22 bits next to its zero (bf16 gates stay 0.0028 away)
    for x, y in ((out, ref), (a.grad, b.grad)):
        assert torch.all((x.double() - y).abs() <= y.abs() * (2.0 ** -8 + 2.0 ** -12) + 1e-30)
    assert torch.equal(swiglu(h), out)


# rows of both kernels' tiles, features that end inside a 32-column chunk, products cut along K
@pytest.mark.parametrize("M,f,K", [(1, 8, 64), (16, 64, 1000), (64, 1000, 4096), (65, 104, 72), (129, 264, 4096), (257, 1000, 264), (500, 200, 8192)])
def test_gate_up_projection(M, f, K):
    from asystem_amem_b200.ops import gemm_swiglu
    x, w = _rand((M, K), 3), _rand((2 * f, K), 4, K ** -0.5)
    h = x.float() @ w.float().t()
    ref = F.silu(h[:, :f]) * h[:, f:]
    for _ in range(2):
        out = gemm_swiglu(x, w)
        assert (out.float() - ref).abs().max().item() <= 2.0 ** -8 * ref.abs().max().item() + 1e-6


# one, two and four vectors a thread, rows that end inside one, more rows than blocks; 16392 and 20: torch's operators
@pytest.mark.parametrize("rows,dim", [(1, 8), (3, 256), (5, 264), (700, 2048), (601, 4104), (9, 8200), (2, 16384), (2, 16392), (7, 20)])
def test_rms_norm_and_its_gradients(rows, dim):
    from asystem_amem_b200.ops import rms_norm
    x, w, g = _rand((rows, dim), 5, 2.0), _rand((dim,), 6), _rand((rows, dim), 7)
    x[0] = 0
    a, b = x.clone().requires_grad_(True), w.clone().requires_grad_(True)
    out = rms_norm(a, b, 1e-5)
    out.backward(g)
    c, d = x.double().requires_grad_(True), w.double().requires_grad_(True)
    ref = c * torch.rsqrt(c.pow(2).mean(-1, keepdim=True) + 1e-5) * d
    ref.backward(g.double())
    # one rounding to bf16 of values computed in fp32: those of the result to a few of its roundings and half that of a
    # sum of dim squares, the gradients' differences to as much of their larger term, the weight's sum to as many
    # roundings of its terms as it has
    assert torch.all((out.double() - ref).abs() <= ref.abs() * (2.0 ** -8 + 2.0 ** -14))
    r = torch.rsqrt(c.detach().pow(2).mean(-1, keepdim=True) + 1e-5)
    n, gw = c.detach() * r, g.double() * w.double()
    larger = r * (gw.abs() + n.abs() * (gw * n).abs().mean(-1, keepdim=True))
    assert torch.all((a.grad.double() - c.grad).abs() <= c.grad.abs() * 2.0 ** -8 + larger * 2.0 ** -14)
    terms = (g.double() * n).abs().sum(0)
    assert torch.all((b.grad.double() - d.grad).abs() <= d.grad.abs() * 2.0 ** -8 + terms * (rows + 16) * 2.0 ** -23)
    assert torch.equal(rms_norm(x, w, 1e-5), out)


def test_rms_norm_in_every_form_that_torch_takes():
    from torch.func import jvp, vmap
    from asystem_amem_b200.ops import rms_norm
    x, w = _rand((6, 64), 8), _rand((64,), 9)
    want = rms_norm(x, w, 1e-5)
    close = dict(rtol=2.0 ** -7, atol=1e-6)       # two roundings of one value
    torch.testing.assert_close(rms_norm(x.t().contiguous().t(), w, 1e-5), want, **close)
    off = torch.empty(6 * 64 + 1, device="cuda", dtype=torch.bfloat16)[1:].view(6, 64).copy_(x)
    torch.testing.assert_close(rms_norm(off, w, 1e-5), want, **close)
    torch.testing.assert_close(rms_norm(x.view(2, 3, 64), w, 1e-5).view(6, 64), want, rtol=0, atol=0)
    torch.testing.assert_close(rms_norm(x.float(), w, 1e-5), want.float(), **close)
    torch.testing.assert_close(vmap(lambda r: rms_norm(r, w, 1e-5))(x), want, **close)
    torch.testing.assert_close(jvp(lambda t: rms_norm(t, w, 1e-5), (x,), (x,))[0], want, **close)
    assert rms_norm(x[:0], w, 1e-5).shape == (0, 64)
    # only the input, only the weight, and a gradient of the gradient
    a = x.clone().requires_grad_(True)
    (gx,) = torch.autograd.grad(rms_norm(a, w, 1e-5).float().pow(2).sum(), a, create_graph=True)
    (hx,) = torch.autograd.grad(gx.float().sum(), a)
    b = x.double().requires_grad_(True)
    r = b * torch.rsqrt(b.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
    (gr,) = torch.autograd.grad(r.pow(2).sum(), b, create_graph=True)
    (hr,) = torch.autograd.grad(gr.sum(), b)
    # some ten roundings to bf16 of terms of the size of the largest
    assert (hx.double() - hr).abs().max().item() <= 10 * 2.0 ** -8 * max(gr.abs().max().item(), hr.abs().max().item())
    v = w.clone().requires_grad_(True)
    rms_norm(x, v, 1e-5).backward(x)
    assert v.grad is not None and v.grad.shape == v.shape


def _turned(x, cos, sin):
    x1, x2, c, s = x[..., 0::2], x[..., 1::2], cos.double(), sin.double()
    return torch.stack((x1 * c - x2 * s, x1 * s + x2 * c), dim=-1).flatten(-2)


# heads inside positions (a projection's output), contiguous, and a slice of a wider tensor; blocks of one warp, items
# that do not fill the last one, more items than threads; 12 is no multiple of 8: torch's operators
@pytest.mark.parametrize("lie", ["tokens", "heads", "slice"])
@pytest.mark.parametrize("b,h,kv,s,d", [(1, 1, 1, 1, 8), (2, 3, 1, 5, 24), (1, 16, 4, 33, 128), (2, 20, 20, 7, 256), (1, 2, 1, 3, 12)])
def test_rotary_embedding_and_its_gradient(lie, b, h, kv, s, d):
    from asystem_amem_b200.models.llama import apply_rope, rope_tables
    from asystem_amem_b200.ops import rotate
    cos, sin = rope_tables(s, d, 10000.0, "cuda")

    def lay(heads, seed):
        if lie == "heads":
            return _rand((b, heads, s, d), seed)
        if lie == "tokens":
            return _rand((b, s, heads, d), seed).transpose(1, 2)
        return _rand((b, s, heads + 1, d + 16), seed)[:, :, 1:, 8:8 + d].transpose(1, 2)

    q, k, gq, gk = lay(h, 1), lay(kv, 2), lay(h, 3), lay(kv, 4)
    a, c = q.clone(memory_format=torch.preserve_format).requires_grad_(True), k.clone(memory_format=torch.preserve_format).requires_grad_(True)
    for x, y, as_they_lie in ((q, k, True), (a, c, False)):
        outs = rotate(cos, sin, x, y, as_they_lie=as_they_lie)
        for t, o in zip((x, y), outs):
            ref = _turned(t.detach().double(), cos, sin)
            # one rounding to bf16 of a difference of products in fp32
            assert torch.all((o.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + t.detach().abs().max().item() * 2.0 ** -22)
            assert as_they_lie or o.is_contiguous()
    torch.autograd.backward(outs, (gq, gk))
    for t, g in ((a, gq), (c, gk)):
        ref = _turned(g.double(), cos, -sin)
        assert torch.all((t.grad.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + g.abs().max().item() * 2.0 ** -22)
    assert torch.equal(apply_rope(q, cos, sin), outs[0]) and apply_rope(q, cos, sin).is_contiguous()
    # the gradient of the gradient: the map is linear, so the turn itself
    (g1,) = torch.autograd.grad(rotate(cos, sin, a)[0], a, gq.clone().requires_grad_(True), create_graph=True)
    assert g1.requires_grad and torch.equal(g1, a.grad)


# ids that repeat within and across the 256 that a block looks at, all the same, few of many; columns in two passes
@pytest.mark.parametrize("shape,rows,d", [((1,), 3, 8), ((2, 300), 40, 24), ((5, 257), 1, 64), ((1000,), 5000, 2056), ((3, 1000), 700, 128)])
def test_embedding_gradient(shape, rows, d):
    from asystem_amem_b200.ops import embedding
    ids = torch.randint(0, rows, shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(21))
    table, g = _rand((rows, d), 22).requires_grad_(True), _rand((*shape, d), 23)
    out = embedding(ids, table)
    out.backward(g)
    assert torch.equal(out.detach(), table.detach()[ids])
    ref, size = (torch.zeros(rows, d, device="cuda", dtype=torch.float64).index_add(0, ids.reshape(-1), t.reshape(-1, d).double()) for t in (g, g.abs()))
    # fp32 sums of as many terms as an id has, rounded once
    assert torch.all((table.grad.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + size * ids.numel() * 2.0 ** -24)
    first = table.grad.clone()
    table.grad = None
    embedding(ids, table).backward(g)
    assert torch.equal(table.grad, first)


@pytest.mark.parametrize("shape", [(1, 8), (3, 5, 24), (2, 100, 1000), (2, 3, 20), (0, 16)])
def test_gated_and_its_gradients(shape):
    from torch.func import vmap
    from asystem_amem_b200.ops import gated
    x, u, g = _rand(shape, 11, 3.0), _rand(shape, 12), _rand(shape, 13)
    a, b = x.clone().requires_grad_(True), u.clone().requires_grad_(True)
    out = gated(a, b)
    out.backward(g)
    c, d = x.double().requires_grad_(True), u.double().requires_grad_(True)
    ref = F.silu(c) * d
    ref.backward(g.double())
    # as swiglu's bound above; torch's operators (rows of 20) round silu and the product of a gradient to bf16 on the way
    roundings = 1 if shape[-1] % 8 == 0 else 4
    for y, r in ((out, ref), (a.grad, c.grad), (b.grad, d.grad)):
        assert torch.all((y.double() - r).abs() <= r.abs() * (roundings * 2.0 ** -8 + 2.0 ** -12) + (1e-30 if roundings == 1 else 2.0 ** -6))
    assert torch.equal(gated(x, u), out)
    if x.numel() and len(shape) == 3:
        torch.testing.assert_close(vmap(gated)(x, u), out.detach(), rtol=3 * 2.0 ** -8, atol=1e-6)   # three roundings
        (ga,) = torch.autograd.grad(gated(a, b), a, g, create_graph=True)
        assert ga.requires_grad


@pytest.mark.parametrize("n", [1, 3, 4, 1000, 1_000_003])
@pytest.mark.parametrize("wd", [0.0, 0.1])
def test_adamw(n, wd):
    from asystem_amem_b200.ops import adamw_step
    gen = torch.Generator(device="cuda").manual_seed(n)
    master = torch.randn(n, device="cuda", generator=gen)
    m, v, shard = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda"), torch.empty(n, device="cuda", dtype=torch.bfloat16)
    p = torch.nn.Parameter(master.double())
    opt = torch.optim.AdamW([p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=wd)
    for step in range(1, 4):
        grad = torch.randn(n, device="cuda", generator=gen) * 0.1
        adamw_step(grad, m, v, master, shard, 1e-2, (0.9, 0.95), 1e-8, wd, step)
        p.grad = grad.double()
        opt.step()
    # three updates of about lr each, every operation to 2^-23
    assert (master.double() - p.detach()).abs().max().item() <= 3 * (p.detach().abs().max().item() * 2.0 ** -23 + 1e-2 * 2.0 ** -20)
    assert torch.equal(shard, master.to(torch.bfloat16))


def test_adamw_takes_a_rate_in_a_tensor_and_counts_as_an_in_place_update():
    from asystem_amem_b200.ops import adamw_step
    got, want = ([torch.full((8,), 0.5, device="cuda") for _ in range(4)] + [torch.empty(8, device="cuda", dtype=torch.bfloat16)] for _ in range(2))
    versions = [t._version for t in got]
    adamw_step(*got, torch.tensor(1e-2), (0.9, 0.95), 1e-8, 0.1, 1)
    adamw_step(*want, 1e-2, (0.9, 0.95), 1e-8, 0.1, 1)
    # the rate passed through fp32: 2^-24 of it
    assert all(torch.allclose(a, b, rtol=2.0 ** -22, atol=0) for a, b in zip(got[:4], want[:4]))
    assert got[0]._version == versions[0] and all(t._version > n for t, n in zip(got[1:], versions[1:]))


def test_a_replaced_projection_is_called():
    from asystem_amem_b200 import Communicator, get_unique_id
    from asystem_amem_b200.models import TPMLP
    from asystem_amem_b200.parallel.tp import ColumnParallelLinear

    class Doubled(ColumnParallelLinear):
        def forward(self, x):
            return 2 * super().forward(x)

    comm = Communicator(1, 0, get_unique_id())
    layer, x = TPMLP(comm, 128, 256), _rand((16, 128), 5)
    with torch.no_grad():
        own = Doubled(128, 512, comm)
        own.weight.copy_(layer.w13.weight)
        layer.w13 = own
        out = layer(x)
        h = 2 * (x.float() @ own.weight.float().t())
        ref = (F.silu(h[:, :256]) * h[:, 256:]) @ layer.w2.weight.float().t()
    # bf16 roundings of h, the activation and the result: a few of 2^-9 each, against the largest result
    assert (out.float() - ref).abs().max().item() <= 2.0 ** -6 * ref.abs().max().item()
    torch.cuda.synchronize()
    comm.destroy()


def test_adamw_other_layouts_take_the_plain_form():
    from asystem_amem_b200.ops import adamw_step
    base = [torch.rand(17, device="cuda") for _ in range(4)]
    got = [t.clone()[1:] for t in base]       # not 16-byte aligned
    want = [t.clone()[1:].clone() for t in base]
    for ts in (got, want):
        shard = torch.empty(16, device="cuda", dtype=torch.bfloat16)
        adamw_step(*ts, shard, 1e-3, (0.9, 0.95), 1e-8, 0.0, 1)
    for a, b in zip(got, want):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-7)


def test_swiglu_keeps_the_precision_of_fp32():
    """Every bf16 gate against 64 bits: half a unit of bf16 for the one rounding, and before it expf (1 ulp, as
    documented), an addition, a quotient and the products at half an ulp each -- for the gradient's 1 + gate *
    (1 - sigmoid) relative to the size of its terms."""
    from asystem_amem_b200.ops import swiglu
    gate = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    gate = gate[torch.isfinite(gate) & (gate.abs() < 1e18)]
    gate = gate[: gate.numel() // 8 * 8]
    rows = [1.0, -3.140625, 1.0078125e3, 2.0 ** -20, 3.0e36]
    up = torch.tensor(rows, device="cuda").to(torch.bfloat16).unsqueeze(1).expand(len(rows), gate.numel())
    h = torch.cat([gate.expand(len(rows), -1), up], dim=1).contiguous().requires_grad_(True)
    g = torch.full(up.shape, 1.5078125, device="cuda", dtype=torch.bfloat16)
    out = swiglu(h)
    (gh,) = torch.autograd.grad(out, h, g)
    x, u, f = gate.double().expand_as(up), up.double(), gate.numel()
    s = torch.sigmoid(x)
    eps = 2.0 ** -24                # half an ulp
    # where exp(-x) leaves fp32 (x < -88.7) the plain form in fp32 gives zero as well
    inside = x > -88.7

    def check(got, want, size, ulps):
        room = 2.0 ** (torch.floor(torch.log2(want.abs().clamp(min=2.0 ** -126))) - 8) + size * ulps * eps + 2.0 ** -133
        bad = inside & want.abs().lt(3e38) & ((got.double() - want).abs() > room)
        assert not bad.any(), (x[bad][:5], got[bad][:5], want[bad][:5])

    check(out.detach(), x * s * u, (x * s * u).abs(), 5)
    check(gh[:, f:], 1.5078125 * x * s, (1.5078125 * x * s).abs(), 5)
    scale = 1.5078125 * u.abs() * s
    check(gh[:, :f], 1.5078125 * u * s * (1 + x * (1 - s)), scale * (1 + (x * (1 - s)).abs()), 10)


# as many rows as change the forward's threads and more, blocks of the gradient that take three rows and more; one, two and four
# vectors a thread, the last of them part-filled
@pytest.mark.parametrize("rows,dim", [(1184, 2048), (2500, 264), (1900, 4104), (1800, 8200)])
def test_rms_norm_of_many_rows(rows, dim):
    test_rms_norm_and_its_gradients(rows, dim)
