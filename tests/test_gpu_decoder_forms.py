"""Where the decoder's kernels step aside: transforms, compilers, and embeddings that are more than a table."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _rand(shape, seed):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).to(BF16)


def test_rotary_embedding_under_transforms():
    from torch.func import jvp, vmap
    from asystem_amem_b200.models.llama import rope_tables
    from asystem_amem_b200.ops import rotate
    cos, sin = rope_tables(5, 16, 10000.0, "cuda")
    x, t = _rand((3, 2, 4, 5, 16), 1), _rand((2, 4, 5, 16), 2)
    turned = torch.stack([rotate(cos, sin, y)[0] for y in x])
    # both round once to bf16 what they compute in fp32
    close = dict(rtol=2.0 ** -7, atol=2.0 ** -20)
    torch.testing.assert_close(vmap(lambda y: rotate(cos, sin, y)[0])(x), turned, **close)
    out, tangent = jvp(lambda y: rotate(cos, sin, y)[0], (x[0],), (t,))
    torch.testing.assert_close(out, turned[0], **close)
    # the map is linear; torch's operators carry the tangent in fp32
    torch.testing.assert_close(tangent, rotate(cos, sin, t)[0], **close)


class _Doubled(nn.Embedding):
    def forward(self, ids):
        return 2 * super().forward(ids)


def _embeddings():
    make = lambda **kw: nn.Embedding(11, 16, **kw)

    def with_hook(register):
        t = make()
        t.calls = []
        getattr(t, register)(lambda *a: t.calls.append(1))
        return t

    def replaced():
        t = make()
        t.forward = lambda ids: F.embedding(ids, t.weight) + 1
        return t
    return {"plain": make, "padding": lambda: make(padding_idx=2), "largest norm": lambda: make(max_norm=0.5), "by frequency": lambda: make(scale_grad_by_freq=True),
            "sparse": lambda: make(sparse=True), "subclass": lambda: _Doubled(11, 16), "replaced": replaced,
            "forward hook": lambda: with_hook("register_forward_hook"), "forward pre-hook": lambda: with_hook("register_forward_pre_hook"),
            "backward hook": lambda: with_hook("register_full_backward_hook"), "backward pre-hook": lambda: with_hook("register_full_backward_pre_hook")}


@pytest.mark.parametrize("kind", _embeddings())
def test_an_embedding_keeps_what_it_does(kind):
    from asystem_amem_b200.models import LlamaConfig
    from asystem_amem_b200.models.llama import Embed
    torch.manual_seed(0)
    e = Embed(LlamaConfig.tiny())
    e.tok = _embeddings()[kind]().to("cuda", BF16)
    weight = e.tok.weight.detach().clone()
    ids = torch.tensor([[1, 2, 2, 7], [2, 10, 0, 1]], device="cuda")
    g = _rand((2, 4, 16), 3)
    out = e(ids)
    out.backward(g)
    hooked = len(getattr(e.tok, "calls", []))
    grad, e.tok.weight.grad = e.tok.weight.grad, None
    with torch.no_grad():
        e.tok.weight.copy_(weight)
    want = e.tok(ids)
    want.backward(g)
    assert torch.equal(out, want)
    assert grad.layout == e.tok.weight.grad.layout == (torch.sparse_coo if kind == "sparse" else torch.strided)
    a, b = (t.float().to_dense() for t in (grad, e.tok.weight.grad))
    # sums of up to three terms, rounded once or, for a sparse gradient and by torch's kernel, once a term
    assert torch.all((a - b).abs() <= 3 * 2.0 ** -8 * torch.zeros_like(a).index_add_(0, ids.reshape(-1), 2 * g.reshape(-1, 16).float().abs()))
    if hasattr(e.tok, "calls"):
        assert hooked == 1 and len(e.tok.calls) == 2
    if kind == "padding":
        assert torch.all(grad[2] == 0)


def test_a_hook_of_all_modules_sees_the_embedding():
    from asystem_amem_b200.models import LlamaConfig
    from asystem_amem_b200.models.llama import Embed
    e = Embed(LlamaConfig.tiny()).to("cuda", BF16)
    seen = []
    hook = nn.modules.module.register_module_forward_hook(lambda m, *_: seen.append(type(m)))
    try:
        e(torch.tensor([[1, 2]], device="cuda"))
    finally:
        hook.remove()
    assert nn.Embedding in seen


def test_the_decoder_compiles_whole():
    from asystem_amem_b200.models import LlamaConfig, LlamaDecoder
    cfg = LlamaConfig.tiny()
    torch.manual_seed(0)
    model = LlamaDecoder(cfg, device="cuda")
    ids = torch.randint(0, cfg.vocab_size, (2, 16), device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))

    def grads(f):
        model.zero_grad(set_to_none=True)
        logits = f(ids)
        F.cross_entropy(logits.float().view(-1, cfg.vocab_size), ids.view(-1)).backward()
        return logits.detach().float(), [p.grad.float() for p in model.parameters()]

    logits, eager = grads(model)
    again, compiled = grads(torch.compile(model, backend="aot_eager", fullgraph=True))
    # kernels round once where torch's operators round several times: a handful of bf16 roundings of the largest values
    assert (again - logits).abs().max() <= 16 * 2.0 ** -8 * logits.abs().max()
    for a, b in zip(compiled, eager):
        assert (a - b).abs().max() <= 32 * 2.0 ** -8 * b.abs().max() + 1e-6
