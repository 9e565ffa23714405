"""The decoder's modules under torch's tracers and compilers, on the CPU: what these take of plain modules they take of them."""
import pytest
import torch
import torch.nn as nn

from asystem_amem_b200.models import LlamaConfig
from asystem_amem_b200.models import llama

CFG = LlamaConfig.tiny()


class Rope(nn.Module):
    def forward(self, x, cos, sin):
        return llama.apply_rope(x, cos, sin)


def _module(name):
    torch.manual_seed(0)
    m = {"norm": lambda: llama.RMSNorm(CFG.dim, 1e-5), "swiglu": lambda: llama.SwiGLU(CFG), "embed": lambda: llama.Embed(CFG), "rope": Rope,
         "head": lambda: llama.Head(CFG), "attention": lambda: llama.Attention(CFG), "block": lambda: llama.Block(CFG)}[name]()
    x = torch.randn(2, 6, CFG.dim)
    cos, sin = llama.rope_tables(6, CFG.dim // CFG.n_heads, CFG.rope_theta, "cpu")
    args = {"embed": (torch.arange(12).view(2, 6), cos, sin), "rope": (torch.randn(2, 4, 6, CFG.dim // CFG.n_heads), cos, sin)}.get(name)
    return m, args or ((x,) if name in ("norm", "swiglu") else (x, cos, sin))


@pytest.mark.parametrize("name", ["norm", "swiglu", "embed", "rope", "head", "attention", "block"])
def test_symbolic_trace(name):
    m, args = _module(name)
    traced = torch.fx.symbolic_trace(m)
    torch.testing.assert_close(traced(*args), m(*args), rtol=0, atol=0)
    if name == "embed":
        assert any(n.op == "call_module" and n.target == "tok" for n in traced.graph.nodes)


@pytest.mark.filterwarnings("ignore::DeprecationWarning")
@pytest.mark.parametrize("name", ["norm", "swiglu", "embed", "rope", "head", "attention", "block"])
def test_script(name):
    m, args = _module(name)
    with torch.no_grad():
        torch.testing.assert_close(torch.jit.script(m)(*args), m(*args), rtol=1e-5, atol=1e-5)     # fp32, its passes fused or not
