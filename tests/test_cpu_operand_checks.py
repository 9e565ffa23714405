"""What the Python entry points of the kernels refuse or re-lay before anything is launched.  No GPU: the
tensors only say that they are on one, and the library is a recorder."""
from types import SimpleNamespace

import pytest
import torch

from asystem_amem_b200 import bindings as B

BF16 = torch.bfloat16


class OnGpu(torch.Tensor):
    is_cuda = property(lambda self: True)


def gpu(*shape, dtype=BF16):
    return torch.zeros(*shape, dtype=dtype).as_subclass(OnGpu)


class Recorder:
    """Stands for the library: every entry point notes its call and succeeds."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append((name, args))
            return 0
        return entry


@pytest.fixture
def lib(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(B, "load_library", lambda *a, **k: rec)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(cuda_stream=0))
    return rec


@pytest.mark.parametrize("make", [gpu, lambda *shape: torch.zeros(*shape, dtype=BF16)])
def test_products_refuse_other_ranks_and_inner_dimensions(lib, make):
    from asystem_amem_b200 import ops
    offs = torch.zeros(3, dtype=torch.int32).as_subclass(OnGpu)
    wrong = [
        lambda: ops.gemm_swiglu(make(2, 16, 64), make(32, 64)),
        lambda: ops.gemm_swiglu(make(16, 64), make(32, 72)),
        lambda: ops.gemm_swiglu(make(16, 64), make(33, 64)),
        lambda: ops.gemm_input_grad(make(16, 64), make(72, 8)),
        lambda: ops.gemm_input_grad(make(2, 16, 64), make(64, 8)),
        lambda: ops.gemm_weight_grad(make(16, 64), make(24, 8)),
        lambda: ops.gemm_weight_grad(make(2, 16, 64), make(2, 8)),
        lambda: ops.grouped_gemm_input_grad(make(16, 64), make(2, 72, 8), offs),
        lambda: ops.grouped_gemm_input_grad(make(16, 64), make(2, 64, 8), offs, out=make(8, 8)),
        lambda: ops.grouped_gemm_input_grad(make(2, 64, 3), make(2, 64, 8), offs),
        lambda: ops.grouped_gemm_weight_grad(make(16, 64), make(24, 8), offs),
        lambda: ops.grouped_gemm_weight_grad(make(16, 64, 2), make(16, 8), offs),
    ]
    for i, call in enumerate(wrong):
        with pytest.raises(ValueError):
            call()
            raise AssertionError(f"call {i} went through")
    assert lib.calls == []


def test_an_mlp_refuses_a_batch_of_sequences(lib):
    from asystem_amem_b200.models import TPMLP
    layer = TPMLP(SimpleNamespace(nranks=1, lib=lib, _h=1), 64, 32, device="cpu")
    layer.w13.weight = torch.nn.Parameter(layer.w13.weight.detach().as_subclass(OnGpu), requires_grad=False)
    with torch.no_grad(), pytest.raises(ValueError):
        layer(gpu(2, 16, 64))
    assert [name for name, _ in lib.calls if "Gemm" in name] == []
