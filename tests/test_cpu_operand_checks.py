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
    monkeypatch.setattr(torch.cuda, "current_device", lambda: -1)
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *args, **kw: empty(*args, **kw).as_subclass(OnGpu))
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
    layer = _mlp(lib)
    with torch.no_grad(), pytest.raises(ValueError):
        layer(gpu(2, 16, 64))
    assert [name for name, _ in lib.calls if "Gemm" in name] == []


# ------------------------------------------------------------------ rows that start at odd addresses

def shifted(*shape):
    """A contiguous tensor that starts 2 bytes behind a 16-byte boundary."""
    n = 1
    for s in shape:
        n *= s
    flat = torch.arange(n + 1, dtype=torch.float32).to(BF16)
    assert flat.data_ptr() % 16 == 0
    return flat[1:].view(*shape).as_subclass(OnGpu)


def _backward(out, g):
    torch.autograd.backward(out.as_subclass(torch.Tensor), g)     # (a subclass's own backward() would shed the subclass inside)


def _dispatcher(lib, E=4, d=8, capacity=64):
    from asystem_amem_b200.ops import MoeDispatcher
    disp = object.__new__(MoeDispatcher)
    disp.comm, disp.E, disp.d, disp.capacity, disp.experts_per_rank, disp.host = SimpleNamespace(nranks=1, lib=lib, _h=1), E, d, capacity, E, False
    disp.y, disp.recv_x = gpu(capacity, d), gpu(capacity, d)
    return disp


def test_moe_steps_hand_over_rows_on_16_bytes(lib):
    from asystem_amem_b200.parallel import ep
    disp, idx, w, pos = _dispatcher(lib), torch.zeros(6, 2, dtype=torch.int32), torch.ones(6, 2), torch.zeros(6, 2, dtype=torch.int32)
    disp.dispatch(shifted(6, 8), idx)
    disp.dispatch_local(shifted(6, 8), idx)
    ep.combine_forward(disp, shifted(12, 8), idx, w, pos)
    ep.dispatch_backward(disp, shifted(12, 8), idx, pos)
    ep.combine_backward(disp, shifted(6, 8), shifted(12, 8), idx, w, pos)
    rows = {"amemMoeDispatchCounted": [0], "amemMoeDispatchLocal": [0, 6], "amemMoeCombineLocal": [3, 5], "amemMoeCombineGradLocal": [0, 1, 4]}
    assert {name for name, _ in lib.calls} == set(rows)
    for name, args in lib.calls:
        assert all(args[i] % 16 == 0 for i in rows[name]), name


def test_moe_steps_between_tensors_take_what_fits_only(lib):
    """More rows than the dispatcher's buffers hold, or gradients of another number of tokens, take the general form."""
    from asystem_amem_b200.parallel import ep
    disp, idx, w, pos = _dispatcher(lib, capacity=8), torch.zeros(6, 2, dtype=torch.int32), torch.ones(6, 2), torch.zeros(6, 2, dtype=torch.int32)
    for call in (lambda: ep.combine_forward(disp, gpu(12, 8), idx, w, pos), lambda: ep.dispatch_backward(disp, gpu(12, 8), idx, pos),
                 lambda: ep.combine_backward(disp, gpu(5, 8), gpu(8, 8), idx, w, pos)):
        with pytest.raises(RuntimeError):
            call()
    assert all("Local" not in name for name, _ in lib.calls)


def test_moe_entry_points_refuse_unaligned_and_missing_rows(monkeypatch):
    """The C side says so too (no GPU: the refusal comes before anything else)."""
    monkeypatch.setenv("AMEM_BACKEND", "mock")
    from asystem_amem_b200 import Communicator, get_unique_id
    comm = Communicator(1, 0, get_unique_id())
    lib = comm.lib
    ok, odd = 4096, 4098     # never dereferenced

    def status(x, y, table):
        return {lib.amemMoeDispatchLocal(x, table, 4, 1, 8, 2, y, 4, table, table, table, None, comm._h, None),
                lib.amemMoeCombineLocal(table, table, table, x, 4, y, 4, 1, 8, 2, comm._h, None),
                lib.amemMoeCombineGradLocal(x, y, table, table, ok, table, 4, 4, 1, 8, comm._h, None),
                lib.amemMoeCombineGradLocal(ok, y, table, table, x, table, 4, 4, 1, 8, comm._h, None)}

    for x, y, table in ((odd, ok, ok), (ok, odd, ok), (None, ok, ok), (ok, None, ok), (ok, ok, None)):
        assert status(x, y, table) == {4}, (x, y, table)      # ncclInvalidArgument
    assert lib.amemMoeDispatch(odd, ok, 4, 1, 8, 2, 4, ok, ok, ok, comm._h, None) == 4
    assert lib.amemMoeCombine(ok, ok, ok, odd, 4, 1, 8, 2, 4, comm._h, None) == 4
    comm.destroy()


def test_gradients_at_odd_addresses_reach_the_kernels_on_16_bytes(lib):
    from asystem_amem_b200.models.moe_layer import GroupedLinear
    from asystem_amem_b200.ops import swiglu
    h = gpu(6, 32).requires_grad_(True)
    _backward(swiglu(h), shifted(6, 16))
    w, offs = gpu(2, 16, 8).requires_grad_(True), torch.tensor([0, 2, 6], dtype=torch.int32).as_subclass(OnGpu)
    _backward(GroupedLinear.apply(gpu(6, 8), w, offs), shifted(6, 16))
    rows = {"amemSwiGLUGrad": 3, "amemGroupedGemmBf16Weight": 0}
    seen = {name: args for name, args in lib.calls}
    assert all(seen[name][i] % 16 == 0 for name, i in rows.items())


# ------------------------------------------------------------------ tensors on another device than the current one

def test_launches_make_the_operands_device_current(lib, monkeypatch):
    from asystem_amem_b200 import ops
    current = [0]

    class Device:
        def __init__(self, index):
            self.index = index

        def __enter__(self):
            current.append(self.index)

        def __exit__(self, *exc):
            current.pop()

    monkeypatch.setattr(torch.cuda, "current_device", lambda: current[-1])
    monkeypatch.setattr(torch.cuda, "device", Device)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(cuda_stream=100 + current[-1]))
    monkeypatch.setattr(OnGpu, "get_device", lambda self: 3, raising=False)
    offs = torch.tensor([0, 2, 6], dtype=torch.int32).as_subclass(OnGpu)
    h = gpu(6, 32).requires_grad_(True)
    _backward(ops.swiglu(h), gpu(6, 16))
    ops.adamw_step(*(gpu(16, dtype=torch.float32) for _ in range(4)), gpu(16), 1e-3, (0.9, 0.95), 1e-8, 0.0, 1)
    ops.gemm_swiglu(gpu(8, 64), gpu(16, 64))
    ops.gemm_input_grad(gpu(8, 64), gpu(64, 16))
    ops.gemm_weight_grad(gpu(8, 64), gpu(8, 16))
    ops.grouped_gemm_input_grad(gpu(6, 16), gpu(2, 16, 64), offs)
    ops.grouped_gemm_weight_grad(gpu(6, 16), gpu(6, 64), offs)
    ops.gemm_input_grad(w=gpu(64, 16), gy=gpu(8, 64))
    ops.adamw_step(lr=1e-3, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.0, step=1, grad=gpu(16, dtype=torch.float32), m=gpu(16, dtype=torch.float32),
                   v=gpu(16, dtype=torch.float32), master=gpu(16, dtype=torch.float32), shard=gpu(16))
    assert len(lib.calls) == 10 and all(args[-1] == 103 for _, args in lib.calls), lib.calls
    assert current == [0]


@pytest.mark.parametrize("short", range(5))
def test_adamw_of_different_sizes_is_refused_as_torch_refuses_it(lib, short):
    from asystem_amem_b200 import ops
    ts = [gpu(16, dtype=torch.float32) for _ in range(4)] + [gpu(16)]
    ts[short] = ts[short][:8]
    with pytest.raises(RuntimeError):
        ops.adamw_step(*ts, 1e-3, (0.9, 0.95), 1e-8, 0.0, 1)
    assert lib.calls == []


# ------------------------------------------------------------------ results, and which kernel writes them

def test_gemm_refuses_a_result_that_no_kernel_can_store(monkeypatch):
    monkeypatch.setenv("AMEM_BACKEND", "mock")
    from asystem_amem_b200 import Communicator, get_unique_id
    comm = Communicator(1, 0, get_unique_id())
    lib = comm.lib
    ok, odd = 4096, 4098     # never dereferenced
    for m in (16, 512):
        assert lib.amemGemmBf16(odd, ok, odd, m, 64, 64, None) == 4      # ncclInvalidArgument
        assert lib.amemAllGatherGemm(ok, odd, odd, m, 64, 64, comm._h, None) == 4
        assert lib.amemGemmReduceScatter(odd, ok, odd, m, 64, 64, comm._h, None) == 4
        assert lib.amemGemmBf16(ok, ok, ok + 1, m, 64, 64, None) == 4
    comm.destroy()


def test_which_gemm_runs_and_how_it_is_tiled(monkeypatch):
    """(form, tile, slices) on 148 SMs: 2 = few rows, 1 = SM pairs, 0 = one SM."""
    import ctypes

    def form(M, N, K):
        v = [ctypes.c_int() for _ in range(3)]
        assert B.load_library().amemGemmForm(M, N, K, 148, *map(ctypes.byref, v)) == 0
        return tuple(x.value for x in v)

    assert form(16, 7168, 8192) == (2, 16, 2)          # 56 weight tiles: cut evenly over the SMs
    assert form(16, 18944, 3584) == (2, 16, 1)         # a weight tile per SM: whole
    assert form(64, 512, 4096)[0] == 2 and form(65, 512, 4096)[0] == 1
    assert form(1000, 3584, 8192) == (1, 224, 1)       # 64 whole tiles for 74 pairs
    assert form(2560, 256, 8192) == (1, 256, 7)        # the most chunks that a cut tile's ring takes
    assert form(8192, 7168, 8192) == (1, 224, 1)       # 1024 tiles: 14 waves of 74, the last 62 of them
    monkeypatch.setenv("AMEM_GEMM_TALL", "0")
    assert form(8192, 7168, 8192)[0] == 0


# ------------------------------------------------------------------ what a fused path must not pass by

def _mlp(lib):
    from asystem_amem_b200.models import TPMLP
    layer = TPMLP(SimpleNamespace(nranks=1, lib=lib, _h=1), 64, 32, device="cpu")
    for m in (layer.w13, layer.w2):
        m.weight = torch.nn.Parameter(m.weight.detach().as_subclass(OnGpu), requires_grad=False)
    return layer


def test_tangents_are_carried_or_refused_not_dropped(lib):
    import torch.autograd.forward_ad as fwad
    from asystem_amem_b200 import ops
    layer = _mlp(lib)
    with fwad.dual_level(), torch.no_grad():
        h = fwad.make_dual(gpu(4, 32), gpu(4, 32) + 1)
        out = ops.swiglu(h)
        assert fwad.unpack_dual(out).tangent is not None
        assert lib.calls == []
        with pytest.raises(NotImplementedError):
            layer(fwad.make_dual(gpu(16, 64), gpu(16, 64)))
    with torch.no_grad():
        layer(gpu(16, 64))
    assert [name for name, _ in lib.calls][-3:] == ["amemCommBegin", "amemGemmSwiGLU", "amemGemmReduceScatter"]


def test_hooks_of_the_projection_run(lib):
    from torch.nn.modules.module import register_module_forward_hook
    layer, seen = _mlp(lib), []
    with torch.no_grad():
        handle = register_module_forward_hook(lambda m, args, out: seen.append(m))
        try:
            layer(gpu(16, 64))
        finally:
            handle.remove()
        assert layer.w13 in seen and layer.w2 in seen
        handle = layer.w13.register_forward_hook(lambda m, args, out: seen.append("own"))
        layer(gpu(16, 64))
        handle.remove()
    assert seen[-1] == "own" and "amemGemmSwiGLU" not in {name for name, _ in lib.calls}


def test_dispatched_rows_can_be_changed_in_place(lib):
    from asystem_amem_b200.ops.moe import DispatchResult
    from asystem_amem_b200.parallel import ep
    disp = _dispatcher(lib)
    disp.local = lambda *rows: True
    disp.dispatch_local = lambda x, idx: DispatchResult(torch.ones(12, 8, dtype=BF16), None, torch.tensor([0, 4, 7, 9, 10], dtype=torch.int32),
                                                        torch.zeros(6, 2, dtype=torch.int32))
    disp.combine_local = lambda g, idx, w, pos: g[:6] * 1.0
    x = torch.zeros(6, 8, dtype=BF16, requires_grad=True)
    rows, _, _ = ep.ep_dispatch(disp, x, torch.zeros(6, 2, dtype=torch.int32))
    rows.mul_(2)
    assert rows.shape == (10, 8) and torch.all(rows == 2)
    rows.sum().backward()
    assert torch.all(x.grad == 2)


def test_a_paused_communicator_of_one_rank_refuses_the_backward_pass(monkeypatch):
    monkeypatch.setenv("AMEM_BACKEND", "mock")
    from asystem_amem_b200 import Communicator, get_unique_id
    from asystem_amem_b200.bindings import NcclError
    from asystem_amem_b200.parallel import ColumnParallelLinear, RowParallelLinear
    comm = Communicator(1, 0, get_unique_id())
    for kind in (ColumnParallelLinear, RowParallelLinear):
        layer, x = kind(64, 32, comm, device="cpu"), torch.ones(4, 64, dtype=BF16, requires_grad=True)
        out = layer(x).sum()
        comm.pause()
        with pytest.raises(NcclError):
            out.backward(retain_graph=True)
        comm.resume()
        out.backward()
        assert torch.isfinite(x.grad).all()
    comm.destroy()


def test_a_bound_on_a_communicators_blocks_holds_on_one_rank():
    """maxCTAs / AMEM_MAX_BLOCKS: what the single-pass form would need more blocks for goes to the general kernel."""
    import ctypes

    def blocks(count, cap, tin="bfloat16", tout="bfloat16", scale=1.0):
        n = ctypes.c_size_t()
        assert B.load_library().amemLocalPlan(ctypes.c_size_t(count), B.DTYPES[tin], B.DTYPES[tout], ctypes.c_float(scale), cap, ctypes.byref(n)) == 0
        return n.value

    assert blocks(8192 * 100, 0) == 100 and blocks(8192 * 100, 100) == 100      # 16 KB a block
    assert blocks(8192 * 100, 99) == 0 and blocks(1, 1) == 1
    assert blocks(8192 * 10 + 4, 0, tout="float32", scale=0.5) == 11 and blocks(8192 * 10 + 4, 10, tout="float32", scale=0.5) == 0
    assert blocks(8192, 0, tout="float16", scale=0.5) == 0


def test_entry_points_refuse_missing_buffers():
    lib, ok = B.load_library(), 4096       # never dereferenced
    for i in range(3):
        bufs = [ok, ok, ok]
        bufs[i] = None
        assert lib.amemSwiGLU(bufs[0], bufs[1], 16, bufs[2], 2, 8, None) == 4      # ncclInvalidArgument
        assert lib.amemGemmBf16(*bufs, 16, 64, 64, None) == 4
    for i in range(5):
        bufs = [ok] * 5
        bufs[i] = None
        assert lib.amemSwiGLUGrad(bufs[0], bufs[1], 16, *bufs[2:], 2, 8, None) == 4
        assert lib.amemAdamW(*bufs, 8, 1e-3, 0.9, 0.95, 1e-8, 0.0, 1, None) == 4
    assert lib.amemSwiGLU(None, None, 16, None, 0, 8, None) == 0
