"""The GEMM for few rows: tile edges, tiles cut along K, groups, SwiGLU, several streams."""
import os

import pytest
import torch

pytestmark = pytest.mark.gpu

# one rounding to bf16 and fp32 sums: see test_gpu_gemm_pair.py
REL = 2.0 ** -8


def _rand(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


def _close(out, ref):
    assert (out.float() - ref).abs().max().item() <= REL * ref.abs().max().item() + 1e-6


@pytest.fixture
def forced():
    os.environ["AMEM_GEMM_SKINNY"] = "1"
    yield
    os.environ.pop("AMEM_GEMM_SKINNY", None)


# the last two: more rows than one tile takes; no workspace (every tile on one SM)
@pytest.mark.parametrize("M,N,K,cut", [(1, 8, 8, True), (16, 128, 64, True), (17, 136, 520, True), (33, 264, 8192, True), (64, 7168, 1000, True),
                                       (127, 1000, 72, True), (300, 264, 1000, True), (20, 520, 4096, False)])
def test_plain(forced, M, N, K, cut):
    from asystem_amem_b200.ops import gemm_bf16
    if not cut:
        os.environ["AMEM_GEMM_SPLITK"] = "0"
    try:
        a, b = _rand((M, K), 1), _rand((N, K), 2)
        outs = [gemm_bf16(a, b) for _ in range(3)]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            outs.append(gemm_bf16(a, b))
        torch.cuda.synchronize()
    finally:
        os.environ.pop("AMEM_GEMM_SPLITK", None)
    _close(outs[0], a.float() @ b.float().t())
    assert all(torch.equal(o, outs[0]) for o in outs)


# long shares of at most half as many tiles as SMs: 56 tiles and their helpers, 37 with a share that just suffices and rows that end
# inside a chunk, 74 with one helper each, two token blocks a weight tile; gate and up halves
@pytest.mark.parametrize("M,N,K", [(16, 7168, 8192), (33, 4720, 8192), (64, 9472, 4160), (200, 2304, 8200)])
def test_tiles_with_owners(forced, M, N, K):
    from asystem_amem_b200.ops import gemm_bf16, gemm_swiglu
    a, b = _rand((M, K), 1), _rand((N, K), 2)
    outs = [gemm_bf16(a, b) for _ in range(6)]
    h = a.float() @ b.float().t()
    _close(outs[0], h)
    assert all(torch.equal(o, outs[0]) for o in outs)
    h = a.float() @ (b * 0.01).float().t()
    _close(gemm_swiglu(a, b * 0.01), torch.nn.functional.silu(h[:, :N // 2]) * h[:, N // 2:])


@pytest.mark.parametrize("counts", [(3, 0, 17, 40), (0, 0, 5), (9, 7, 8, 8), (200, 1, 0, 130), (0, 0)])
@pytest.mark.parametrize("ffn,K", [(32, 64), (96, 520), (512, 4096)])
def test_groups(forced, counts, ffn, K):
    from asystem_amem_b200.ops import grouped_gemm_bf16, interleave_gate_up
    E, rows, N = len(counts), sum(counts), 2 * ffn
    offs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    a, w = _rand((rows + 5, K), 3), _rand((E, N, K), 4, 0.1)
    out, act = torch.full((rows + 5, N), 7.0, device="cuda", dtype=torch.bfloat16), torch.full((rows + 5, ffn), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm_bf16(a, w, offs, out=out, rows_hint=rows)
    grouped_gemm_bf16(a, interleave_gate_up(w, ffn), offs, out=act, rows_hint=rows, swiglu=True)
    assert torch.all(out[rows:] == 7.0) and torch.all(act[rows:] == 7.0)
    lo = 0
    for e, c in enumerate(counts):
        if c:
            h = a[lo:lo + c].float() @ w[e].float().t()
            _close(out[lo:lo + c], h)
            _close(act[lo:lo + c], torch.nn.functional.silu(h[:, :ffn]) * h[:, ffn:])
        lo += c


def test_under_capture_and_back_to_back():
    """Launches overlap their predecessor's end; each still reads what that one wrote."""
    from asystem_amem_b200.ops import gemm_bf16
    w = [_rand((512, 512), 10 + i, 0.05) for i in range(4)]
    x = _rand((16, 512), 9)

    def chain(t):
        for i in range(12):
            t = gemm_bf16(t, w[i % 4])
        return t

    ref = x
    for i in range(12):
        ref = gemm_bf16(ref, w[i % 4])
        torch.cuda.synchronize()
    assert torch.equal(chain(x), ref)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        chain(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        out = chain(x)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, ref)


def test_only_a_product_that_is_cut_makes_a_workspace():
    """Grouped products and those of whole tiles allocate nothing on a stream that they are the first to use."""
    from asystem_amem_b200 import mem_stats
    from asystem_amem_b200.ops import gemm_bf16, gemm_swiglu, grouped_gemm_bf16
    x, w, offs = _rand((64, 256), 9), _rand((4, 128, 256), 10), torch.tensor([0, 3, 9, 40, 64], dtype=torch.int32, device="cuda")
    big, wide = _rand((4096, 512), 11), _rand((4096, 512), 12)
    gemm_bf16(x, w[0])          # the process's own words
    torch.cuda.synchronize()
    live = mem_stats()["live_bytes"]
    side = torch.cuda.Stream(priority=-1)       # of a pool that no other test draws from
    with torch.cuda.stream(side):
        grouped_gemm_bf16(x, w, offs, rows_hint=64)
        gemm_bf16(x, w[0])
        gemm_swiglu(x, w[0])
        gemm_bf16(big, wide)
        side.synchronize()
        assert mem_stats()["live_bytes"] == live
        gemm_bf16(_rand((16, 8192), 13), _rand((7168, 8192), 14))      # 56 tiles on 148 SMs: cut
        side.synchronize()
        assert mem_stats()["live_bytes"] > live


# sizes that run with owners: 74 tiles with one helper each, two token blocks a weight tile and a ragged last block in the owner's share
# (tests/test_cpu_gemm_schedules.py asks which way they go)
@pytest.mark.parametrize("M,N,K", [(64, 9472, 9216), (200, 2304, 8456)])
def test_owners_at_their_limits(forced, M, N, K):
    test_tiles_with_owners(None, M, N, K)


# more rows than one tile takes, cut evenly
@pytest.mark.parametrize("M,N,K", [(300, 264, 2008)])
def test_even_cuts_of_several_token_blocks(forced, M, N, K):
    test_plain(None, M, N, K, True)
