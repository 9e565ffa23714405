"""The GEMM on SM pairs: operand layouts, ragged tiles, groups, cuts along K."""
import os

import pytest
import torch

pytestmark = pytest.mark.gpu

# One rounding of the fp32 sum to bf16 (8 significant bits) is at most 2^-8 of the value, less where the
# value is not just above a power of two; the sum's own error (K <= 8192 terms in fp32, any order) is far
# below: 2^-8 of the largest result covers both.
REL = 2.0 ** -8


def _rand(shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


def _close(out, ref):
    assert (out.float() - ref).abs().max().item() <= REL * ref.abs().max().item() + 1e-6


@pytest.fixture
def on_pairs():
    os.environ["AMEM_GEMM_PAIR"] = "1"
    yield
    os.environ.pop("AMEM_GEMM_PAIR", None)


@pytest.fixture
def groups_on_pairs():
    """(Few rows a group would go to the kernel for few rows otherwise.)"""
    os.environ["AMEM_GEMM_SKINNY"] = "0"
    yield
    os.environ.pop("AMEM_GEMM_SKINNY", None)


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (128, 128, 64), (129, 136, 72), (255, 264, 328), (257, 1000, 2056), (520, 776, 4096), (300, 256, 8192),
                                   (2200, 2568, 512)])
def test_products_of_a_linear_and_its_gradients(on_pairs, M, N, K):
    from asystem_amem_b200.ops import gemm_bf16, gemm_input_grad, gemm_weight_grad
    x, w, gy = _rand((M, K), 1), _rand((N, K), 2), _rand((M, N), 3)
    for _ in range(2):      # twice: the counters of a cut product are back at zero
        _close(gemm_bf16(x, w), x.float() @ w.float().t())
        _close(gemm_input_grad(gy, w), gy.float() @ w.float())
        _close(gemm_weight_grad(gy, x), gy.float().t() @ x.float())


@pytest.mark.parametrize("T", [1, 15, 16, 17, 63, 64, 65, 1001])
def test_weight_gradient_of_any_number_of_rows(on_pairs, T):
    from asystem_amem_b200.ops import gemm_weight_grad
    gy, x = _rand((T, 264), 4), _rand((T, 136), 5)
    _close(gemm_weight_grad(gy, x), gy.float().t() @ x.float())


@pytest.mark.parametrize("counts", [(1, 0, 63, 64, 65, 300), (0, 0, 5), (256, 256), (17,), (0, 1000, 31)])
@pytest.mark.parametrize("N,K", [(192, 128), (264, 72)])
def test_groups(groups_on_pairs, counts, N, K):
    from asystem_amem_b200.ops import grouped_gemm_bf16, grouped_gemm_input_grad, grouped_gemm_weight_grad
    E, rows, pad = len(counts), sum(counts), 9
    offs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    a, g, w = _rand((rows + pad, K), 6), _rand((rows + pad, N), 7), _rand((E, N, K), 8)
    out, gin = torch.full((rows + pad, N), 7.0, device="cuda", dtype=torch.bfloat16), torch.full((rows + pad, K), 7.0, device="cuda", dtype=torch.bfloat16)
    grouped_gemm_bf16(a, w, offs, out=out)
    grouped_gemm_input_grad(g, w, offs, out=gin)
    gw = grouped_gemm_weight_grad(g, a, offs)
    assert torch.all(out[rows:] == 7.0) and torch.all(gin[rows:] == 7.0)     # rows of no group stay as they are
    lo = 0
    for e, c in enumerate(counts):
        sl = slice(lo, lo + c)
        lo += c
        if c:
            _close(out[sl], a[sl].float() @ w[e].float().t())
            _close(gin[sl], g[sl].float() @ w[e].float())
            _close(gw[e], g[sl].float().t() @ a[sl].float())
        else:
            assert torch.all(gw[e] == 0)


def test_a_group_does_not_see_its_neighbours_values(groups_on_pairs):
    """Infinities and NaN in the rows and matrices next to a group's own stay out of its results."""
    from asystem_amem_b200.ops import grouped_gemm_bf16, grouped_gemm_input_grad, grouped_gemm_weight_grad
    counts, N, K = (37, 50, 41), 200, 72
    offs = torch.tensor([0, 37, 87, 128], dtype=torch.int32, device="cuda")
    a, g, w = _rand((128, K), 9), _rand((128, N), 10), _rand((3, N, K), 11)
    ref = [t.clone() for t in (grouped_gemm_bf16(a, w, offs), grouped_gemm_input_grad(g, w, offs), grouped_gemm_weight_grad(g, a, offs))]
    for bad in (0, 2):
        sl = slice(int(offs[bad]), int(offs[bad + 1]))
        a[sl], g[sl], w[bad] = float("nan"), float("inf"), float("nan")
    mine = slice(37, 87)
    assert torch.equal(grouped_gemm_bf16(a, w, offs)[mine], ref[0][mine])
    assert torch.equal(grouped_gemm_input_grad(g, w, offs)[mine], ref[1][mine])
    assert torch.equal(grouped_gemm_weight_grad(g, a, offs)[1], ref[2][1])


@pytest.mark.parametrize("ffn", [32, 96, 160, 1024])
def test_swiglu_epilogue(groups_on_pairs, ffn):
    from asystem_amem_b200.ops import grouped_gemm_bf16, interleave_gate_up
    offs = torch.tensor([0, 130, 130, 400], dtype=torch.int32, device="cuda")
    a, w = _rand((400, 256), 12), _rand((3, 2 * ffn, 256), 13, 0.1)
    out = grouped_gemm_bf16(a, interleave_gate_up(w, ffn), offs, swiglu=True)
    for e in range(3):
        sl = slice(int(offs[e]), int(offs[e + 1]))
        if sl.stop > sl.start:
            h = a[sl].float() @ w[e].float().t()
            _close(out[sl], torch.nn.functional.silu(h[:, :ffn]) * h[:, ffn:])


def test_seven_cuts_of_a_wide_tile(on_pairs):
    """Ten tiles of 256 x 256 on 74 pairs are cut in seven: the first slice collects two chunks from each of
    the others, the most that the idle operand ring ever holds."""
    from asystem_amem_b200.ops import gemm_bf16
    x, w = _rand((2560, 8192), 14), _rand((256, 8192), 15)
    for _ in range(2):
        _close(gemm_bf16(x, w), x.float() @ w.float().t())
