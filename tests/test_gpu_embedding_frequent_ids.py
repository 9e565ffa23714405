"""Gradient of an embedding where ids are frequent: their rows are shared out between blocks."""
import statistics

import pytest
import torch

pytestmark = pytest.mark.gpu

# around what counts as many (32, 64 and 128 of up to 512, 4096 and more tokens); what one look at the ids and one list of positions hold, and more; tables of less than a slice of
# columns, of slices that do not fill, of many; marks in the first and in later stretches of the tokens
KINDS = {"one": lambda n, rows, g: torch.full((n,), rows - 1, device="cuda"),
         "half": lambda n, rows, g: torch.where(torch.rand(n, device="cuda", generator=g) < 0.5, 0, torch.randint(0, rows, (n,), device="cuda", generator=g)),
         "few": lambda n, rows, g: torch.randint(0, min(rows, max(1, n // 40)), (n,), device="cuda", generator=g),
         "late": lambda n, rows, g: torch.cat([torch.arange(n - n // 3, device="cuda") % rows, torch.randint(0, 3, (n // 3,), device="cuda", generator=g)]),
         "evenly": lambda n, rows, g: torch.arange(n, device="cuda") % max(1, min(rows, n // 33))}


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,rows,d", [(31, 5, 8), (32, 5, 72), (33, 5, 64), (600, 9, 64), (5120, 40, 136), (2047, 300, 264), (2049, 2000, 8), (4500, 50, 2056), (9000, 5000, 128),
                                      (16384, 700, 72), (16384, 20000, 520)])
def test_gradient(kind, n, rows, d):
    from asystem_amem_b200.ops import embedding
    gen = torch.Generator(device="cuda").manual_seed(n)
    ids = KINDS[kind](n, rows, gen)
    table = torch.randn(rows, d, device="cuda", generator=gen).to(torch.bfloat16).requires_grad_(True)
    g = torch.randn(n, d, device="cuda", generator=gen).to(torch.bfloat16)
    embedding(ids, table).backward(g)
    ref, size = (torch.zeros(rows, d, device="cuda", dtype=torch.float64).index_add(0, ids, t.double()) for t in (g, g.abs()))
    # fp32 sums of as many terms as an id has, rounded once
    terms = torch.bincount(ids, minlength=rows).unsqueeze(1)
    assert torch.all((table.grad.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + size * terms * 2.0 ** -24)
    first, table.grad = table.grad, None
    embedding(ids, table).backward(g)
    assert torch.equal(table.grad, first)
    # with work memory of its own
    from asystem_amem_b200 import bindings as B
    out = torch.empty_like(first)
    B.check(B.load_library().amemEmbeddingGrad(g.data_ptr(), ids.data_ptr(), out.data_ptr(), n, d, rows, torch.cuda.current_stream().cuda_stream), "amemEmbeddingGrad")
    assert torch.equal(out, first)


@pytest.mark.parametrize("kind", ["one", "half", "few"])
def test_a_frequent_id_is_no_matter_of_one_block(kind):
    """Half or all of 8192 rows of 8 KB on one id kept one block busy for milliseconds, several times as long as torch's kernel."""
    from asystem_amem_b200.ops.elementwise import _embedding_gradient
    gen = torch.Generator(device="cuda").manual_seed(3)
    ids, g = KINDS[kind](8192, 30000, gen), torch.randn(8192, 4096, device="cuda", generator=gen).to(torch.bfloat16)

    def time(f):
        times = []
        for _ in range(8):
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            f()
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        return statistics.median(times[3:])

    assert time(lambda: _embedding_gradient(g, ids, 30000)) <= 1.5 * time(lambda: torch.ops.aten.embedding_dense_backward(g, ids, 30000, -1, False))
