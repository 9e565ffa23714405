"""Which of the decoder's passes go to the kernels: those that they were measured to be the faster way for."""
import pytest

from asystem_amem_b200.ops import elementwise as EW


@pytest.mark.parametrize("rows,dim,gradients,kernel", [(65536, 8, False, False), (65536, 8, True, False), (65536, 64, False, False), (65536, 64, True, True),
                                                       (1_000_000, 72, False, False), (1_000_000, 96, False, True), (65536, 128, False, True), (4096, 64, False, True), (8192, 8, True, True),
                                                       (1, 8, False, True), (32768, 4096, True, True)])
def test_norm(rows, dim, gradients, kernel):
    assert EW._norm_pays(rows, dim, gradients) == kernel


def test_gated_rows_are_one():
    """Many short rows: most of a block's threads would have no vector."""
    import torch
    assert EW._as_rows(torch.empty(65536, 64, device="meta")) == (1, 65536 * 64) and EW._as_rows(torch.empty(2, 3, 8, device="meta")) == (1, 48)
    assert EW._as_rows(torch.empty(2 ** 22, 1024, device="meta")) == (2 ** 22, 1024)


@pytest.mark.parametrize("tokens,elements,kernel", [(65536, 16, False), (65536, 8, False), (65536, 128, True), (1, 8, True), (8192, 5120, True)])
def test_rotary_embedding(tokens, elements, kernel):
    assert EW._turn_pays(tokens, elements) == kernel
