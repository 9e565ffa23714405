"""Which routings go to the kernel: only those that it was measured to be the faster way for."""
import pytest

from asystem_amem_b200.ops.moe import _route_pays


# tokens, width, experts
@pytest.mark.parametrize("T,d,E", [(8192, 4096, 72), (16384, 4096, 80), (8192, 4096, 96), (8192, 4096, 128), (16384, 3072, 96), (8192, 3072, 128),
                                   (1, 4096, 256), (32, 4096, 256), (256, 4096, 256), (4096, 4096, 256), (16384, 4096, 256), (1, 16384, 64), (8192, 16384, 64)])
def test_a_library_product_where_it_is_faster(T, d, E):
    assert not _route_pays(T, d, E)


@pytest.mark.parametrize("T", [1, 32, 1024, 4096, 8192, 16384])
@pytest.mark.parametrize("d,E", [(1024, 8), (4096, 8), (4096, 16), (4096, 64), (8192, 32), (8192, 64), (16384, 32), (1024, 256), (2048, 96), (2048, 128), (2048, 192)])
def test_the_kernel_where_it_is_faster(T, d, E):
    assert _route_pays(T, d, E)


@pytest.mark.parametrize("E", [72, 96, 128])
def test_the_kernel_for_few_tokens_of_many_experts(E):
    assert _route_pays(1, 4096, E) and _route_pays(4096, 4096, E)
