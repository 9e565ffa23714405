"""Which one-rank combines gather their rows by bulk copies: those that it was measured to be the faster way for."""
import ctypes

import pytest

from asystem_amem_b200 import bindings as B


def _streams(T, k, d):
    got = ctypes.c_int(-1)
    assert B.load_library().amemMoeCombinePlan(T, k, d, ctypes.byref(got)) == 0
    return bool(got.value)


# rows of 4 to 5.5 KB in numbers, and rows that come to pieces of such a length; few choices, few rows, short rows
@pytest.mark.parametrize("T,k,d", [(16384, 8, 2048), (8192, 8, 2048), (16384, 12, 2048), (16384, 5, 2560), (4096, 12, 2176), (520, 8, 4104), (8192, 5, 4104),
                                   (8192, 8, 4608), (8192, 12, 5120), (4096, 8, 5632), (8192, 8, 8200), (16384, 4, 4096), (500, 8, 4096), (8192, 8, 2040)])
def test_loads_where_they_are_faster(T, k, d):
    assert not _streams(T, k, d)


@pytest.mark.parametrize("T,k,d", [(16384, 8, 4096), (520, 8, 4096), (1024, 5, 4096), (16384, 5, 3072), (16384, 12, 3584), (4096, 6, 6144), (8192, 8, 7168),
                                   (4096, 8, 12288), (4096, 5, 2048), (1024, 12, 2560)])
def test_bulk_copies_where_they_are_faster(T, k, d):
    assert _streams(T, k, d)


# the sizes at which the GPU tests of the bulk copies mean to run them
@pytest.mark.parametrize("T,k,d", [(1400, 5, 2056), (1000, 8, 4096), (700, 16, 2048), (170, 33, 12288), (530, 9, 7000)])
def test_sizes_of_the_kernels_tests(T, k, d):
    assert _streams(T, k, d)


def test_refusals():
    lib, got = B.load_library(), ctypes.c_int()
    assert lib.amemMoeCombinePlan(1, 1, 8, None) == 4 and lib.amemMoeCombinePlan(0, 1, 8, ctypes.byref(got)) == 4
