"""How the GEMM for few rows shares out its blocks of K: the listed sizes, and those at which the GPU tests mean to run each way."""
import ctypes

import pytest

from asystem_amem_b200 import bindings as B

WHOLE, EVEN, OWNERS = 0, 1, 2


def schedule(M, N, K):
    how = ctypes.c_int(7)
    assert B.load_library().amemGemmSchedule(M, N, K, 148, ctypes.byref(how)) == 0
    return how.value


@pytest.mark.parametrize("M,N,K,how", [(16, 7168, 8192, OWNERS), (16, 3584, 8192, EVEN), (4, 1024, 8192, EVEN), (16, 8192, 3584, WHOLE), (16, 18944, 3584, WHOLE),
                                       (64, 9472, 4160, WHOLE), (1000, 3584, 8192, -1)])
def test_of_a_product(M, N, K, how):
    assert schedule(M, N, K) == how


# 56 tiles, 37 with rows that end inside a chunk, 74 with one helper each, two token blocks a weight tile with a ragged last block of K
@pytest.mark.parametrize("M,N,K", [(16, 7168, 8192), (33, 4720, 8192), (64, 9472, 9216), (200, 2304, 8456)])
def test_of_the_tests_of_owners(monkeypatch, M, N, K):
    monkeypatch.setenv("AMEM_GEMM_SKINNY", "1")
    assert schedule(M, N, K) == OWNERS


@pytest.mark.parametrize("M,N,K", [(300, 264, 2008), (33, 264, 8192)])
def test_of_the_tests_of_even_cuts(monkeypatch, M, N, K):
    monkeypatch.setenv("AMEM_GEMM_SKINNY", "1")
    assert schedule(M, N, K) == EVEN
    monkeypatch.setenv("AMEM_GEMM_SPLITK", "0")
    assert schedule(M, N, K) == WHOLE


# where cutting was measured to be the faster way, and where whole tiles were
@pytest.mark.parametrize("M,N,K", [(1, 512, 1536), (1, 2560, 2048), (16, 3584, 1536), (16, 4608, 2048), (24, 3072, 2048), (32, 4096, 2048), (16, 7168, 3584), (48, 2048, 2048)])
def test_cuts_that_pay(M, N, K):
    assert schedule(M, N, K) > 0


@pytest.mark.parametrize("M,N,K", [(16, 5120, 2048), (16, 8192, 3584), (32, 5120, 2560), (64, 4096, 2560), (64, 7168, 4096), (48, 5120, 3072), (64, 512, 1024)])
def test_cuts_that_do_not(M, N, K):
    assert schedule(M, N, K) == 0
