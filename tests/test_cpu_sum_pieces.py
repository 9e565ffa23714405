"""The sum of gradients into a shard: what its launches are, and what its entry points refuse.  Host arithmetic."""
import ctypes

import pytest

from asystem_amem_b200 import bindings as B


def _most_blocks(sizes, cap):
    n = ctypes.c_size_t()
    assert B.load_library().amemSumPiecesPlan((ctypes.c_longlong * len(sizes))(*sizes), len(sizes), cap, ctypes.byref(n)) == 0
    return n.value


def test_a_bound_on_a_communicators_blocks_holds():
    assert _most_blocks([4096 * 100], 0) == 100 and _most_blocks([4096 * 100], 100) == 100     # 4096 elements a block
    assert _most_blocks([4096 * 100], 99) == 99 and _most_blocks([4096 * 100], 3) == 3
    assert _most_blocks([1, 4097, 0, 4096], 0) == 1 + 2 + 1 and _most_blocks([1, 4097, 0, 4096], 2) == 2
    assert _most_blocks([5] * 33 + [0, 0], 0) == 32 and _most_blocks([], 0) == 0 and _most_blocks([0], 4) == 0


def test_what_a_communicator_refuses_is_refused(monkeypatch):
    monkeypatch.setenv("AMEM_BACKEND", "mock")
    from asystem_amem_b200 import Communicator, get_unique_id
    lib, comm = B.load_library(), Communicator(1, 0, get_unique_id())
    none = ((ctypes.c_void_p * 0)(), (ctypes.c_void_p * 0)(), (ctypes.c_longlong * 0)(), 0, 1.0)
    assert lib.amemSumPiecesLocal(*none, comm._h, None) == 0
    comm.pause()
    assert lib.amemSumPiecesLocal(*none, comm._h, None) != 0
    comm.resume()
    assert lib.amemSumPiecesLocal(*none, comm._h, None) == 0 and lib.amemSumPiecesLocal(*none, None, None) == 4
    odd = ((ctypes.c_void_p * 1)(4097), (ctypes.c_void_p * 1)(4096), (ctypes.c_longlong * 1)(8), 1, 1.0)     # never dereferenced
    assert lib.amemSumPiecesLocal(*odd, comm._h, None) == 4 and lib.amemSumPieces(*odd, None) == 4
    comm.destroy()
