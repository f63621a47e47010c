"""Descents of more starts than one kernel takes: exact integers on both sides of the pieces'
ends, in the caller's own arrays too, and a bounded device room."""
import ctypes

import numpy as np
import pytest
import torch

import bk_b200 as bk

pytestmark = pytest.mark.gpu

PIECE = 1 << 17


@pytest.mark.parametrize("n,count", [(20, PIECE - 1), (20, PIECE), (20, PIECE + 1), (28, 3 * PIECE + 5), (40, PIECE + 7)])
def test_pieces_equal_the_host_form(n, count):
    starts = bk.random_states(n, count, count)
    with bk.Engine(0) as eng:
        for a, b in zip(eng.steepest_descent(n, starts), bk.steepest_descent(n, starts)):
            assert np.array_equal(a, b)


def test_final_states_may_replace_the_starts():
    n, count = 24, 2 * PIECE + 3
    starts = bk.random_states(n, 5, count)
    want = bk.steepest_descent(n, starts)
    u64p = ctypes.POINTER(ctypes.c_uint64)
    x, e = starts.copy(), np.zeros(count, dtype=np.int64)
    with bk.Engine(0) as eng:
        p = x.ctypes.data_as(u64p)
        assert eng.L.bk_steepest_descent_gpu(eng.ctx, n, p, count, 0, p, e.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)),
                                             None) == 0
    assert np.array_equal(x, want[0]) and np.array_equal(e, want[1])


def test_device_room_is_a_pieces():
    torch.cuda.synchronize()
    with bk.Engine(0) as eng:
        before = torch.cuda.mem_get_info()[0]
        eng.steepest_descent(20, bk.random_states(20, 1, 2_000_000))
        assert before - torch.cuda.mem_get_info()[0] <= 16 << 20  # a piece is 2 MB, the whole batch 32
