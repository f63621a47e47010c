"""The device descent against the host form: exact integers for every chain length
(one and two bytes-of-correlations halves, each lane's first and last spin) and for
budgets that stop in the middle of a descent."""
import numpy as np
import pytest

import bk_b200 as bk

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = bk.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("n", [2, 3, 4, 5, 31, 32, 33, 34, 62, 63])
def test_descent_equals_the_host_form(eng, n):
    starts = np.concatenate([bk.random_states(n, 40 + n, 400),
                             np.array([0, (1 << n) - 1, 0x5555555555555555 & ((1 << n) - 1)], dtype=np.uint64)])
    for budget in (0, 1, n, n + 1, 3 * n + 1, 4 * n):
        dev, host = eng.steepest_descent(n, starts, budget), bk.steepest_descent(n, starts, budget)
        for a, b in zip(dev, host):
            assert np.array_equal(a, b)


def test_large_and_small_counts(eng):
    for count in (1, 7, 40000):
        starts = bk.random_states(20, 3, count)
        for a, b in zip(eng.steepest_descent(20, starts), bk.steepest_descent(20, starts)):
            assert np.array_equal(a, b)
