"""The gradient's value is that of the run bk_evolve makes of the same schedule, in the default
mode: complex64 schedules up to 18 qubits compute in complex128 in both (they differed by
FP32 rounding, and TrotterObjective's value changed with requires_grad), and both refuse the
phase angles that the complex64 level table does not hold."""
import numpy as np
import pytest

import bk_b200 as bk
from bk_b200.adjoint import TrotterSchedule

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = bk.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("n", [14, 16, 18])
@pytest.mark.parametrize("objective", [bk.BK_OBJ_P_LESS, bk.BK_OBJ_D_H])
def test_value_does_not_depend_on_requires_grad(eng, n, objective):
    bits, e0 = bk.select_trap(n, 11, 100, 0.3)
    sched = TrotterSchedule(eng, n, bits, [0.31, 0.36, 0.42], 0.05, 24, precision=bk.BK_C64, objective=objective,
                            checkpoint_every=7, e0=e0)
    with_grad = float(sched().detach())
    sched.g.requires_grad_(False)
    without = float(sched())
    # the plain run divides by its norm, 1 to the rounding of 24 complex128 steps
    assert abs(with_grad - without) <= 1e-12 * max(1.0, abs(without))


@pytest.mark.parametrize("n", [14, 18])
def test_single_precision_request_is_the_double_gradient(eng, n):
    bits, e0 = bk.select_trap(n, 12, 100, 0.3)
    g = np.linspace(0.3, 0.4, 12)
    a = eng.adjoint(n, bits, g, 0.05, 12, e0=e0, precision=bk.BK_C64, checkpoint_every=5)
    b = eng.adjoint(n, bits, g, 0.05, 12, e0=e0, precision=bk.BK_C128, checkpoint_every=5)
    assert a[0] == b[0] and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("n,checkpoint_every", [(16, 64), (20, 64), (20, 2)])
def test_angles_beyond_the_level_table_are_refused(eng, n, checkpoint_every):
    bits, e0 = bk.select_trap(n, 12, 100, 0.3)
    for call in (lambda: eng.evolve(n, bits, 0.3, 0.05, 4, e0=e0, precision=bk.BK_C64, diag_scale=4.0),
                 lambda: eng.adjoint(n, bits, [0.3], 0.05, 4, e0=e0, precision=bk.BK_C64, diag_scale=4.0,
                                     checkpoint_every=checkpoint_every)):
        with pytest.raises(bk.BkError) as e:
            call()
        assert e.value.status == bk._lib.BK_ERR_UNSUPPORTED
