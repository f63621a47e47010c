"""A complex64 step turns by a rounded tangent; what it misses is made up for in the next
step, as an angle: half an ulp of a large tangent t is 1 + t^2 times as much as the angle it
stands for. A step of large tangent is followed by a small one, for which the full tangent
residue would be 60 times the complex64 resolution; single runs (turning and tile passes),
batches and the gradient's forward run share the schedule.

The diagonal phase is all but off, so the state is a product of n equal qubits turned by
a = theta_1 + theta_2, and <d_H> = n sin^2 a has the slope n sin 2a = -9 to an error of a.
Its bar: the second tangent's own rounding (1.5e-8 rad: 1.4e-7) and FP32 rounding of the
rotations, n x 2 x 6e-8 x p (1 - p) = 5e-7 if all of it had one sign; 1.5e-6 allows twice
that. A residue taken for an angle (9e-7 rad) makes 8e-6."""
import math

import numpy as np
import pytest

import bk_b200 as bk

pytestmark = pytest.mark.gpu

N, DT, SCALE, BAR = 19, 0.05, 1e-9, 1.5e-6


def _angles():
    # the tangent in [16, 24) whose FP32 rounding is farthest off
    t = max(np.linspace(16.0, 24.0, 4001), key=lambda x: abs(float(np.float32(x)) - float(x)))
    assert abs(float(np.float32(t)) - t) > 9e-7
    return np.array([math.atan(t), 0.3])


@pytest.fixture(scope="module")
def eng():
    e = bk.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("mode", [1, 4])
def test_small_step_after_a_large_tangent(eng, mode):
    a = _angles()
    eng.set_option("engine_mode", mode)
    _, d, _ = eng.evolve(N, 0b1011, a / DT, DT, 2, measure=[2], e0=100, precision=bk.BK_C64, diag_scale=SCALE)
    assert abs(d[0] - N * math.sin(a.sum()) ** 2) <= BAR


def test_in_a_batch(eng):
    a = _angles()
    eng.set_option("engine_mode", 4)
    inst = [dict(n=N, s0=0b1011 + i, e0=100, g=a / DT) for i in range(3)]
    _, d, _ = eng.evolve_batch(inst, DT, 2, measure=[2], precision=bk.BK_C64, diag_scale=SCALE)
    assert np.max(np.abs(d[:, 0] - N * math.sin(a.sum()) ** 2)) <= BAR


def test_in_a_gradient(eng):
    a = _angles()
    eng.set_option("engine_mode", 4)
    v, _, st = eng.adjoint(N, 0b1011, a / DT, DT, 2, e0=100, precision=bk.BK_C64, objective=bk.BK_OBJ_D_H,
                           diag_scale=SCALE)
    assert abs(v / st["norm"] - N * math.sin(a.sum()) ** 2) <= BAR
