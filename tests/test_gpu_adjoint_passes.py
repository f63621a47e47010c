"""The gradient's reverse sweep with a launch per pass (engine mode 1): the 12-bit and the
warp-local A1, with the complex64 level table and with the full phase table (D^dagger as the
negated half-angle shear rotations of each level's entry), against the oracle within the
complex64 gradient's bars. In the default mode these schedules run in turning passes."""
import numpy as np
import pytest

import bk_b200 as bk
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,adj_a1", [(16, 0), (18, 0), (22, 0), (23, 0), (22, 1)])
@pytest.mark.parametrize("phase_table", [0, 1])
def test_launch_per_pass_gradient_matches_the_oracle(n, adj_a1, phase_table):
    T, K = (24, 8) if n >= 22 else (40, 16)
    bits, e0 = bk.select_trap(n, n, 200, 0.05)
    gs, seg = np.random.default_rng(n).uniform(0.25, 0.45, 4), O.segment_steps(T, 4)
    with bk.Engine(0) as eng:
        eng.set_option("engine_mode", 1)
        eng.set_option("phase_table", phase_table)
        eng.set_option("adj_a1", adj_a1)
        eng.set_kernel_timing(True)
        val, grad, st = eng.adjoint(n, bits, gs, 0.05, T, e0=e0, precision=bk.BK_C64, checkpoint_every=K, per_step=True)
        assert not any(name.startswith("adj_turn") for name in eng.kernel_timing())
    oval, ograd = O.trotter_adjoint(n, bits, e0, gs[seg], 0.05, T)
    scale = np.max(np.abs(ograd))
    assert abs(val - oval) <= 1e-6
    assert np.max(np.abs(st["grad_steps"] - ograd)) <= 1e-4 * scale
    assert st["max_drift"] <= 1e-4
