"""Batches in the default mode (turning passes): each member reproduces its own single run
bit for bit, in both precisions, whatever shares the launch with it (several members of a
size, so that the groups of CTAs differ from a single run's; complex64 members up to 18
qubits, which compute in complex128 as single runs do; members too large for a group), and
follows its own schedule (per-step ramps, another for every member)."""
import numpy as np
import pytest

import bk_b200 as bk
from conftest import C64_DH_BAR, C64_DP_BAR
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = bk.Engine(0)
    yield e
    e.close()


def _instances(ns, seed, steps):
    rng = np.random.default_rng(seed)
    out = []
    for j, n in enumerate(ns):
        bits, e0 = bk.select_trap(n, seed + j, 40, 0.5)
        out.append(dict(n=n, s0=bits, e0=e0, g=rng.uniform(0.2, 0.5, steps) if j % 3 else float(rng.uniform(0.2, 0.5))))
    return out


@pytest.mark.parametrize("precision,ns", [
    (bk.BK_C64, [16, 14, 18, 20, 16, 22, 15, 19, 17, 20, 21, 21, 22, 23, 24, 18]),
    (bk.BK_C64, [17] * 33), (bk.BK_C64, [20] * 9), (bk.BK_C64, [25, 16, 24, 20, 26]),
    (bk.BK_C128, [13, 16, 18, 20, 14, 21, 18, 19, 19, 22, 23, 22, 20]),
    (bk.BK_C128, [15] * 40), (bk.BK_C128, [24, 16, 25, 21])])
def test_members_are_their_single_runs(eng, precision, ns):
    steps, meas = 9, [0, 1, 5, 9]
    inst = _instances(ns, 31, steps)
    got = eng.evolve_batch(inst, 0.04, steps, measure=meas, precision=precision)
    for i, x in enumerate(inst):
        one = eng.evolve(x["n"], x["s0"], x["g"], 0.04, steps, measure=meas, e0=x["e0"], precision=precision)
        for a, b in zip(got, one):
            assert np.array_equal(a[i], b), (i, x["n"], np.max(np.abs(a[i] - b)))


@pytest.mark.parametrize("precision,ns", [(bk.BK_C128, [13, 15, 17, 17, 19]), (bk.BK_C64, [16, 18, 14, 19, 20, 20])])
def test_schedules_match_the_oracle(eng, precision, ns):
    steps, dt = 24, 0.02
    inst = _instances(ns, 3, steps)
    p, d, nn = eng.evolve_batch(inst, dt, steps, precision=precision)
    for i, x in enumerate(inst):
        po, do, _ = O.trotter_evolve(x["n"], x["s0"], x["e0"], x["g"], dt, steps)
        c64 = precision == bk.BK_C64
        assert np.max(np.abs(p[i] - po)) <= (C64_DP_BAR if c64 else 1e-10)
        assert np.max(np.abs(d[i] - do)) <= (C64_DH_BAR if c64 else 1e-10 * x["n"])
        assert np.max(np.abs(nn[i] - 1.0)) <= (1e-5 if c64 else 1e-10)


def test_a_batch_leaves_the_last_run_alone(eng):
    """Export and sampling after a batch are still those of the last bk_evolve."""
    bits, _ = bk.select_trap(16, 4, 100, 0.3)
    eng.evolve(16, bits, 0.35, 0.05, 5, precision=bk.BK_C64)
    before = eng.export_state(16)
    eng.evolve_batch(_instances([14, 25, 20], 5, 3), 0.04, 3, precision=bk.BK_C64)
    assert np.array_equal(before, eng.export_state(16))
