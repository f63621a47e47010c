"""Device memory of long schedules: partial sums take a bounded room, whatever the number of
measured rows or steps, and a run that is cut into launches for it gives the same rows."""
import numpy as np
import pytest
import torch

import bk_b200 as bk

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _held(call):
    """Device bytes a fresh engine holds after `call`, and its result."""
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with bk.Engine(0) as eng:
        out = call(eng)
        return before - torch.cuda.mem_get_info()[0], out


def test_batch_of_many_measured_rows():
    n, steps, count = 14, 20000, 64
    inst = [dict(n=n, s0=bk.select_trap(n, 30 + i, 40, 0.5)[0], g=0.2 + 0.002 * i) for i in range(count)]

    def call(eng):
        got = eng.evolve_batch(inst, 0.02, steps, precision=bk.BK_C64)
        return got, [eng.evolve(n, x["s0"], x["g"], 0.02, steps, precision=bk.BK_C64) for x in (inst[0], inst[37])]

    held, (got, ones) = _held(call)
    # rows 41 MB, tangents and rescales 20 MB, states 17 MB, the single run's rows and sums
    # 66 MB, 64 MiB of partial sums (all rows at once: 530 MB in sums by CTA, 2 GB by tile)
    assert held <= 320 * MIB
    for i, one in zip((0, 37), ones):
        for a, b in zip(got, one):
            assert np.array_equal(a[i], b)


def test_batch_that_does_not_fit_at_once():
    """States that the free memory does not hold together run in several launches."""
    inst = [dict(n=22, s0=bk.select_trap(22, 30 + i, 40, 0.5)[0], g=0.3 + 0.01 * i) for i in range(40)]
    with bk.Engine(0) as eng:
        want = eng.evolve_batch(inst, 0.04, 3, precision=bk.BK_C128)
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - 3 * 1024 * MIB, dtype=torch.uint8, device="cuda")  # 40 states are 2.7 GB
    try:
        with bk.Engine(0) as eng:
            got = eng.evolve_batch(inst, 0.04, 3, precision=bk.BK_C128)
    finally:
        del held
        torch.cuda.empty_cache()
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_gradient_of_many_steps():
    """One stretch of reverse steps (no checkpoint), cut for the room of its partial sums."""
    n, steps = 18, 60000
    bits, e0 = bk.select_trap(n, 3, 100, 0.3)

    def call(eng):
        return eng.adjoint(n, bits, [0.3], 0.02, steps, e0=e0, precision=bk.BK_C128, checkpoint_every=1 << 30,
                           per_step=True)

    held, (value, _, st) = _held(call)
    # both vectors 8 MB, per-step arrays 2 MB, 64 MiB of partial sums (all passes': 246 MB)
    assert held <= 128 * MIB
    with bk.Engine(0) as eng:
        ref, _, rst = eng.adjoint(n, bits, [0.3], 0.02, steps, e0=e0, precision=bk.BK_C128, checkpoint_every=1000,
                                  per_step=True)
    # the same steps with psi put back from checkpoints: FP64 rounding of 60000 steps of 36
    # rotations, 1.5e-13 an amplitude as a walk, 2e-10 in one direction
    assert value == ref
    assert np.max(np.abs(st["grad_steps"] - rst["grad_steps"])) <= 1e-9 * np.max(np.abs(rst["grad_steps"]))


@pytest.mark.parametrize("n", [18, 22])
def test_cut_sweeps_give_the_same_gradient(n):
    """Checkpoints that cut the sweep in stretches of 1, 3 and 7 steps."""
    T, g = 15, np.linspace(0.3, 0.42, 15)
    bits, e0 = bk.select_trap(n, 13, 100, 0.3)
    with bk.Engine(0) as eng:
        out = [eng.adjoint(n, bits, g, 0.04, T, e0=e0, precision=bk.BK_C128, checkpoint_every=K) for K in (64, 7, 3, 1)]
    for v, grad, _ in out[1:]:
        assert v == out[0][0]
        assert np.max(np.abs(grad - out[0][1])) <= 1e-11 * np.max(np.abs(out[0][1]))


def test_small_run_of_many_measured_rows():
    n, steps, every = 12, 1000000, 1000
    bits, e0 = bk.select_trap(n, 3, 100, 0.3)
    held, got = _held(lambda eng: eng.evolve(n, bits, 0.3, 0.02, steps, e0=e0, precision=bk.BK_C128))
    # rows 32 MB, steps 32 MB, 64 MiB of partial sums (all rows': 192 MB)
    assert held <= 160 * MIB
    with bk.Engine(0) as eng:
        ref = eng.evolve(n, bits, 0.3, 0.02, steps, measure=range(0, steps + 1, every), e0=e0, precision=bk.BK_C128)
    # one run cut in launches, one whole: the same rotations, sums in another order
    for a, b in zip(got, ref):
        assert np.max(np.abs(a[::every] - b)) <= 1e-13 * n
