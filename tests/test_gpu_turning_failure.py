"""Failure paths of the turning passes, without a GPU fault: the test hook leaves a launch's
pass barrier one arrival short, the bounded wait runs out, every CTA leaves, the call
returns BK_ERR_TIMEOUT, and the same context then runs the same call to the right result."""
import numpy as np
import pytest
import torch

import bk_b200 as bk
from conftest import C64_DH_BAR, C64_DP_BAR
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture
def eng():
    with bk.Engine(0) as e:
        e.set_option("wait_polls", 2000)
        yield e


def _fails(eng, step, call):
    eng.set_option("test_hold_step", step)
    with pytest.raises(bk.BkError) as e:
        call()
    assert e.value.status == bk._lib.BK_ERR_TIMEOUT
    assert "bounded device wait" in str(e.value)
    eng.set_option("test_hold_step", -1)
    eng.set_option("wait_polls", 0)
    return call()


# 2^10-element tiles (read without TMA), 2^12 and 2^13 with two sets, 2^12 with three
@pytest.mark.parametrize("n,precision", [(13, bk.BK_C128), (16, bk.BK_C64), (20, bk.BK_C64), (20, bk.BK_C128),
                                         (23, bk.BK_C64), (24, bk.BK_C128)])
def test_lost_arrival_in_a_run(eng, n, precision):
    bits, e0 = bk.select_trap(n, 5, 100, 0.3)
    p, d, _ = _fails(eng, 1, lambda: eng.evolve(n, bits, 0.35, 0.05, 4, e0=e0, precision=precision))
    po, do, _ = O.trotter_evolve(n, bits, e0, 0.35, 0.05, 4)
    c64 = precision == bk.BK_C64
    assert np.max(np.abs(p - po)) <= (C64_DP_BAR if c64 else 1e-10)
    assert np.max(np.abs(d - do)) <= (C64_DH_BAR if c64 else 1e-10 * n)


@pytest.mark.parametrize("ns", [[16, 14, 20], [20] * 5])
def test_lost_arrival_in_a_batch(eng, ns):
    inst = [dict(n=n, s0=bk.select_trap(n, 30 + i, 40, 0.5)[0], g=0.2 + 0.01 * i) for i, n in enumerate(ns)]
    p, _, _ = _fails(eng, 0, lambda: eng.evolve_batch(inst, 0.04, 5, precision=bk.BK_C64))
    for i, x in enumerate(inst):
        q, _, _ = eng.evolve(x["n"], x["s0"], x["g"], 0.04, 5, precision=bk.BK_C128)
        assert np.max(np.abs(p[i] - q)) <= C64_DP_BAR


@pytest.mark.parametrize("n", [14, 19, 22])
@pytest.mark.parametrize("reverse", [False, True])
def test_lost_arrival_in_a_gradient(eng, n, reverse):
    """In the forward run, and in the reverse sweep's second stretch (its steps follow the
    forward ones)."""
    T, g = 8, np.linspace(0.3, 0.4, 8)
    bits, e0 = bk.select_trap(n, 5, 100, 0.3)
    call = lambda: eng.adjoint(n, bits, g, 0.05, T, e0=e0, precision=bk.BK_C128, checkpoint_every=3)  # noqa: E731
    value, grad, _ = _fails(eng, T + 4 if reverse else 2, call)
    ov, og = O.trotter_adjoint(n, bits, e0, g, 0.05, T)
    assert abs(value - ov) <= 1e-10 and np.max(np.abs(grad - og)) <= 1e-9 * np.max(np.abs(og))


@pytest.mark.parametrize("n", [23, 24])
def test_lost_arrival_in_a_full_space_product(eng, n):
    """The counter's wait gives up while the task's tile copy is on its way: the CTAs wait
    for it before they leave."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(1 << n, generator=gen, device="cuda", dtype=torch.float64)
    y, ref = torch.empty_like(x), torch.empty_like(x)
    _fails(eng, 0, lambda: eng.fullspace_matvec(n, 0.35, x, y))
    eng.fullspace_matvec(n, 0.35, x, ref, method=bk.BK_PLAIN)
    assert float(y.sub_(ref).abs().max()) <= 1e-14 * (n + 1) * float(ref.abs().max())
