"""Turning passes (the default schedule) at the edges of their dispatch: every tile
size and set width against the tile-pass schedule (BK_OPT_ENGINE_MODE 1) in
complex128, runs split at sampling points, and batches against single runs.

Bars. complex128: the same rotations in another order, at most 32 qubits x 10 steps
of rounding on amplitudes of norm 1: 1e-13 absolute on P_< and the norm, n times
that on <d_H>. complex64: the engine's own bars (conftest)."""
import numpy as np
import pytest
import torch

import bk_b200 as bk
from tests.conftest import C64_DH_BAR, C64_DP_BAR

pytestmark = pytest.mark.gpu

BAR128 = 1e-13


@pytest.fixture(scope="module")
def eng():
    e = bk.Engine(0)
    yield e
    e.close()


def _both(eng, n, precision, steps, **kw):
    bits, e0 = bk.select_trap(n, 21, 100, 0.3)
    g = np.linspace(0.3, 0.45, steps)
    out = []
    for mode in (1, 4):
        eng.set_option("engine_mode", mode)
        out.append(eng.evolve(n, bits, g, 0.05, steps, e0=e0, precision=precision, **kw))
    return out


# element bits: 13 / 18 (first and last of the 2^10 tiles), 14, 15 (a set of 4 and of 5
# bits: turn in the first and in the second round), 19, 20, 21, 23 and the three-set
# sizes from 24 on, up to the widest sets (30: 9 + 9 bits)
@pytest.mark.parametrize("n", [13, 14, 15, 16, 17, 18, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29, 30])
@pytest.mark.parametrize("steps", [1, 6])
def test_sizes_match_the_tile_passes_c128(eng, n, steps):
    a, b = _both(eng, n, bk.BK_C128, steps)
    assert np.max(np.abs(a[0] - b[0])) <= BAR128
    assert np.max(np.abs(a[1] - b[1])) <= BAR128 * n
    assert np.max(np.abs(a[2] - b[2])) <= BAR128


@pytest.mark.parametrize("n", [14, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28, 29, 30])
def test_sizes_match_the_tile_passes_c64(eng, n):
    a, b = _both(eng, n, bk.BK_C64, 7, measure=[0, 3, 7])
    assert np.max(np.abs(a[0] - b[0])) <= C64_DP_BAR
    assert np.max(np.abs(a[1] - b[1])) <= C64_DH_BAR


def test_no_steps_measures_the_trap(eng):
    eng.set_option("engine_mode", 4)
    bits, e0 = bk.select_trap(16, 3, 100, 0.3)
    p, d, nn = eng.evolve(16, bits, 0.35, 0.05, 0, e0=e0, precision=bk.BK_C128)
    assert (p[0], d[0], nn[0]) == (0.0, 0.0, 1.0)


@pytest.mark.parametrize("n,precision", [(14, bk.BK_C128), (20, bk.BK_C64)])
def test_sampling_points_do_not_change_the_series(eng, n, precision):
    """A run split into launches at its sampling points has the same passes."""
    eng.set_option("engine_mode", 4)
    bits, _ = bk.select_trap(n, 4, 100, 0.3)
    kw = dict(n=n, g=0.35, dt=0.05, t_max=1.0, verbose=False, num_sampling_seeds=1)
    a = eng.sampler_run(bits, precision=precision, shots_per_point=0, num_sample_points=21, dt_sample=0.05, **kw)
    b = eng.sampler_run(bits, precision=precision, shots_per_point=16, num_sample_points=4, record_trajectory=True,
                        dt_trajectory=0.05, **kw)
    assert np.array_equal(a["p_less_history"], b["p_less_history"])
    assert np.array_equal(a["dh_history"], b["dh_history"])


@pytest.mark.parametrize("precision,ns", [(bk.BK_C64, [14, 19, 20, 21, 22, 24, 16, 16]), (bk.BK_C128, [13, 18, 19, 21, 22, 13]),
                                          (bk.BK_C64, [17] * 33)])
def test_batch_matches_single_runs(eng, precision, ns):
    """Groups of CTAs, one statevector each in turn: complex128, and complex64 from 19
    qubits on, have the single runs' states (sums over other CTA shares, so FP64 rounding
    apart); smaller complex64 single runs compute in complex128."""
    eng.set_option("engine_mode", 4)
    inst = [dict(n=n, s0=bk.select_trap(n, 30 + i, 40, 0.5)[0], g=0.2 + 0.01 * i) for i, n in enumerate(ns)]
    steps, meas = 9, [0, 1, 5, 9]
    p, d, nn = eng.evolve_batch(inst, 0.04, steps, measure=meas, precision=precision)
    for i, x in enumerate(inst):
        q, e, m = eng.evolve(x["n"], x["s0"], x["g"], 0.04, steps, measure=meas, precision=precision)
        same = precision == bk.BK_C128 or x["n"] >= 19
        assert np.max(np.abs(p[i] - q)) <= (BAR128 if same else C64_DP_BAR)
        assert np.max(np.abs(d[i] - e)) <= (BAR128 * x["n"] if same else C64_DH_BAR)
        assert np.max(np.abs(nn[i] - m)) <= (BAR128 if same else 1e-5)


def test_wait_limit_is_an_error_not_a_hang(eng):
    """The smallest poll limit of the barrier either suffices or ends in BK_ERR_TIMEOUT
    with the engine usable afterwards."""
    eng.set_option("engine_mode", 4)
    bits, e0 = bk.select_trap(23, 3, 100, 0.3)
    eng.set_option("wait_polls", 1000)
    try:
        eng.evolve(23, bits, 0.35, 0.02, 4, e0=e0, precision=bk.BK_C64)
    except bk.BkError as e:
        assert e.status == 4
    finally:
        eng.set_option("wait_polls", 0)
    p, _, nn = eng.evolve(16, bk.select_trap(16, 3, 100, 0.3)[0], 0.35, 0.02, 4, precision=bk.BK_C128)
    assert np.max(np.abs(nn - 1.0)) <= 1e-12


# the whole-state kernel (up to 13 / 12 qubits): every tile (2^8 padded to 2^12
# elements), runs that end in either round layout, against the per-qubit path
@pytest.mark.parametrize("precision", [bk.BK_C64, bk.BK_C128])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 10, 11, 12, 13])
@pytest.mark.parametrize("steps", [0, 1, 6, 7])
def test_small_states_match_the_plain_path(eng, n, precision, steps):
    s0, g = (0b1011001110101 & ((1 << n) - 1)), np.linspace(0.3, 0.5, steps)
    a = eng.evolve(n, s0, g, 0.05, steps, precision=precision)
    psi = eng.export_state(n)
    b = eng.evolve(n, s0, g, 0.05, steps, precision=bk.BK_C128, method=bk.BK_PLAIN)
    ref = eng.export_state(n)
    c64 = precision == bk.BK_C64
    assert np.max(np.abs(a[0] - b[0])) <= (C64_DP_BAR if c64 else BAR128)
    assert np.max(np.abs(a[1] - b[1])) <= (C64_DH_BAR if c64 else BAR128 * n)
    assert np.max(np.abs(psi - ref)) <= BAR128  # complex64 runs of these sizes compute in complex128


@pytest.mark.parametrize("n", [5, 9, 12])
def test_small_runs_split_at_sampling_points(eng, n):
    s0 = 0b110100101110 & ((1 << n) - 1)
    kw = dict(n=n, g=0.35, dt=0.05, t_max=1.0, verbose=False, num_sampling_seeds=1)
    a = eng.sampler_run(s0, shots_per_point=0, num_sample_points=21, dt_sample=0.05, **kw)
    b = eng.sampler_run(s0, shots_per_point=16, num_sample_points=7, record_trajectory=True, dt_trajectory=0.05, **kw)
    # launches begin in round 0's layout: the sums of a step are the same terms, those
    # of a step in the other layout are summed in another order
    assert np.max(np.abs(a["p_less_history"] - b["p_less_history"])) <= BAR128
    assert np.max(np.abs(a["dh_history"] - b["dh_history"])) <= BAR128 * n


# the reverse sweep's tiles: 2^10 (13, 14, 18 element bits: a set of 3, 4, 8 bits), 2^12
# with two sets (19, 20, 21) and with three (22, 23, 25), against the launch-per-pass sweep;
# checkpoints that split the sweep into stretches of odd and even length
@pytest.mark.parametrize("n", [13, 14, 16, 17, 18, 19, 20, 21, 22, 23, 24, 25, 26, 27, 28])
def test_reverse_sweep_matches_the_launch_per_pass_sweep(eng, n):
    T, g = 11, np.linspace(0.3, 0.42, 11)
    bits, e0 = bk.select_trap(n, 13, 100, 0.3)
    out = []
    for mode in (1, 4):
        eng.set_option("engine_mode", mode)
        out.append([eng.adjoint(n, bits, g, 0.04, T, e0=e0, precision=bk.BK_C128, checkpoint_every=K)[:2] for K in (64, 4, 3)])
    for a, b in zip(*out):
        # FP64 rounding of ~32 T rotations on sums of products of amplitudes of norm 1
        assert abs(a[0] - b[0]) <= BAR128
        assert np.max(np.abs(a[1] - b[1])) <= 1e-11 * max(1e-3, np.max(np.abs(a[1])))


@pytest.mark.parametrize("n", [14, 20, 22, 24])
def test_reverse_sweep_complex64(eng, n):
    T, g = 8, np.linspace(0.3, 0.42, 8)
    bits, e0 = bk.select_trap(n, 13, 100, 0.3)
    eng.set_option("engine_mode", 4)
    a = eng.adjoint(n, bits, g, 0.04, T, e0=e0, precision=bk.BK_C64, checkpoint_every=3)
    b = eng.adjoint(n, bits, g, 0.04, T, e0=e0, precision=bk.BK_C128, checkpoint_every=3)
    assert np.max(np.abs(a[1] - b[1])) <= 1e-4 * np.max(np.abs(b[1]))  # the complex64 gradient's bar
    assert a[2]["max_drift"] <= 1e-5


# the full-space product in tile passes (from 23 bits on): every split of the far bits,
# against the per-state form on the same vectors
@pytest.mark.parametrize("n", [23, 24, 25, 26, 27, 28, 29, 30])
def test_full_space_tile_passes_match_the_per_state_form(eng, n):
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(1 << n, generator=gen, device="cuda", dtype=torch.float64)
    y, ref = torch.empty_like(x), torch.empty_like(x)
    torch.cuda.synchronize()
    eng.fullspace_matvec(n, 0.35, x, y)
    eng.fullspace_matvec(n, 0.35, x, ref, method=bk.BK_PLAIN)
    # n + 1 terms summed in another order
    bound = 1e-14 * (n + 1) * float(ref.abs().max())
    assert float(y.sub_(ref).abs().max()) <= bound
