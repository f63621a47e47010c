"""Performance cases: what a user of this package has it do, through its public calls.

Each case is a plain dict; ``prepare`` builds what a program holds before the
call (an engine with its tuned options, traps, schedules, vectors), ``run`` is
one call as such a program makes it, ``exact`` the same result in 64 bits from
plain torch. Sizes are those of the package's own workloads (single traps at
N = 12 to 28, the reference sampler's defaults at N = 16, batches of uneven N
from 16 to 22, schedule gradients, full-space products, trap generation) and
the sizes between them.

complex64 runs hand back their series in float32, the type they are computed
in; complex128 runs in float64. Their step counts are stretches of such a run:
every step is the same work, and a complex64 run rounds each amplitude N times a
step, so the error of a long run is a random walk of its own.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bernasconi-krylov_b200"))

import bk_b200 as bk  # noqa: E402
from bk_b200 import tune  # noqa: E402
from bk_b200.adjoint import TrotterSchedule  # noqa: E402

L2_BYTES = 126e6  # a state that fits here need not go to HBM between two steps


def listed():
    return [
        # the dense-ED comparison size: one trap, 400 steps of 0.05, measured every 10
        dict(name="evolve_n12_c128", kind="evolve", n=12, prec="c128", steps=400, every=10, dt=0.05, ramp=False),
        # the smallest call: a short run of a small trap, every step measured
        dict(name="evolve_n9_c64", kind="evolve", n=9, prec="c64", steps=100, every=1, dt=0.02, ramp=False),
        # the reference sampler with its own defaults (T = 60, dt = 0.05, 20 points x 100 shots x 3 seeds)
        dict(name="sampler_n16", kind="sampler", n=16, t_max=60.0, points=20, shots=100, seeds=3, trajectory=False),
        # ordinary single traps: a size with no tuned entry, in both precisions, and a field ramp
        dict(name="evolve_n19_c64", kind="evolve", n=19, prec="c64", steps=16, every=4, dt=0.02, ramp=True),
        dict(name="evolve_n21_c128", kind="evolve", n=21, prec="c128", steps=120, every=20, dt=0.02, ramp=False),
        # the N = 24 configuration (a tuned entry)
        dict(name="evolve_n24_c64", kind="evolve", n=24, prec="c64", steps=12, every=4, dt=0.02, ramp=False),
        # a large odd size in complex128 without a tuned entry
        dict(name="evolve_n25_c128", kind="evolve", n=25, prec="c128", steps=20, every=20, dt=0.02, ramp=False),
        # the headline size: N = 28 complex64
        dict(name="evolve_n28_c64", kind="evolve", n=28, prec="c64", steps=12, every=4, dt=0.02, ramp=False),
        # many traps x fields of uneven N in one call, P_< at every step
        dict(name="batch_40", kind="batch", count=40, n_lo=16, n_hi=22, step=2, prec="c64", steps=24, dt=0.02),
        # one optimiser step on a 16-segment schedule: objective and gradient
        dict(name="adjoint_n22_c64", kind="adjoint", n=22, prec="c64", steps=16, segments=16, keep=128, dt=0.02),
        # one product with the full-space Hamiltonian, the inner call of a Krylov solver
        dict(name="matvec_n27", kind="matvec", n=27),
        # trap generation: seeded single-flip descents in one batch
        dict(name="descent_n28", kind="descent", n=28, count=65536),
    ]


def draw(rng):
    kind = rng.choice(["evolve"] * 6 + ["sampler", "batch", "adjoint", "matvec", "descent"])
    if kind == "evolve":
        prec = rng.choice(["c64", "c64", "c128"])
        n = rng.randint(7, 28 if prec == "c64" else 26)
        # whole runs in complex128, stretches in complex64 (work at most the largest listed case's)
        if prec == "c64":
            steps = rng.randint(6, 12 if n > 26 else 16 if n > 13 else 60)
        else:
            steps = int(round(10 ** rng.uniform(1.0, min(2.6, math.log10(24 * 2.0 ** (26 - n))))))
        return dict(kind="evolve", n=n, prec=prec, steps=steps, every=rng.choice([1, 3, 4, 10]),
                    dt=rng.choice([0.02, 0.05]), ramp=rng.random() < 0.3)
    if kind == "sampler":
        return dict(kind="sampler", n=rng.randint(8, 20), t_max=float(rng.randint(5, 60)), points=rng.randint(2, 24),
                    shots=rng.randint(20, 400), seeds=rng.randint(1, 4), trajectory=rng.random() < 0.5)
    if kind == "batch":
        lo = rng.randint(14, 18)
        return dict(kind="batch", count=rng.randint(3, 40), n_lo=lo, n_hi=min(22, lo + rng.randint(0, 6)),
                    step=rng.choice([1, 2]), prec=rng.choice(["c64", "c64", "c128"]), steps=rng.randint(8, 24), dt=0.02)
    if kind == "adjoint":
        n = rng.randint(15, 22)
        prec = rng.choice(["c64", "c64", "c128"])
        seg = rng.choice([1, 4, 8, 16])
        return dict(kind="adjoint", n=n, prec=prec, steps=seg * rng.randint(1, (16 if prec == "c64" else 96) // seg),
                    segments=seg, keep=rng.choice([12, 64, 128]), dt=0.02)
    if kind == "matvec":
        return dict(kind="matvec", n=rng.randint(8, 27))
    return dict(kind="descent", n=rng.randint(14, 48), count=int(10 ** rng.uniform(2.5, 4.8)))


def _prec(case):
    return bk.BK_C64 if case.get("prec", "c128") == "c64" else bk.BK_C128


def _trap(n, seed):
    """A local minimum among a few hundred seeded descents, as the trap policy picks them."""
    return bk.select_trap(n, seed % (1 << 31), 200, 0.3)


def _field(case, seed):
    """The transverse field: a constant, or a linear ramp over the run."""
    r = random.Random(seed)
    g = 0.25 + 0.2 * r.random()
    return np.linspace(g, g + 0.1, case["steps"]) if case["ramp"] else g


def _measured(case):
    return list(range(0, case["steps"] + 1, case["every"]))


def _batch(case, seed):
    r = random.Random(seed)
    sizes = list(range(case["n_lo"], case["n_hi"] + 1, case["step"]))
    out = []
    for i in range(case["count"]):
        n = sizes[i % len(sizes)]
        bits, e0 = bk.select_trap(n, r.randrange(1 << 30), 40, 0.5)
        out.append(dict(n=n, s0=bits, e0=e0, g=0.2 + 0.3 * r.random()))
    return out


def _sampler_cfg(case, seed):
    return dict(n=case["n"], g=0.25 + 0.2 * random.Random(seed).random(), dt=0.05, t_max=case["t_max"],
                num_sample_points=case["points"], shots_per_point=case["shots"], num_sampling_seeds=case["seeds"],
                seed=seed % 100000, record_trajectory=case["trajectory"], verbose=False)


def _segments(case, seed):
    return np.random.default_rng(seed).uniform(0.25, 0.45, case["segments"])


def prepare(case, seed):
    kind, st = case["kind"], dict(case=case, eng=bk.Engine(0))
    if kind == "evolve":
        tune.apply(st["eng"], case["n"], _prec(case))
        st.update(trap=_trap(case["n"], seed), g=_field(case, seed), measure=_measured(case))
    elif kind == "sampler":
        st.update(trap=_trap(case["n"], seed), cfg=_sampler_cfg(case, seed))
    elif kind == "batch":
        st.update(inst=_batch(case, seed))
    elif kind == "adjoint":
        bits, e0 = _trap(case["n"], seed)
        st.update(sched=TrotterSchedule(st["eng"], case["n"], bits, _segments(case, seed), case["dt"], case["steps"],
                                        precision=_prec(case), checkpoint_every=case["keep"], e0=e0))
    elif kind == "matvec":
        gen = torch.Generator("cuda").manual_seed(seed)
        x = torch.randn(1 << case["n"], generator=gen, device="cuda", dtype=torch.float64)
        st.update(x=x, y=torch.empty_like(x), g=0.2 + 0.3 * random.Random(seed).random())
    else:
        st.update(starts=bk.random_states(case["n"], seed, case["count"]))
    return st


def run(st):
    case, eng, kind = st["case"], st["eng"], st["case"]["kind"]
    if kind == "evolve":
        bits, e0 = st["trap"]
        return _typed(case, eng.evolve(case["n"], bits, st["g"], case["dt"], case["steps"], measure=st["measure"], e0=e0,
                                       precision=_prec(case)))
    if kind == "sampler":
        r = eng.sampler_run(st["trap"][0], **st["cfg"])
        stats = r.pop("seed_stats")
        # as many states are distinct as the draws give: the rest of their room is empty
        distinct = np.zeros(case["points"] * case["shots"] * case["seeds"] + 1, dtype=np.uint64)
        distinct[:len(r["unique_basis"])] = r["unique_basis"]
        return r | {"unique_basis": distinct, "best": [s["best_energy"] for s in stats],
                    "flips": [s["mean_hamming_flips"] for s in stats]}
    if kind == "batch":
        return _typed(case, eng.evolve_batch(st["inst"], case["dt"], case["steps"], precision=_prec(case)))
    if kind == "adjoint":
        sched = st["sched"]
        sched.zero_grad()
        value = sched()
        value.backward()
        return _typed(case, (value.detach().numpy(), sched.g.grad.numpy()))
    if kind == "matvec":
        return eng.fullspace_matvec(case["n"], st["g"], st["x"], st["y"])
    return eng.steepest_descent(case["n"], st["starts"])


def _typed(case, series):
    t = np.float32 if case["prec"] == "c64" else np.float64
    return tuple(np.asarray(s).astype(t) for s in series)


def work(case):
    """Bytes and operations of one call. A step is one complex phase (6 operations) and N butterflies (4 operations
    an amplitude) on 2^N amplitudes; a state that no L2 holds is read and written once a step, a smaller one never."""
    def steps_of(n, steps, amp):
        state = 2.0 ** n * amp
        return (2 * state * steps if state > L2_BYTES else 2 * state), 2.0 ** n * steps * (4 * n + 6)

    kind = case["kind"]
    amp = 8 if case.get("prec") == "c64" else 16
    if kind == "evolve":
        b, f = steps_of(case["n"], case["steps"], amp)
    elif kind == "sampler":
        b, f = steps_of(case["n"], round(case["t_max"] / 0.05), amp)
        b += case["points"] * 2.0 ** case["n"] * amp
    elif kind == "batch":
        sizes = list(range(case["n_lo"], case["n_hi"] + 1, case["step"]))
        each = [steps_of(sizes[i % len(sizes)], case["steps"], amp) for i in range(case["count"])]
        b, f = sum(x[0] for x in each), sum(x[1] for x in each)
    elif kind == "adjoint":
        # forward, then the inverse steps on two states with one overlap product per qubit
        b, f = steps_of(case["n"], case["steps"], amp)
        b, f = 3 * b + 2.0 ** case["n"] * amp * (case["steps"] // case["keep"]) * 2, f * 4
    elif kind == "matvec":
        b, f = 18.0 * 2 ** case["n"], (case["n"] + 2.0) * 2 ** case["n"]
    else:
        # about n/3 flips of a random start, each after n trial energies of n - 1 correlations
        b, f = 32.0 * case["count"], case["count"] * (case["n"] / 3.0 + 1) * case["n"] * case["n"] * 4.0
    return {"bytes": b, "flops": f}


# ---- 64-bit results from plain torch ----

def _popcount(x):
    x = x - ((x >> 1) & 0x55555555)
    x = (x & 0x33333333) + ((x >> 2) & 0x33333333)
    x = (x + (x >> 4)) & 0x0F0F0F0F
    return (x + (x >> 8) + (x >> 16) + (x >> 24)) & 0x3F


def _energies(n, dev="cuda"):
    """E(s) of every state, from the spin autocorrelations C_k = (n - k) - 2 popcount((s ^ s >> k) & mask)."""
    out = torch.empty(1 << n, dtype=torch.int32, device=dev)
    piece = 1 << min(n, 24)
    for at in range(0, 1 << n, piece):
        s = torch.arange(at, at + piece, dtype=torch.int32, device=dev)
        e = torch.zeros_like(s)
        for k in range(1, n):
            c = (n - k) - 2 * _popcount((s ^ (s >> k)) & ((1 << (n - k)) - 1))
            e += c * c
        out[at:at + piece] = e
    return out


class _State:
    """A complex128 statevector and the step exp(i g dt sum X) exp(-i dt E / N)."""

    def __init__(self, n, s0, e0, dt):
        self.n, self.dt = n, dt
        self.E = _energies(n)
        self.below = (self.E < e0)
        self.phase = torch.polar(torch.ones(1, dtype=torch.float64, device="cuda"),
                                 torch.arange(int(self.E.max()) + 1, device="cuda", dtype=torch.float64) * (-dt / n))
        self.flips = _popcount(torch.arange(1 << n, dtype=torch.int32, device="cuda") ^ s0)
        self.psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        self.psi[s0] = 1.0

    def mix(self, v, angle):
        c, s = math.cos(angle), 1j * math.sin(angle)
        rx = torch.tensor([[c, s], [s, c]], dtype=torch.complex128, device="cuda")
        lo = 0
        while lo < self.n:
            w = min(7, self.n - lo)
            u = rx
            for _ in range(w - 1):
                u = torch.kron(u, rx)
            if lo == 0:
                v = (v.view(-1, 1 << w) @ u).view(-1)
            else:
                v = torch.matmul(u, v.view(-1, 1 << w, 1 << lo)).view(-1)
            lo += w
        return v

    def step(self, g):
        piece = 1 << min(self.n, 24)
        for at in range(0, 1 << self.n, piece):
            self.psi[at:at + piece] *= self.phase[self.E[at:at + piece].long()]
        self.psi = self.mix(self.psi, g * self.dt)

    def measure(self):
        p = self.psi.real ** 2 + self.psi.imag ** 2
        return float((p * self.below).sum()), float((p * self.flips).sum()), float(p.sum())


def _series(n, trap, dt, g_of, steps, measured):
    st = _State(n, trap[0], trap[1], dt)
    want, rows = set(measured), []
    for k in range(steps + 1):
        if k in want:
            rows.append(st.measure())
        if k < steps:
            st.step(g_of(k))
    return [np.array([r[i] for r in rows]) for i in range(3)]


def _exact_adjoint(case, seed):
    n, T, dt = case["n"], case["steps"], case["dt"]
    trap, g = _trap(n, seed), _segments(case, seed)
    per = T // case["segments"]
    st = _State(n, trap[0], trap[1], dt)
    for k in range(T):
        st.step(g[k // per])
    value = st.measure()[0]
    psi, lam = st.psi, st.psi * st.below
    grad = np.zeros(len(g))
    back = torch.conj(st.phase)[st.E.long()]
    for k in range(T - 1, -1, -1):
        gx = torch.zeros_like(psi)
        for q in range(n):
            gx += psi.view(-1, 2, 1 << q).flip(1).reshape(-1)
        grad[k // per] += -2.0 * dt * float(torch.vdot(lam, gx).imag)
        psi, lam = st.mix(psi, -g[k // per] * dt) * back, st.mix(lam, -g[k // per] * dt) * back
    return np.array(value), grad


def exact(case, seed):
    kind = case["kind"]
    if kind == "evolve":
        g = _field(case, seed)
        return tuple(_series(case["n"], _trap(case["n"], seed), case["dt"], (lambda k: g[k]) if case["ramp"] else (lambda k: g),
                             case["steps"], _measured(case)))
    if kind == "sampler":
        # the two recorded series; the drawn states and what is counted of them have no exact value
        cfg = _sampler_cfg(case, seed)
        steps, dt = round(case["t_max"] / 0.05), 0.05
        bits, _ = _trap(case["n"], seed)
        times, at = _sampler_times(cfg, steps)
        e0 = int(bk.labs_energy(case["n"], [bits])[0])
        p, d, _ = _series(case["n"], (bits, e0), dt, lambda k: cfg["g"], steps, at)
        return {"time_points": np.array(times), "p_less_history": p, "dh_history": d}
    if kind == "batch":
        inst = _batch(case, seed)
        rows = [_series(i["n"], (i["s0"], i["e0"]), case["dt"], lambda k, i=i: i["g"], case["steps"], range(case["steps"] + 1))
                for i in inst]
        return tuple(np.stack([r[k] for r in rows]) for k in range(3))
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind == "matvec":
        n, gen = case["n"], torch.Generator("cuda").manual_seed(seed)
        x = torch.randn(1 << n, generator=gen, device="cuda", dtype=torch.float64)
        y = torch.zeros_like(x)
        for q in range(n):
            y += x.view(-1, 2, 1 << q).flip(1).reshape(-1)
        g = 0.2 + 0.3 * random.Random(seed).random()
        return (_energies(n).double() / n) * x - g * y
    return None


def _sampler_times(cfg, steps):
    """The steps the sampler measures at: every step of a trajectory, else its sampling points."""
    if cfg["record_trajectory"]:
        at = list(range(steps + 1))
    else:
        at, due, taken = [], 0.0, 0
        for k in range(steps + 1):
            t = k * cfg["dt"]
            if t >= due - 1e-9 and due <= cfg["t_max"] + 1e-9:
                at.append(k)
            if t >= due - 1e-9 and due <= cfg["t_max"] + 1e-9 and taken < cfg["num_sample_points"]:
                taken += 1
                due += cfg["t_max"] / cfg["num_sample_points"]
    return [k * cfg["dt"] for k in at], at
