"""The persistent batched kernels (systems whose coupling fits on chip) at the
sizes where their layout can go wrong: one-row blocks, blocks much longer or
shorter than their neighbours, every row tile, pulse counts around the chunks
of 8 and the column groups, pulses without steps, single steps.

Each pulse against the single-pulse path (or, for adaptive steps, the CPU
oracle).  A step is 12 products whose sums round at 1e-16 of |h M v| <= 2.4 |v|
in two different orders, so n steps agree within n x 13 x 2.4 x ~50 eps:
3e-13 per step in any coefficient of a unit-norm state, twice that in norms
and populations.
"""
import numpy as np
import pytest

import mpc_tdse
from mpc_tdse.systems import random_system

pytestmark = pytest.mark.gpu

SYSTEMS = [[1, 1], [1, 7, 1, 2], [60, 70, 50], [97] * 5, [201] * 8, [292] * 6, [33] * 16,
           [388, 387, 386, 385, 384, 383, 382, 381, 380], [5, 500, 7]]


def _case(n, gauge, B):
    s = random_system(n, gauge=gauge, seed=len(n), e_max=8.0, d_scale=0.3)
    rng = np.random.default_rng(B)
    pulses = []
    for b in range(B):
        Io, w = mpc_tdse.to_au(2e14 * (1 + b % 5), 4.0 + 0.1 * (b % 7))
        pulses.append(mpc_tdse.pulse_setup("gaussian" if b % 3 == 2 else "sine", gauge, Io, w,
                                           0.1 * b, 2, mpc_tdse.period(w, 2)))
    X = rng.standard_normal((B, s.ntot)) + 1j * rng.standard_normal((B, s.ntot))
    return s, pulses, X / np.linalg.norm(X, axis=1, keepdims=True)


@pytest.mark.parametrize("gauge", ["l", "v"])
@pytest.mark.parametrize("B", [1, 7, 8, 9, 35])
@pytest.mark.parametrize("n", SYSTEMS, ids=lambda n: f"{len(n)}x{max(n)}")
def test_fixed_steps_match_single_pulse(n, B, gauge):
    s, pulses, X = _case(n, gauge, B)
    steps = np.array([(5 * b + 3) % 7 for b in range(B)])   # 0 to 6, one of them 0 from B = 7
    t0 = 0.3 * np.arange(B)
    with mpc_tdse.Context.from_system(s) as ctx:
        Y, pop, nrm = ctx.batch_advance(pulses, t0, 0.1, steps, X, pop_index=s.ntot - 1,
                                        history=True)
        for b in range(B):
            k = int(steps[b])
            if k == 0:
                assert np.array_equal(Y[b], X[b])
                continue
            ct, p1, _, n1 = ctx.propagate(pulses[b], t0[b], 0.1, k, X[b], pop_index=s.ntot - 1)
            assert np.max(np.abs(Y[b] - ct)) < 3e-13 * k, b
            assert np.max(np.abs(pop[b, :k + 1] - p1)) < 6e-13 * k, b
            assert np.max(np.abs(nrm[b, :k] - n1)) < 6e-13 * k, b
            assert np.all(np.isnan(nrm[b, k:])) and np.all(np.isnan(pop[b, k + 1:]))


@pytest.mark.parametrize("gauge", ["l", "v"])
@pytest.mark.parametrize("B", [1, 9, 20])
@pytest.mark.parametrize("n", SYSTEMS, ids=lambda n: f"{len(n)}x{max(n)}")
def test_gradient_matches_single_pulse(n, B, gauge):
    """Gradients relative to the largest component (both factors of each
    Re<M1 vbar, v> carry the bound above: 1e-11 over 5 steps); segments of one
    step, shorter than the window, and one for all; a second reverse pass."""
    s, pulses, X = _case(n, gauge, B)
    U = np.random.default_rng(3).standard_normal((B, 6)) * 1e-3
    T = np.full(B, 2.0)
    with mpc_tdse.Context.from_system(s) as ctx:
        first = None
        for steps, ckpt in ((1, 64), (5, 2), (5, 64), (5, 1)):
            J, G, Fb = ctx.batch_objective_gradient(pulses, U, T, 0.1, 0.1, steps, X, 0, ckpt)
            G2, Fb2 = ctx.batch_objective_backward()
            assert np.array_equal(G, G2) and np.array_equal(Fb, Fb2)
            if steps == 5:
                first = first or (J, G, Fb)
                assert all(np.array_equal(x, y) for x, y in zip(first, (J, G, Fb)))
            for b in range(0, B, 4):
                j, g, f = ctx.objective_gradient(pulses[b], U[b], 2.0, 0.1, 0.1, steps, X[b], 0)
                assert abs(J[b] - j) < 4e-12
                assert np.max(np.abs(Fb[b] - f)) <= 1e-11 * max(np.max(np.abs(f)), 1e-3)
                assert np.max(np.abs(G[b] - g)) <= 1e-11 * max(np.max(np.abs(g)), 1e-3)


@pytest.mark.parametrize("gauge", ["l", "v"])
@pytest.mark.parametrize("B", [1, 9, 20])
@pytest.mark.parametrize("n", [[1, 1], [60, 70, 50], [97] * 5, [201] * 8, [5, 500, 7]],
                         ids=lambda n: f"{len(n)}x{max(n)}")
def test_adaptive_steps_match_stage_gemm(n, B, gauge):
    """Against the stage-GEMM path (the same controller on other sums): the
    same accepted and rejected steps and end times; states within 1e-9, ten
    times the local tolerance of 1e-10, since the step sizes follow an error
    estimate that is itself rounding noise of the slopes.  A pulse with nothing
    to do comes back as it went in."""
    s, pulses, X = _case(n, gauge, B)
    t0 = 0.3 * np.arange(B)
    t_end = t0 + 0.8 + 0.1 * (np.arange(B) % 9)
    if B > 1:
        t_end[1] = t0[1]
    out = []
    for path in ("auto", "streaming"):
        with mpc_tdse.Context.from_system(s) as ctx:
            ctx.set_path(path)
            out.append(ctx.batch_propagate(pulses, t0, t_end, X, dt_max=0.2))
    (Y, acc, rej, tf), (Z, acc2, rej2, tf2) = out
    assert np.array_equal(tf, tf2) and np.array_equal(tf, t_end)
    assert np.array_equal(acc, acc2) and np.array_equal(rej, rej2)
    assert np.max(np.abs(Y - Z)) < 1e-9
    if B > 1:
        assert np.array_equal(Y[1], X[1]) and acc[1] == 0
