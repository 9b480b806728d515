"""The batched gradient on the stage GEMM, which wide batches and systems too
large for the persistent kernels take: here on the streaming path, at sizes those
kernels would take otherwise, against the single-pulse adjoint, the CPU oracle
and central differences.

Tolerances as for the persistent kernels' gradient: objectives 1e-12 absolute,
dJ/du and dJ/dF_n 1e-9 relative to the largest component; central differences
1e-6 relative.
"""
import numpy as np
import pytest

import mpc_tdse
from mpc_tdse.systems import helium_like_2e, hydrogen_like_1e, random_system

pytestmark = pytest.mark.gpu


def _batch(g, B, K=40, seed=0):
    rng = np.random.default_rng(seed)
    ps, T = [], []
    for _ in range(B):
        Io, w = mpc_tdse.to_au(10 ** rng.uniform(13.5, 14.5), rng.uniform(1.4, 3.0))
        T.append(mpc_tdse.period(w, 1))
        ps.append(mpc_tdse.pulse_setup("sine", g, Io, w, 0.0, 1, T[-1]))
    U = np.stack([rng.standard_normal(K) * 0.01 * p.Eo for p in ps])
    return ps, U, np.array(T)


# blocks, pulses: 4 row tiles; 9 of ragged size, 33 columns; 36; one row, one column
@pytest.mark.parametrize("g", ["l", "v"])
@pytest.mark.parametrize("target", [-1, 4])
@pytest.mark.parametrize("n,B", [([36] * 4, 5), ([70, 90, 100, 165], 33), ([200] * 9, 3),
                                 ([1, 5, 1], 1), ([130, 7, 65], 66)],
                         ids=lambda v: str(v) if isinstance(v, int) else f"{len(v)}x{max(v)}")
def test_gradient_matches_single_pulse_adjoint(n, B, target, g):
    s = random_system(n, gauge=g, seed=len(n), e_max=8.0, d_scale=0.3)
    pulses, U, T = _batch(g, B)
    rng = np.random.default_rng(2)
    X = rng.standard_normal((B, s.ntot)) + 1j * rng.standard_normal((B, s.ntot))
    X /= np.linalg.norm(X, axis=1, keepdims=True)
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path("streaming")
        ctx.objective_threshold(2.0)
        J, G, Fb = ctx.batch_objective_gradient(pulses, U, T, 0.0, 0.1, 40, X, target, ckpt_every=16)
        for b in range(0, B, max(1, B // 6)):
            j1, g1, f1 = ctx.objective_gradient(pulses[b], U[b], T[b], 0.0, 0.1, 40, X[b], target,
                                                ckpt_every=16)
            assert abs(J[b] - j1) < 1e-12, b
            assert np.max(np.abs(G[b] - g1)) <= 1e-9 * np.max(np.abs(g1)), b
            assert np.max(np.abs(Fb[b] - f1)) <= 1e-9 * np.max(np.abs(f1)), b


def test_gradient_matches_oracle(oracle):
    s = hydrogen_like_1e(30, 3, gauge="l", seed=2)
    pulses, U, T = _batch("l", 3, K=48, seed=5)
    X0 = np.zeros((3, s.ntot), complex)
    X0[:, 0] = 1.0
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path("streaming")
        J, G, _ = ctx.batch_objective_gradient(pulses, U, T, 0.0, 0.1, 250, X0, -1)
    for b in range(3):
        Jo, go, _, _ = oracle.objective_gradient(s.n, s.eig, s.dip, "l", "sineEE",
                                                 pulses[b].as_array(), U[b], T[b], 0.0, 0.1, 250,
                                                 X0[b], -1)
        assert abs(J[b] - Jo) < 1e-12
        assert np.max(np.abs(G[b] - go)) <= 1e-9 * np.max(np.abs(go))


def test_2e_yield_and_central_difference():
    s = helium_like_2e((40, 48, 44, 36), gauge="v", seed=4, e_max=8.0)
    rng = np.random.default_rng(7)
    pulses, T = [], []
    for _ in range(4):
        Io, w = mpc_tdse.to_au(10 ** rng.uniform(14.5, 15), rng.uniform(5.0, 7.0))
        T.append(mpc_tdse.period(w, 2))
        pulses.append(mpc_tdse.pulse_setup("sine", "v", Io, w, 0.0, 2, T[-1]))
    U = np.stack([rng.standard_normal(32) * 0.01 * p.Eo for p in pulses])
    T = np.array(T)
    steps = int(max(T) / 0.05) + 1
    X0 = np.zeros((4, s.ntot), complex)
    X0[:, 0] = 1.0
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path("streaming")
        ctx.objective_threshold(-2.0)
        J, G, _ = ctx.batch_objective_gradient(pulses, U, T, 0.0, 0.05, steps, X0, -1)
        h = 1e-6
        k = [int(np.argmax(np.abs(G[b]))) for b in range(4)]
        Up, Um = U.copy(), U.copy()
        for b in range(4):
            Up[b, k[b]] += h
            Um[b, k[b]] -= h
        Jp = ctx.batch_objective(pulses, Up, T, 0.0, 0.05, steps, X0, -1)
        Jm = ctx.batch_objective(pulses, Um, T, 0.0, 0.05, steps, X0, -1)
    for b in range(4):
        fd = (Jp[b] - Jm[b]) / (2 * h)
        assert 0.0 < J[b] < 1.0
        assert abs(fd - G[b, k[b]]) <= 1e-6 * abs(fd), (b, fd, G[b, k[b]])


def test_checkpoint_interval_and_reallocation_are_bit_identical():
    """Intervals that make the work buffers grow and shrink between calls, on 35
    columns; 0: sized to the free memory; a second reverse pass."""
    s = random_system([100, 130, 65], gauge="v", seed=3, e_max=8.0, d_scale=0.3)
    pulses, U, T = _batch("v", 35, K=24, seed=9)
    X0 = np.zeros((35, s.ntot), complex)
    X0[:, 0] = 1.0
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path("streaming")
        r = []
        for c in (64, 9, 500, 100, 1, 0):
            r.append(ctx.batch_objective_gradient(pulses, U, T, 0.0, 0.1, 101, X0, 0, ckpt_every=c))
            G2, Fb2 = ctx.batch_objective_backward()
            assert np.array_equal(G2, r[-1][1]) and np.array_equal(Fb2, r[-1][2])
    for got in r[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(got, r[0]))
