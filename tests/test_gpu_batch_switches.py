"""Switches that say how the batched stage GEMM runs keep a batch on it, also
on a system that the persistent batched kernels would take: the same bits as on
the streaming path, whose sums those kernels add in another order.  Twelve
pulses that end together, so that no narrower tail takes over.
"""
import numpy as np
import pytest

import mpc_tdse
from mpc_tdse.systems import random_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op,switch", [("fixed", "MPC_BATCH_VARIANT=1"),
                                       ("adaptive", "MPC_BATCH_VARIANT=1"),
                                       ("gradient", "MPC_BATCH_VARIANT=1"),
                                       ("fixed", "MPC_NO_PERSIST=1"),
                                       ("fixed", "MPC_FORCE_PERSIST=1"),
                                       ("fixed", "MPC_FORCE_TMA=2")])
def test_switch_keeps_the_batch_on_the_stage_gemm(monkeypatch, switch, op):
    s = random_system([60, 70, 50], gauge="l", seed=3, e_max=8.0, d_scale=0.3)
    B = 12
    rng = np.random.default_rng(1)
    X = rng.standard_normal((B, s.ntot)) + 1j * rng.standard_normal((B, s.ntot))
    X /= np.linalg.norm(X, axis=1, keepdims=True)
    Io, w = mpc_tdse.to_au(2e14, 4.0)
    p = mpc_tdse.pulse_setup("sine", "l", Io, w, 0.0, 2, mpc_tdse.period(w, 2))
    U = rng.standard_normal((B, 6)) * 1e-3

    def run(path):
        with mpc_tdse.Context.from_system(s) as ctx:
            ctx.set_path(path)
            if op == "fixed":
                return ctx.batch_advance([p] * B, 0.0, 0.1, [9] * B, X, history=True)
            if op == "adaptive":   # one start state, so that the step counts agree
                return ctx.batch_propagate([p] * B, 0.0, [1.0] * B, X[[0] * B], dt_max=0.2)
            return ctx.batch_objective_gradient([p] * B, U, np.full(B, 2.0), 0.0, 0.1, 9, X, 0, 4)

    plain = run("auto")
    monkeypatch.setenv(*switch.split("="))
    got, want = run("auto"), run("streaming")
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    # (what the switch would otherwise leave it on)
    assert not all(np.array_equal(a, b) for a, b in zip(plain, want))
