"""Device memory: a call that does not get its work space fails with
MPC_ERR_NOMEM and leaves the context as usable as before.  The memory is taken
by one tensor, up to a few hundred megabytes, and given back before the check.
"""
import numpy as np
import pytest

import mpc_tdse
from mpc_tdse.systems import random_system

pytestmark = pytest.mark.gpu

NOMEM = -4


def _setup(B):
    s = random_system([300] * 7, gauge="l", seed=2, e_max=8.0, d_scale=0.3)
    Io, w = mpc_tdse.to_au(2e14, 4.0)
    p = mpc_tdse.pulse_setup("sine", "l", Io, w, 0.0, 2, mpc_tdse.period(w, 2))
    X = np.zeros((B, s.ntot), complex)
    X[:, 0] = 1.0
    return s, [p] * B, X


def _gradient(ctx, pulses, X, B, steps):
    return ctx.batch_objective_gradient(pulses[:B], np.full((B, 6), 1e-3), np.full(B, 2.0), 0.0,
                                        0.1, steps, X[:B], 0, steps)


@pytest.mark.parametrize("op,path,B", [("fixed", "streaming", 1024),
                                       ("adaptive", "streaming", 1024),
                                       ("gradient", "streaming", 1024), ("gradient", "auto", 32)])
def test_context_survives_a_failed_allocation(op, path, B):
    """1024 pulses on 2100 states: 34 MB per vector of all pulses, of which the
    stage GEMM's work space has 18 and its gradient of 8 steps over 100; 32
    pulses: 1 MB, and 13 of them per step of a gradient on the persistent
    kernels."""
    import torch

    s, pulses, X = _setup(B)
    steps = 8 if B > 32 else 80

    def run(ctx, B):
        if op == "fixed":
            return ctx.batch_advance(pulses[:B], 0.0, 0.1, [3] * B, X[:B], history=True)
        if op == "adaptive":
            return ctx.batch_propagate(pulses[:B], 0.0, [0.3] * B, X[:B], dt_max=0.1)
        return _gradient(ctx, pulses, X, B, steps)

    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path(path)
        run(ctx, 2)   # loads the kernels
        torch.cuda.init()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8,
                          device="cuda")
        with pytest.raises(mpc_tdse.MpcError) as ei:
            run(ctx, B)
        assert ei.value.code == NOMEM
        del hog
        torch.cuda.empty_cache()
        got = run(ctx, B)
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path(path)
        want = run(ctx, B)
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(got, want))


def test_batched_objective_keeps_one_path_s_buffers():
    """The batched gradient's buffers may be sized to most of the free memory:
    what one path held (32 pulses, 160 steps: 2.2 GB and up) is free again once
    the other has run, and a larger set replaces a smaller one."""
    import torch

    s, pulses, X = _setup(32)
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    with mpc_tdse.Context.from_system(s) as ctx:
        want = {}
        for path in ("auto", "streaming"):
            ctx.set_path(path)
            want[path] = _gradient(ctx, pulses, X, 32, 2)
        held = free()
        for big, small in (("auto", "streaming"), ("streaming", "auto")):
            ctx.set_path(big)
            _gradient(ctx, pulses, X, 32, 160)
            assert held - free() > 2e9
            ctx.set_path(small)
            got = _gradient(ctx, pulses, X, 32, 2)
            assert abs(held - free()) < 0.2e9
            assert all(np.array_equal(a, b) for a, b in zip(got, want[small]))
        # the other way round in size, on one path: 160 steps replace 2
        ctx.set_path("auto")
        _gradient(ctx, pulses, X, 32, 2)
        first = _gradient(ctx, pulses, X, 32, 160)
        again = _gradient(ctx, pulses, X, 32, 160)
        assert all(np.array_equal(a, b) for a, b in zip(first, again))


def test_objective_without_gradient_holds_one_segment():
    """Two segments of 10,000 steps on 180 states (0.41 GB each): the objective
    alone takes the memory of one, and the gradient has the bits of another
    interval's."""
    import torch

    s = random_system([60, 70, 50], gauge="l", seed=2, e_max=8.0, d_scale=0.3)
    Io, w = mpc_tdse.to_au(2e14, 4.0)
    p = mpc_tdse.pulse_setup("sine", "l", Io, w, 0.0, 2, mpc_tdse.period(w, 2))
    x = np.zeros(s.ntot, complex)
    x[0] = 1.0
    u = np.full(6, 1e-3)
    with mpc_tdse.Context.from_system(s) as ctx:
        want = ctx.objective_gradient(p, u, 2.0, 0.0, 0.1, 20000, x, 0, 64)
        ctx.objective(p, u, 2.0, 0.0, 0.1, 3, x, 0, 2)
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.objective_gradient(p, u, 2.0, 0.0, 0.1, 3, x, 0, 2)   # loads the kernels
        free = torch.cuda.mem_get_info()[0]
        J = ctx.objective(p, u, 2.0, 0.0, 0.1, 20000, x, 0, 10000)
        assert free - torch.cuda.mem_get_info()[0] < 0.6e9
        g = ctx.objective_backward()
    assert J == want[0] and all(np.array_equal(a, b) for a, b in zip(g, want[1:]))
