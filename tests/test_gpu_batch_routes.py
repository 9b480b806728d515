"""The routes a batch can take beyond the plain ones: a scan that narrows from
the stage GEMM to the persistent batched kernels, more pulses than one launch
takes, slopes that do not fit shared memory, and the resident kernel for at most
8 pulses, which serves systems with a window of more than 800 states (no layout
on the persistent kernels) and what a wide adaptive batch has left at its end.

Fixed steps against the single-pulse path or the streaming path, within 3e-13
per step in any coefficient of a unit-norm state and twice that in norms and
populations: a step is 12 products whose sums round at 1e-16 of |h M v| <= 2.4 |v|
in two different orders.  Adaptive steps against the streaming path (the same
controller on other sums): end times equal, step counts within one, states within
1e-9, ten times the local tolerance.  (batch_advance gives NaN beyond a pulse's
own steps.)
"""
import numpy as np
import pytest

import mpc_tdse
from mpc_tdse.systems import random_system

pytestmark = pytest.mark.gpu

NO_LAYOUT = [450, 500, 450]   # the middle block's window has 900 states


def _case(n, gauge, B, seed=1):
    s = random_system(n, gauge=gauge, seed=len(n), e_max=8.0, d_scale=0.3)
    rng = np.random.default_rng(seed)
    pulses = []
    for b in range(B):
        Io, w = mpc_tdse.to_au(2e14 * (1 + b % 5), 4.0 + 0.1 * (b % 7))
        pulses.append(mpc_tdse.pulse_setup("gaussian" if b % 3 == 2 else "sine", gauge, Io, w,
                                           0.1 * b, 2, mpc_tdse.period(w, 2)))
    X = rng.standard_normal((B, s.ntot)) + 1j * rng.standard_normal((B, s.ntot))
    return s, pulses, X / np.linalg.norm(X, axis=1, keepdims=True)


def _check_fixed(ctx, pulses, X, t0, steps, which, Y, pop, nrm, pop_index):
    for b in which:
        k = int(steps[b])
        if k == 0:
            assert np.array_equal(Y[b], X[b])
            continue
        ct, p1, _, n1 = ctx.propagate(pulses[b], t0[b], 0.1, k, X[b], pop_index=pop_index)
        assert np.max(np.abs(Y[b] - ct)) < 3e-13 * k, b
        assert np.max(np.abs(pop[b, :k + 1] - p1)) < 6e-13 * k, b
        assert np.max(np.abs(nrm[b, :k] - n1)) < 6e-13 * k, b
        assert np.all(np.isnan(nrm[b, k:])) and np.all(np.isnan(pop[b, k + 1:]))


@pytest.mark.parametrize("gauge", ["l", "v"])
def test_fixed_scan_moves_from_the_gemm_to_the_persistent_kernels(gauge):
    """256 pulses on 1752 states start on the stage GEMM and move over at about
    190: 20 pulses end with step 1 and 30 with step 3, so that the batch has
    been compacted before; two have no steps at all."""
    n, B = [292] * 6, 256
    s, pulses, X = _case(n, gauge, B)
    steps = np.array([5 + (7 * b) % 31 for b in range(B)])
    steps[5::13] = 1
    steps[3::8] = 3
    steps[[0, 77]] = 0
    t0 = 0.05 * np.arange(B)
    with mpc_tdse.Context.from_system(s) as ctx:
        l0 = ctx.launches
        Y, pop, nrm = ctx.batch_advance(pulses, t0, 0.1, steps, X, pop_index=s.ntot - 1,
                                        history=True)
        assert ctx.launches - l0 < 60   # (at least 3 for each of 35 steps on the GEMM)
        _check_fixed(ctx, pulses, X, t0, steps, list(range(0, B, 9)) + [5, 77, 255], Y, pop, nrm,
                     s.ntot - 1)
        ctx.set_path("streaming")
        Z, pop2, nrm2 = ctx.batch_advance(pulses, t0, 0.1, steps, X, pop_index=s.ntot - 1,
                                          history=True)
    tol = 3e-13 * np.maximum(steps, 1)
    assert np.all(np.max(np.abs(Y - Z), axis=1) < tol)
    assert np.nanmax(np.abs(pop - pop2)) < 2 * tol.max()
    assert np.array_equal(np.isnan(nrm), np.isnan(nrm2))
    assert not np.array_equal(Y, Z)   # (the tail's sums are in another order)


def _check_adaptive(s, pulses, X, t0, t_end, paths=("auto", "streaming")):
    out = []
    for path in paths:
        with mpc_tdse.Context.from_system(s) as ctx:
            ctx.set_path(path)
            out.append(ctx.batch_propagate(pulses, t0, t_end, X, dt_max=0.2))
    (Y, acc, rej, tf), (Z, acc2, rej2, tf2) = out
    assert np.array_equal(tf, tf2) and np.array_equal(tf, t_end)
    assert np.max(np.abs(acc.astype(int) - acc2)) <= 1
    assert np.max(np.abs(Y - Z)) < 1e-9
    return Y, Z


@pytest.mark.parametrize("n,B", [([380] * 10, 200), ([388] * 9, 60)],
                         ids=["two-launches", "slopes-in-global-memory"])
def test_adaptive_batches_beyond_one_launch_and_shared_memory(n, B):
    """25 chunks of 8 pulses on one column group (a launch takes 16), and 8
    chunks of 24 or more rows, whose slopes have no room in shared memory."""
    s, pulses, X = _case(n, "l", B)
    t0 = 0.02 * np.arange(B)
    _check_adaptive(s, pulses, X, t0, t0 + 0.2 + 0.05 * (np.arange(B) % 5))


@pytest.mark.parametrize("gauge", ["l", "v"])
@pytest.mark.parametrize("B", [1, 3, 8, 20])
def test_resident_kernel_fixed_steps(B, gauge):
    """Up to 8 pulses from the start, and the last 8 of 20."""
    s, pulses, X = _case(NO_LAYOUT, gauge, B)
    steps = np.array([(5 * b + 3) % 17 + (b % 2) * 20 for b in range(B)])
    t0 = 0.3 * np.arange(B)
    with mpc_tdse.Context.from_system(s) as ctx:
        l0 = ctx.launches
        Y, pop, nrm = ctx.batch_advance(pulses, t0, 0.1, steps, X, pop_index=700, history=True)
        if B <= 8:
            assert ctx.launches - l0 < 2 * B + 12   # (not a launch per product)
        _check_fixed(ctx, pulses, X, t0, steps, range(B), Y, pop, nrm, 700)


@pytest.mark.parametrize("n,B", [(NO_LAYOUT, 1), (NO_LAYOUT, 3), (NO_LAYOUT, 8), (NO_LAYOUT, 20),
                                 ([300] * 7, 96)], ids=lambda v: str(v) if isinstance(v, int) else
                         f"{len(v)}x{max(v)}")
def test_resident_kernel_adaptive_steps(n, B):
    """The same, and a batch that starts too wide for the persistent kernels (96
    pulses on 2100 states), of which 7 pulses run on."""
    s, pulses, X = _case(n, "v", B)
    t0 = 0.1 * np.arange(B)
    t_end = t0 + 0.3 + 0.1 * (np.arange(B) % 4)
    t_end[::14] += 1.0
    if B > 2:
        t_end[1] = t0[1]
    Y, Z = _check_adaptive(s, pulses, X, t0, t_end)
    assert not np.array_equal(Y, Z)
    if B > 2:
        assert np.array_equal(Y[1], X[1])


def test_resident_kernel_in_two_contexts_of_different_size():
    """The kernel's shared-memory limit belongs to the function: a second,
    smaller system must not take it from the first."""
    big, pb, Xb = _case(NO_LAYOUT, "l", 2)
    small, ps, Xs = _case([401, 30, 402], "l", 2)
    with mpc_tdse.Context.from_system(big) as a, mpc_tdse.Context.from_system(small) as b:
        Y0 = a.batch_advance(pb, 0.0, 0.1, [4, 5], Xb)
        b.batch_advance(ps, 0.0, 0.1, [4, 5], Xs)
        assert np.array_equal(a.batch_advance(pb, 0.0, 0.1, [4, 5], Xb), Y0)


# ---- failures ----

@pytest.mark.parametrize("op,n,B", [("fixed", [60, 70, 50], 9), ("fixed", [97] * 5, 20),
                                    ("fixed", NO_LAYOUT, 3), ("adaptive", [97] * 5, 20),
                                    ("adaptive", NO_LAYOUT, 3), ("gradient", [60, 70, 50], 9),
                                    ("gradient", [97] * 5, 20)],
                         ids=lambda v: f"{len(v)}x{max(v)}" if isinstance(v, list) else str(v))
def test_wait_that_runs_out_is_reported(op, n, B):
    """Arrival targets one beyond what the CTAs can make (limit 1 ms), in every
    mode of the persistent batched kernels and in the resident kernel: the call
    fails, the context goes on and gives the bits it gave before."""
    s, pulses, X = _case(n, "l", B)
    U, T = np.full((B, 6), 1e-3), np.full(B, 2.0)

    def run(ctx, inject=False):
        if op == "gradient":
            ctx.batch_objective(pulses, U, T, 0.1, 0.1, 6, X, 0, 2)
        if inject:
            ctx.set_wait_limit(1e-3)
            ctx.inject_barrier_timeout()
        if op == "fixed":
            return ctx.batch_advance(pulses, 0.0, 0.1, [6 + b % 3 for b in range(B)], X,
                                     history=True)
        if op == "adaptive":
            return ctx.batch_propagate(pulses, 0.0, [0.5] * B, X, dt_max=0.1)
        return ctx.batch_objective_backward()

    with mpc_tdse.Context.from_system(s) as ctx:
        want = run(ctx)
        with pytest.raises(mpc_tdse.MpcError) as ei:
            run(ctx, inject=True)
        assert ei.value.code == -3
        ctx.set_wait_limit(2.0)
        assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(run(ctx), want))


@pytest.mark.parametrize("path", ["auto", "streaming"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_pulse_beside_finite_ones(bad, path):
    """Fixed steps fail as a whole; an adaptive pulse that is not finite gives up
    alone: the call reports it, and the others' states, counts and times are
    written; the objective and its gradient are NaN for that pulse.  The others
    have the bits they have beside a finite pulse."""
    import ctypes as C

    s, pulses, X = _case([97] * 5, "l", 12)
    Xbad = X.copy()
    Xbad[4, 200] = bad
    U, T = np.full((12, 6), 1e-3), np.full(12, 2.0)
    dp, ip = C.POINTER(C.c_double), C.POINTER(C.c_int)
    arr = (mpc_tdse.Pulse * 12)(*pulses)
    t0, te = np.zeros(12), 0.3 + 0.05 * np.arange(12)
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path(path)

        def adaptive(x):
            xf = x.view(np.float64).copy()
            acc, rej, tf = np.zeros(12, np.int32), np.zeros(12, np.int32), np.zeros(12)
            rc = mpc_tdse.lib().mpc_batch_propagate(
                ctx._h, 12, arr, t0.ctypes.data_as(dp), te.ctypes.data_as(dp), 0.05, 0.2, 1e-10,
                1e-10, 0, xf.ctypes.data_as(dp), acc.ctypes.data_as(ip), rej.ctypes.data_as(ip),
                tf.ctypes.data_as(dp))
            return rc, xf.view(np.complex128), acc, rej, tf

        with pytest.raises(mpc_tdse.MpcError) as ei:
            ctx.batch_advance(pulses, 0.0, 0.1, [5] * 12, Xbad)
        assert ei.value.code == -3
        rc, Y, acc, rej, tf = adaptive(Xbad)
        rc0, Y0, acc0, rej0, tf0 = adaptive(X)
        assert rc == -3 and rc0 == 0
        ok = np.arange(12) != 4
        grads = [ctx.batch_objective_gradient(pulses, U, T, 0.0, 0.1, 5, x, 0, 2) for x in (Xbad, X)]
        for a, b in zip(*grads):
            assert np.array_equal(a[ok], b[ok]) and np.all(np.isfinite(b))
            assert np.all(np.isnan(a[4]) | (a[4] == 0.0)) and np.any(np.isnan(a[4]))
        for a, b in ((Y, Y0), (acc, acc0), (rej, rej0), (tf, tf0)):
            assert np.array_equal(a[ok], b[ok])
        assert acc[4] == 0 and tf[4] == 0.0
