"""The resident path's persistent kernels at the sizes where their layout can
go wrong: every register tile of the forward and the reverse pass and the
shared-memory form, blocks of one row, blocks much longer or shorter than their
neighbours, one step and several, checkpoint segments shorter than the window.

Forward against the CPU oracle's loop.  Both are the same frozen-field RKF78
step, evaluated in two orders: per step about 13 products whose sums of up to
a few thousand terms round at 1e-16 of |h M v| <= 2.4 |v|, so 6 steps stay
within 6 x 13 x 2.4 x ~50 eps = 2e-12 in any coefficient of a unit-norm state.
Gradients against the streamed kernels' stage-by-stage adjoint, relative to the
largest component: the same bound on both factors of Re<M1 v, v>, 1e-11.
"""
import numpy as np
import pytest

import mpc_tdse
from mpc_tdse.systems import random_system

pytestmark = pytest.mark.gpu

SYSTEMS = [[1, 1], [1, 7, 1, 2], [60, 70, 50], [97] * 5, [150] * 7, [292] * 6, [201] * 10,
           [301] * 9, [388, 387, 386, 385, 384, 383, 382, 381, 380], [399] * 10,
           [1156, 1063, 182], [5, 2500, 7], [297, 10, 205, 132, 226, 3, 185], [33] * 16]


def _case(n, gauge):
    s = random_system(n, gauge=gauge, seed=len(n), e_max=8.0, d_scale=0.3)
    Io, w = mpc_tdse.to_au(2e14, 6.0)
    p = mpc_tdse.pulse_setup("sine", gauge, Io, w, 0.2, 2, mpc_tdse.period(w, 2))
    rng = np.random.default_rng(len(n))
    x = rng.standard_normal(s.ntot) + 1j * rng.standard_normal(s.ntot)
    return s, p, x / np.linalg.norm(x)


@pytest.mark.parametrize("gauge", ["l", "v"])
@pytest.mark.parametrize("n", SYSTEMS, ids=lambda n: f"{len(n)}x{max(n)}")
def test_forward_matches_oracle(oracle, n, gauge):
    s, p, x = _case(n, gauge)
    kind = "sineEE" if gauge == "l" else "sineAA"
    with mpc_tdse.Context.from_system(s) as ctx:
        ctx.set_path("resident")
        for steps in (1, 2, 6):
            ct, pop, fld, nrm = ctx.propagate(p, 9.0, 0.1, steps, x, pop_index=s.ntot - 1)
            co, po, fo, no = oracle.propagate(s.n, s.eig, s.dip, gauge, kind, p.as_array(), 9.0,
                                              0.1, steps, x, pop_index=s.ntot - 1)
            assert np.array_equal(fld, fo)
            assert np.max(np.abs(ct - co)) < 2e-12, steps
            assert np.max(np.abs(pop - po)) < 4e-12, steps
            assert np.max(np.abs(nrm - no)) < 4e-12, steps


@pytest.mark.parametrize("gauge", ["l", "v"])
@pytest.mark.parametrize("n", SYSTEMS, ids=lambda n: f"{len(n)}x{max(n)}")
def test_gradient_matches_streamed(n, gauge):
    s, p, x = _case(n, gauge)
    u = np.random.default_rng(7).standard_normal(6) * 1e-3
    with mpc_tdse.Context.from_system(s) as ctx:
        for steps, ckpt in ((1, 64), (5, 2), (4, 4)):
            out = []
            for path in ("resident", "streaming"):
                ctx.set_path(path)
                J, g, f = ctx.objective_gradient(p, u, 2.0, 0.1, 0.1, steps, x, 0, ckpt)
                # a second reverse pass recomputes what the first overwrote
                g2, f2 = ctx.objective_backward()
                assert np.array_equal(g, g2) and np.array_equal(f, f2)
                out.append((J, g, f))
            (J1, g1, f1), (J2, g2, f2) = out
            assert abs(J1 - J2) < 4e-12
            assert np.max(np.abs(f1 - f2)) <= 1e-11 * max(np.max(np.abs(f2)), 1e-3)
            assert np.max(np.abs(g1 - g2)) <= 1e-11 * max(np.max(np.abs(g2)), 1e-3)
