"""The persistent fixed-step launch of the stage GEMM, whose wider tiles run on a
ring with barriers per slot, against one launch per product with a CTA barrier
per chunk: the same sums in the same order, so the same bits.  Windows of fewer
chunks (32 rows) than the ring has slots, of as many, and of many; rows and
columns that end inside a tile."""
import numpy as np
import pytest

import mpc_tdse
from mpc_tdse.systems import random_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [2, 3, 4])   # 32 columns x 3 and 6 slots, 64 x 3
@pytest.mark.parametrize("n", [[3, 5], [33, 64, 31, 97], [300, 7, 250, 129, 64]])
@pytest.mark.parametrize("pulses", [5, 41])
def test_ring_equals_barrier_per_chunk(monkeypatch, variant, n, pulses):
    s = random_system(n, gauge="v", seed=sum(n))
    Io, w = mpc_tdse.to_au(1e13, 1.5498)
    tau = mpc_tdse.period(w, 1)
    ps = [mpc_tdse.pulse_setup("sine", "v", Io * (0.5 + 0.01 * b), w, 0.0, 1, tau)
          for b in range(pulses)]
    rng = np.random.default_rng(5)
    X0 = rng.standard_normal((pulses, s.ntot)) + 1j * rng.standard_normal((pulses, s.ntot))
    X0 /= np.linalg.norm(X0, axis=1)[:, None]
    steps = [1 + b % 6 for b in range(pulses)]
    monkeypatch.setenv("MPC_BATCH_VARIANT", str(variant))
    out = []
    for env in ("MPC_FORCE_PERSIST", "MPC_NO_PERSIST"):
        monkeypatch.delenv("MPC_FORCE_PERSIST", raising=False)
        monkeypatch.setenv(env, "1")
        with mpc_tdse.Context.from_system(s) as ctx:
            ctx.set_path("streaming")
            out.append(ctx.batch_advance(ps, 0.0, 0.002, steps, X0, history=True))
    for a, b in zip(*out):
        assert np.isfinite(np.asarray(out[0][0])).all()
        assert np.array_equal(a, b, equal_nan=True)
