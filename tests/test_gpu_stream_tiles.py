"""The dipole stream at the edges of its tiles (16 x 256), of its pairs of
tiles and of its runs of 512 staged rows, against the plain products.

Tolerance: an n-term sum of products errs by at most (n + 2) eps sum |terms|,
in any order; the terms here are the row and column sums of both neighbouring
blocks and the diagonal one."""
import numpy as np
import pytest

import mpc_tdse
from mpc_tdse.systems import random_system

pytestmark = pytest.mark.gpu

SIZES = {
    "one-tile": [1, 1],
    "tile-edges": [15, 255, 16, 256, 17, 257],
    "pairs": [31, 33, 32, 513, 47, 49, 63],
    "ragged": [129, 1031, 511, 300],
    "long-runs": [4500, 4417],   # more than 32 tiles of one strip per CTA
}


@pytest.mark.parametrize("gauge", ["l", "v"])
@pytest.mark.parametrize("name", list(SIZES))
def test_stream_tile_edges(name, gauge):
    n = SIZES[name]
    s = random_system(n, gauge=gauge, seed=len(n))
    rng = np.random.default_rng(3)
    x = rng.standard_normal(s.ntot) + 1j * rng.standard_normal(s.ntot)
    F = 0.43
    off = np.concatenate([[0], np.cumsum(n)])
    eig, dip = np.asarray(s.eig), np.asarray(s.dip)
    want = -1j * eig * x
    size = np.abs(eig * x)
    at = 0
    for L in range(len(n) - 1):
        d = dip[at:at + n[L] * n[L + 1]].reshape(n[L], n[L + 1])
        at += d.size
        lo, hi = slice(off[L], off[L + 1]), slice(off[L + 1], off[L + 2])
        up, down = (-1j * F, -1j * F) if gauge == "l" else (-F, F)
        want[lo] += up * (d @ x[hi])
        want[hi] += down * (d.T @ x[lo])
        size[lo] += F * (np.abs(d) @ np.abs(x[hi]))
        size[hi] += F * (np.abs(d.T) @ np.abs(x[lo]))
    with mpc_tdse.Context.from_system(s) as ctx:
        got = ctx.rhs(F, x)
    bound = 2 * (2 * max(n) + 4) * np.finfo(float).eps * size
    assert np.all(np.abs(got - want) <= bound)
