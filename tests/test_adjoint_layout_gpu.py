"""The adjoint's buffers are aligned for row copies whatever the numbers of steps and gauges."""
from __future__ import annotations

import time

import numpy as np
import pytest

import sgnb
from conftest import bits_equal
from sgnb.adjoint import SGNAdjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [40, 41])
def test_one_gauge_more(steps):
    """One gauge more changes no record and costs no time to speak of (per-value copies of the
    states made the forward run 1.15 times as long)."""
    Nx, Ny = 256, 128
    kw = dict(Nx=Nx, Ny=Ny, Lx=20.0, Ly=10.0, c=9.0, bc_x=1, bc_y=1, bathy_kind=sgnb.BATHY_CELLS,
              bathy_par=np.concatenate([[Nx, Ny, 20.0, 10.0], np.ones(Nx * Ny)]))
    rng = np.random.default_rng(5)
    eta0, means = 0.01 * rng.standard_normal(25 * Nx * Ny), np.ones(Nx * Ny)
    gauges = rng.choice(25 * Nx * Ny, 17, replace=False).astype(np.int64)
    with sgnb.SGN2DB200(precision=sgnb.FP64_FAST, **kw) as d:
        adj = [SGNAdjoint(d, np.full(steps, 1e-6), gauges[:n], 8) for n in (16, 17)]
        best, rec = [np.inf, np.inf], [None, None]
        for _ in range(25):
            for i, a in enumerate(adj):
                t0 = time.perf_counter()
                rec[i] = a.forward(means, eta0)
                best[i] = min(best[i], time.perf_counter() - t0)
        for a in adj:
            a.close()
    assert bits_equal(rec[0], rec[1][:, :16])
    assert max(best) < 1.1 * min(best)  # the least of 25 runs each, taken in turn
