"""The mixed mode's third and end-point stages: the candidate state leaves with the third stage.

One frozen BS3(2) step against the same combination of the device's own right-hand sides, in
64 bits on the host with the stage derivatives rounded to 32 bits. A stage kernel may contract a
right-hand side differently from the right-hand-side kernel; both are within 2e-5 per field of
the exact one (the bound of the mixed right-hand side against the oracle), so the step's result
may differ by 2 * 2e-5 * dt * max|k| per field (the weights of k1..k3 sum to one; the stages'
own differences enter with another factor dt)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
import sgnb
from cases import bump_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Ny", [(2, 2), (7, 3), (8, 4), (9, 5), (16, 8), (17, 9)])
@pytest.mark.parametrize("bc", [0, 1])
def test_step_from_right_hand_sides(Nx, Ny, bc):
    kw, U = bump_case(bc, Nx=Nx, Ny=Ny, Lx=1.25 * Nx, Ly=8.0 / 6.0 * Ny)
    dt = 0.4 * O.Oracle(**kw).cfl_time_step(U, 0.5)
    with sgnb.SGN2DB200(precision=sgnb.MIXED, **kw) as d:
        k = []
        for coef in (0.0, 0.5, 0.75):
            y = U + (coef * dt) * k[-1] if k else U
            k.append(d.rhs(y).astype(np.float32).astype(np.float64))
        want = U + dt * (2.0 / 9.0 * k[0] + 1.0 / 3.0 * k[1] + 4.0 / 9.0 * k[2])
        d.upload(U)
        d.bs3_steps(0.0, np.full(1, dt))
        got = d.download()
    err = np.abs(got - want).reshape(5, -1).max(axis=1)
    kmax = np.max([np.abs(x).reshape(5, -1).max(axis=1) for x in k], axis=0)
    assert np.all(err <= 4e-5 * dt * kmax), (err, dt * kmax)


def test_batch_takes_the_same_steps():
    """Mixed batch and single instances: the same steps from the same states."""
    kws, states = [], []
    for Nx, Ny in ((8, 4), (13, 6), (16, 8)):
        kw, U = bump_case(1, Nx=Nx, Ny=Ny, Lx=1.25 * Nx, Ly=8.0 / 6.0 * Ny)
        kws.append(kw)
        states.append(U)
    b = sgnb.SGNBatch(kws, precision=sgnb.MIXED)
    dt0 = np.zeros(len(kws))
    for i, U in enumerate(states):
        b[i].upload(U)
        dt0[i] = 0.4 * b[i].cfl_time_step(0.5)
    st = b.integrate_steps(dt0, 2)
    for i, (kw, U) in enumerate(zip(kws, states)):
        with sgnb.SGN2DB200(precision=sgnb.MIXED, **kw) as d:
            d.upload(U)
            s1 = d.integrate_steps(0.0, dt0[i], 2)
            a, c = d.download(), b[i].download()
        assert (st[i].accepted, st[i].rejected) == (s1.accepted, s1.rejected)
        # two steps of at most five times dt0, each within the bound above of exact ones
        kmax = np.abs(a - U).reshape(5, -1).max(axis=1) + 1e-3
        assert np.all(np.abs(a - c).reshape(5, -1).max(axis=1) <= 8e-5 * kmax)
