"""A purely relative tolerance (atol = 0): the fast mode looks at each scale by itself, and its
attempts are the exact mode's."""
from __future__ import annotations

import numpy as np
import pytest

import sgnb
from cases import bump_case

pytestmark = pytest.mark.gpu


def case(Nx, Ny):
    """No field passes through zero: a relative tolerance alone means nothing there."""
    kw, U = bump_case(0, Nx=Nx, Ny=Ny, Lx=1.25 * Nx, Ly=8.0 / 6.0 * Ny)
    U.reshape(5, -1)[1:] += 1.0
    return kw, U


@pytest.mark.parametrize("Nx,Ny", [(6, 4), (13, 9)])
def test_same_attempts_as_exact(Nx, Ny):
    kw, U = case(Nx, Ny)
    opt = sgnb.AdaptiveRKOptions(atol=0.0, rtol=1e-4)
    logs = []
    for precision in (sgnb.FP64_EXACT, sgnb.FP64_FAST):
        with sgnb.SGN2DB200(precision=precision, **kw) as d:
            d.upload(U)
            st = d.integrate_steps(0.0, 5e-3, 3, opt)
            logs.append((st.accepted, st.rejected, np.asarray(d.attempt_log())[0, 2]))
    assert logs[0][:2] == logs[1][:2]
    # the error is the difference of two states of order 1, which the modes round apart by some tens
    # of 2^-53; it is itself above 1e-8 here (a norm above 1e-4 of the tolerance 1e-4)
    assert logs[0][2] > 1e-4
    assert abs(logs[1][2] - logs[0][2]) < 1e-6 * logs[0][2]
