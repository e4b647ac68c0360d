"""The exact mode's kernels with the registers of two and of three CTAs per SM (up to 296 tiles of
6 x 4 elements, and more): the CPU solver's bits on both sides, also for slabs."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as O
import sgnb
from cases import bump_case
from conftest import bits_equal
from sgnb.slabs import SlabSolver

pytestmark = pytest.mark.gpu


def case(Nx, Ny, bc):
    return bump_case(bc, Nx=Nx, Ny=Ny, Lx=1.25 * Nx, Ly=8.0 / 6.0 * Ny)


@pytest.mark.parametrize("Nx,Ny", [(108, 64), (114, 64), (111, 61), (131, 61)])  # 288, 304, 304, 352 tiles
@pytest.mark.parametrize("bc", [0, 1])
def test_whole_mesh(Nx, Ny, bc):
    kw, U = case(Nx, Ny, bc)
    ref = O.Oracle(**kw)
    dt = 0.4 * ref.cfl_time_step(U, 0.5)
    u = U
    for k in range(2):
        u = ref.bs3_step(u, k * dt, dt)
    v = ref.rk4_step(U, 0.0, dt)
    with sgnb.SGN2DB200(precision=sgnb.FP64_EXACT, **kw) as d:
        assert bits_equal(d.rhs(U), ref.rhs(U))
        d.upload(U)
        d.bs3_steps(0.0, np.full(2, dt))
        assert bits_equal(d.download(), u)
        d.upload(U)
        d.rk4_steps(0.0, [dt])
        assert bits_equal(d.download(), v)


@pytest.mark.parametrize("Nx", [200, 231])  # slabs of 100 (255 tiles), of 115 and 116 columns (300)
def test_slabs(Nx):
    kw, U = case(Nx, 59, 1)
    ref = O.Oracle(**kw)
    dt = 0.4 * ref.cfl_time_step(U, 0.5)
    u = U
    for k in range(2):
        u = ref.bs3_step(u, k * dt, dt)
    with SlabSolver(dict(kw, precision=sgnb.FP64_EXACT), nslabs=2) as s:
        assert bits_equal(s.rhs(U), ref.rhs(U))
        s.upload(U)
        s.integrate_steps(0.0, dt, 2, dts=np.full(2, dt))
        assert bits_equal(s.download(), u)
