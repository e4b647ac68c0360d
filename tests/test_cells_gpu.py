"""The adjoint's bathymetry from element means on the device: its statics have the bits of the
host set-up, and the gradient of the means is their transpose."""
from __future__ import annotations

import numpy as np
import pytest

import sgnb
from sgnb.adjoint import SGNAdjoint

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (3, 2), (2, 5), (9, 5), (17, 3)]  # wraps onto itself, partial and whole tiles


def problem(Nx, Ny, bc):
    rng = np.random.default_rng(7)
    means = 1.0 + 0.1 * rng.standard_normal(Nx * Ny)
    kw = dict(Nx=Nx, Ny=Ny, Lx=1.1 * Nx, Ly=0.9 * Ny, c=9.0, bc_x=bc, bc_y=bc,
              bathy_kind=sgnb.BATHY_CELLS,
              bathy_par=np.concatenate([[Nx, Ny, 1.1 * Nx, 0.9 * Ny], means]))
    eta0 = 0.02 * rng.standard_normal(25 * Nx * Ny)
    return kw, means, eta0


@pytest.mark.parametrize("Nx,Ny", SIZES)
@pytest.mark.parametrize("bc", [0, 1])
def test_statics_bitwise(Nx, Ny, bc):
    """A context whose statics the forward run replaced gives the right-hand side of one that
    was created with them, bit for bit (nodal depths, gradients, face depths)."""
    kw, means, eta0 = problem(Nx, Ny, bc)
    U = np.concatenate([1.2 + eta0] + [0.1 * np.roll(eta0, k) for k in range(1, 5)])
    other = dict(kw, bathy_par=np.concatenate([kw["bathy_par"][:4], np.full(Nx * Ny, 2.0)]))
    with sgnb.SGN2DB200(precision=sgnb.FP64_EXACT, **kw) as ref, \
            sgnb.SGN2DB200(precision=sgnb.FP64_EXACT, **other) as dev:
        with SGNAdjoint(dev, [1e-5], [0], 1) as adj:
            adj.forward(means, eta0)
            a, b = dev.rhs(U), ref.rhs(U)
    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("Nx,Ny", SIZES)
@pytest.mark.parametrize("bc", [0, 1])
def test_gradient_of_means(Nx, Ny, bc):
    """<grad, d> against central differences of the forward run (two gauges share a node). The
    difference step 1e-4 leaves a truncation error of order 1e-8 and a rounding error of order
    1e-12 relative to the derivative: within 1e-6."""
    kw, means, eta0 = problem(Nx, Ny, bc)
    rng = np.random.default_rng(11)
    Nd = 25 * Nx * Ny
    gauges = np.array([0, Nd // 2, Nd // 2, Nd - 1, Nd // 3], dtype=np.int64)
    with sgnb.SGN2DB200(precision=sgnb.FP64_FAST, **kw) as dev:
        with SGNAdjoint(dev, np.full(4, 2e-3), gauges, 3) as adj:
            bar = rng.standard_normal((4, gauges.size))
            adj.forward(means, eta0)
            gm, _ = adj.vjp(bar)
            d = rng.standard_normal(means.size)
            h = 1e-4
            num = ((adj.forward(means + h * d, eta0) - adj.forward(means - h * d, eta0)) * bar).sum() / (2 * h)
    scale = np.linalg.norm(gm) * np.linalg.norm(d)
    assert abs(gm @ d - num) <= 1e-6 * scale
