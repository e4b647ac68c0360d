"""The fast mode's rounding, against extended precision: its derivatives act on differences along
a line, and its reciprocal and square root round like the IEEE operations."""
from __future__ import annotations

import numpy as np
import pytest

import sgnb
from test_fast_math_gpu import fast_math

pytestmark = pytest.mark.gpu

LD = np.longdouble


def tables():
    """Differentiation matrix of the five GLL points and the derivatives of the two g_DG
    correction functions."""
    s = np.sqrt(LD(3) / LD(7))
    x = np.array([-1, -s, 0, s, 1], dtype=LD)
    w = [1 / np.prod([x[j] - x[k] for k in range(5) if k != j]) for j in range(5)]
    D = np.array([[w[j] / w[i] / (x[i] - x[j]) if i != j else LD(0) for j in range(5)] for i in range(5)])
    D[np.arange(5), np.arange(5)] = -D.sum(axis=1)
    d4, d5 = (140 * x**3 - 60 * x) / 8, (315 * x**4 - 210 * x**2 + 15) / 8
    return D, (d4 - d5) / 2, (d4 + d5) / 2


def mass_rhs(U, hx, hy, g, c):
    """dh/dt on a periodic mesh, U = [5, Ny, Nx, 5 (y node), 5 (x node)]."""
    D, gL, gR = tables()
    U = U.astype(LD)
    out = np.zeros_like(U[0])
    for d, J in ((0, LD(hx) / 2), (1, LD(hy) / 2)):
        V = U if d == 0 else np.swapaxes(U, 3, 4)  # nodes of a line last
        lo, hi = V[..., 0], V[..., 4]
        ax = 2 - d
        nlo, nhi = np.roll(hi, 1, ax), np.roll(lo, -1, ax)
        speed = lambda a: np.abs(a[1 + d] / a[0]) + np.sqrt(LD(g) * a[0] + a[4] / a[0] + LD(c) ** 2)
        jl = (nlo[1 + d] - lo[1 + d] + np.maximum(speed(lo), speed(nlo)) * (nlo[0] - lo[0])) / 2
        jh = (nhi[1 + d] - hi[1 + d] - np.maximum(speed(hi), speed(nhi)) * (nhi[0] - hi[0])) / 2
        r = np.einsum("mk,...k->...m", D, V[1 + d]) + jl[..., None] * gL + jh[..., None] * gR
        out -= (r if d == 0 else np.swapaxes(r, 2, 3)) / J
    return out


@pytest.mark.parametrize("Nx,Ny", [(8, 8), (13, 6), (7, 9)])
def test_derivative_of_a_small_variation(Nx, Ny):
    """Discharges 1 + 1e-3 sin: a value of dh/dt takes some 12 roundings per direction, each at
    most 2^-53 of the sum of |D| (16.3 at an end node) times the variation over a line; relative to
    the largest derivative that is below 24 * 16.3 * 2^-53 = 4.3e-14. Rounding at the size of the
    discharge itself would cost 1e-12."""
    hx = hy = 0.5
    kx, ky = 2 * np.pi / (Nx * hx), 2 * np.pi / (Ny * hy)
    with sgnb.SGN2DB200(precision=sgnb.FP64_FAST, Nx=Nx, Ny=Ny, Lx=Nx * hx, Ly=Ny * hy, c=9.0,
                        bathy_kind=sgnb.BATHY_CONST, bathy_par=(1.0,)) as d:
        x, y = d.node_coords()
        s = np.sin(kx * x + 0.3) + np.cos(ky * y + 0.2)
        U = np.concatenate([1.0 + 1e-3 * s, 1.0 + 1e-3 * np.sin(kx * x), 1.0 + 1e-3 * np.cos(ky * y),
                            0.01 * s, 0.01 * np.sin(ky * y)])
        got = d.rhs(U)[:U.size // 5]
    want = mass_rhs(U.reshape(5, Ny, Nx, 5, 5), hx, hy, 9.81, 9.0).reshape(-1)
    assert float(np.abs(got - want).max() / np.abs(want).max()) < 4.3e-14


@pytest.mark.parametrize("fn", [0, 1])
def test_reciprocal_and_root_round_once(fn):
    """Two Newton steps (the root: a series step and one Newton step) leave a relative error of
    order 2^-70 before the last rounding: 0.5 ulp, and 1e-4 for that error."""
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.uniform(1e-3, 1e2, 1 << 20), 10.0 ** rng.uniform(-300, 300, 1 << 18)])
    _, yd = fast_math(fn, x)
    y = yd.cpu().numpy()
    want = 1 / x.astype(LD) if fn == 0 else np.sqrt(x.astype(LD))
    assert float((np.abs(y - want) / np.spacing(y)).max()) < 0.5001
