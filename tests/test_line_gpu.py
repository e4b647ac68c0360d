"""The fast mode's line kernels at the edges of their tiles (rows of 6 elements, 4 rows) and on
every way their rows are loaded and stored.

Meshes keep the element size of bump_case (1.25 x 1.33), where one rounding of the hydrostatic
flux, times the largest entries of D over J, is 1e-14 of a field's largest right-hand side; with
some tens of them in a value, the fast mode and the CPU agree within 5e-13 (1e-12 after three
steps)."""
from __future__ import annotations

import os

import numpy as np
import pytest

import oracle as O
import sgnb
from cases import bump_case
from conftest import bits_equal, rel_per_field

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (3, 2), (5, 3), (6, 4), (7, 4), (6, 5), (11, 7), (12, 8), (13, 9), (18, 6), (25, 4)]


def case(Nx, Ny, bc):
    return bump_case(bc, Nx=Nx, Ny=Ny, Lx=1.25 * Nx, Ly=8.0 / 6.0 * Ny)


@pytest.mark.parametrize("Nx,Ny", SIZES)
@pytest.mark.parametrize("bc", [0, 1])
def test_rhs_and_steps(Nx, Ny, bc):
    kw, U = case(Nx, Ny, bc)
    ref = O.Oracle(**kw)
    dt = 0.4 * ref.cfl_time_step(U, 0.5)
    u = U
    for k in range(3):
        u = ref.bs3_step(u, k * dt, dt)
    with sgnb.SGN2DB200(precision=sgnb.FP64_FAST, **kw) as d:
        assert rel_per_field(d.rhs(U), ref.rhs(U)) < 5e-13
        d.upload(U)
        d.bs3_steps(0.0, np.full(3, dt))
        assert rel_per_field(d.download(), u) < 1e-12


@pytest.mark.parametrize("Nx,Ny", [(6, 4), (8, 5), (14, 7)])
def test_row_copies_bitwise(Nx, Ny):
    """Bulk row copies (Nx even), per-value copies (SGNB_TMA=0) and buffers that are only
    8-byte aligned give the same bits."""
    import torch

    kw, U = case(Nx, Ny, 1)
    out = []
    for tma in ("1", "0"):
        old = os.environ.get("SGNB_TMA")
        os.environ["SGNB_TMA"] = tma
        try:
            with sgnb.SGN2DB200(precision=sgnb.FP64_FAST, **kw) as d:
                out.append(d.rhs(U))
                for off in (0, 1):
                    a = torch.zeros(U.size + 2, dtype=torch.float64, device="cuda")
                    b = torch.zeros_like(a)
                    a[off:off + U.size] = torch.from_numpy(U).cuda()
                    torch.cuda.synchronize()
                    d.rhs_device(a.data_ptr() + 8 * off, b.data_ptr() + 8 * off,
                                 torch.cuda.current_stream().cuda_stream)
                    out.append(b[off:off + U.size].cpu().numpy())
                    assert float(b[:off].abs().sum() + b[off + U.size:].abs().sum()) == 0.0
        finally:
            if old is None:
                del os.environ["SGNB_TMA"]
            else:
                os.environ["SGNB_TMA"] = old
    for x in out[1:]:
        assert bits_equal(x, out[0])


def test_tables_without_reflection_symmetry():
    """FR tables that the split derivatives cannot take run on the kernels that take any."""
    kw, U = case(9, 5, 1)
    t = sgnb.fr_tables()
    t["gLp"] = t["gLp"] * np.array([1.0, 1.01, 1.0, 0.99, 1.0])
    with sgnb.SGN2DB200(precision=sgnb.FP64_FAST, tables=t, **kw) as f, \
            sgnb.SGN2DB200(precision=sgnb.FP64_EXACT, tables=t, **kw) as e:
        assert bits_equal(f.rhs(U), e.rhs(U))
    with sgnb.SGNBatch([dict(kw, tables=t), dict(kw, tables=t)]) as b, \
            sgnb.SGN2DB200(precision=sgnb.FP64_FAST, tables=t, **kw) as f:
        dt = 1e-3
        for i in range(2):
            b[i].upload(U)
        st = b.integrate_steps(dt, 3)
        f.upload(U)
        sf = f.integrate_steps(0.0, dt, 3)
        assert [(s.accepted, s.rejected) for s in st] == [(sf.accepted, sf.rejected)] * 2
        assert bits_equal(b[1].download(), f.download())
