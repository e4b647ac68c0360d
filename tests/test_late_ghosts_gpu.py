"""A whole-mesh context that is given ghosts after its creation runs the kernels with slab edges:
with its own wrapped edge nodes as ghosts it gives the bits of the periodic mesh, and without them
again as well."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import sgnb
from cases import bump_case
from conftest import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [sgnb.FP64_EXACT, sgnb.FP64_FAST])
@pytest.mark.parametrize("manning", [0.0, 0.03])
@pytest.mark.parametrize("Nx,Ny", [(6, 4), (9, 5)])
def test_own_edges_as_ghosts(precision, manning, Nx, Ny):
    import torch

    kw, U = bump_case(0, Nx=Nx, Ny=Ny, Lx=1.25 * Nx, Ly=8.0 / 6.0 * Ny)
    kw.update(nManning=manning, bathy_kind=sgnb.BATHY_CONST, bathy_par=(1.0,))
    ptr = lambda t: C.cast(C.c_void_p(t.data_ptr() if t is not None else None), sgnb._dp)
    with sgnb.SGN2DB200(precision=precision, **kw) as d:
        d.upload(U)
        want = d.rhs_once()
        first, last = (torch.zeros(25 * Ny, dtype=torch.float64, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        sgnb._check(sgnb.lib().sgnb_slab_pack(d._h, 0, None, ptr(first), ptr(last), None), d._h)
        for left, right in ((last, first), (last, None), (None, first), (None, None)):
            sgnb._check(sgnb.lib().sgnb_set_ghosts(d._h, ptr(left), ptr(right)), d._h)
            assert bits_equal(d.rhs_once(), want)
