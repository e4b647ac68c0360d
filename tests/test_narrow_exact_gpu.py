"""The exact mode on long meshes a few elements wide, where its tiles are 2 x 12 elements: the CPU
solver's bits at the tiles' edges, on every way their rows are loaded, with friction and with ghosts."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle as O
import sgnb
from cases import bump_case
from conftest import bits_equal, rel_per_field

pytestmark = pytest.mark.gpu

# more than one wave of 6 x 4 tiles; Ny 0, 1, 2 and 11 more than a multiple of 12
SIZES = [(2, 1784), (3, 1789), (7, 900), (8, 889), (8, 911), (13, 614), (14, 600)]


def case(Nx, Ny, bc):
    return bump_case(bc, Nx=Nx, Ny=Ny, Lx=1.25 * Nx, Ly=8.0 / 6.0 * Ny)


@pytest.mark.parametrize("Nx,Ny", SIZES)
@pytest.mark.parametrize("bc", [0, 1])
@pytest.mark.parametrize("tma", ["1", "0"])
def test_bits_of_the_cpu(Nx, Ny, bc, tma, monkeypatch):
    import torch

    monkeypatch.setenv("SGNB_TMA", tma)
    kw, U = case(Nx, Ny, bc)
    ref = O.Oracle(**kw)
    R = ref.rhs(U)
    dt = 0.4 * ref.cfl_time_step(U, 0.5)
    u = U
    for k in range(3):
        u = ref.bs3_step(u, k * dt, dt)
    with sgnb.SGN2DB200(precision=sgnb.FP64_EXACT, **kw) as d:
        assert bits_equal(d.rhs(U), R)
        for off in (0, 1):  # 16-byte and 8-byte aligned
            a = torch.zeros(U.size + 2, dtype=torch.float64, device="cuda")
            b = torch.zeros_like(a)
            a[off:off + U.size] = torch.from_numpy(U).cuda()
            torch.cuda.synchronize()
            d.rhs_device(a.data_ptr() + 8 * off, b.data_ptr() + 8 * off, torch.cuda.current_stream().cuda_stream)
            assert bits_equal(b[off:off + U.size].cpu().numpy(), R)
            assert float(b[:off].abs().sum() + b[off + U.size:].abs().sum()) == 0.0
        d.upload(U)
        d.bs3_steps(0.0, np.full(3, dt))
        assert bits_equal(d.download(), u)
        d.upload(U)
        st = d.integrate_steps(0.0, dt, 4)
        uo, so, _ = ref.integrate_adaptive(U, 0.0, 1e300, dt, stop_after=4)
        assert (st.accepted, st.rejected) == (so["accepted"], so["rejected"])
        assert rel_per_field(d.download(), uo) < 1e-12  # (the error sum's order differs)


@pytest.mark.parametrize("Nx,Ny", [(7, 901), (8, 900)])
def test_friction_and_ghosts(Nx, Ny):
    """Friction within the cube root's last bits of the CPU; a mesh's own edges as its ghosts give the
    bits of the periodic one."""
    import torch

    kw, U = case(Nx, Ny, 0)
    kw.update(nManning=0.03, bathy_kind=sgnb.BATHY_CONST, bathy_par=(1.0,))
    ptr = lambda t: C.cast(C.c_void_p(t.data_ptr() if t is not None else None), sgnb._dp)
    with sgnb.SGN2DB200(precision=sgnb.FP64_EXACT, **kw) as d:
        d.upload(U)
        want = d.rhs_once()
        assert rel_per_field(want, O.Oracle(**kw).rhs(U)) < 1e-14
        first, last = (torch.zeros(25 * Ny, dtype=torch.float64, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        sgnb._check(sgnb.lib().sgnb_slab_pack(d._h, 0, None, ptr(first), ptr(last), None), d._h)
        for left, right in ((last, first), (last, None), (None, first), (None, None)):
            sgnb._check(sgnb.lib().sgnb_set_ghosts(d._h, ptr(left), ptr(right)), d._h)
            assert bits_equal(d.rhs_once(), want)
