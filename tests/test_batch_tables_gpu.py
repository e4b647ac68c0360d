"""A batch whose instances bring their own FR tables: every instance runs its own scheme, as it does
alone, and instances whose face rows are not those of GLL points are refused."""
from __future__ import annotations

import numpy as np
import pytest

import sgnb
from cases import bump_case
from conftest import bits_equal

pytestmark = pytest.mark.gpu


def other_correction(scale):
    """Tables with scaled correction functions, which keep the reflection symmetry."""
    t = sgnb.fr_tables()
    t["gLp"] = scale * t["gLp"]
    t["gRp"] = -t["gLp"][::-1]
    return t


@pytest.mark.parametrize("precision", [sgnb.FP64_FAST, sgnb.MIXED])
@pytest.mark.parametrize("first", [1.0, 0.8])
def test_each_instance_has_its_own_tables(precision, first):
    kws = []
    for (Nx, Ny), scale in (((7, 5), first), ((12, 4), 0.9), ((6, 9), first)):
        kw, U = bump_case(1, Nx=Nx, Ny=Ny, Lx=1.25 * Nx, Ly=8.0 / 6.0 * Ny)
        kws.append((dict(kw, tables=other_correction(scale)), U))
    dt, steps = 1e-3, 4
    with sgnb.SGNBatch([kw for kw, _ in kws], precision=precision) as b:
        for i, (_, U) in enumerate(kws):
            b[i].upload(U)
        stats = b.integrate_steps(dt, steps)
        launches = 0
        for i, (kw, U) in enumerate(kws):
            with sgnb.SGN2DB200(precision=precision, **kw) as d:
                d.upload(U)
                st = d.integrate_steps(0.0, dt, steps)
                assert bits_equal(b[i].download(), d.download())
            assert (stats[i].accepted, stats[i].rejected, stats[i].dtLast) == (st.accepted, st.rejected, st.dtLast)
            launches += st.kernel_launches
        assert all(s.kernel_launches == launches for s in stats)


def test_interpolating_face_rows_are_refused():
    t = sgnb.fr_tables()
    t["lL"] = np.array([1.0, 1e-3, 0.0, 0.0, 0.0])
    kw = dict(Nx=6, Ny=4, Lx=7.5, Ly=5.0, c=9.0, bathy_kind=sgnb.BATHY_NONE)
    with pytest.raises(sgnb.SgnbError, match="GLL"):
        sgnb.SGNBatch([dict(kw), dict(kw, tables=t)])
