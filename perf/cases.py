"""What a user of the solver has it do, as cases that can be timed and checked.

A case is one call (or one short call sequence) through the Python front end ``sgnb``, on
inputs made from a seed. The listed cases cover the entry points that a program spends its
time in, each in the arithmetic modes and boundary conditions that go with it, from the
smallest mesh of the configurations (128 x 64 elements, the launch-bound end) to the
benchmark's 2048 x 1024 (52 M nodes); odd meshes, whose edge tiles are partial, are among
them. ``draw`` gives further cases of the same ranges.

``exact`` is a plain torch implementation of the same discretisation in 64-bit floating
point (flux reconstruction, P = 4, on the five Gauss-Lobatto-Legendre points), written
from the equations: whole-array operations, no kernel of this repository.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "sgn-hyperbolic-gpu_b200"))

import sgnb  # noqa: E402
from sgnb.adjoint import SGNAdjoint  # noqa: E402
from sgnb.slabs import SlabSolver  # noqa: E402

DEV = "cuda:0"
G, GAMMA, ALPHA = 9.81, 1.5, 3.0
PRECISION = {"exact": sgnb.FP64_EXACT, "fast": sgnb.FP64_FAST, "mixed": sgnb.MIXED}


# ---------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------
def listed():
    return [
        # one right-hand side on device arrays, as a program with its own integrator calls it;
        # configuration 1's mesh: 1 M values, a launch-bound call
        dict(name="rhs_small", kind="rhs", mode="fast", nx=128, ny=64, bed="flat", wall=False,
             manning=0.0),
        # the drop-in default (bit-identical to the CPU solver) on a mesh with partial tiles
        dict(name="rhs_exact_odd", kind="rhs", mode="exact", nx=301, ny=173, bed="bump", wall=True,
             manning=0.0),
        # a coastal run's right-hand side with bottom friction, partial tiles
        dict(name="rhs_friction_odd", kind="rhs", mode="fast", nx=517, ny=259, bed="shoal",
             wall=True, manning=0.02),
        # a large right-hand side over the shoal
        dict(name="rhs_large", kind="rhs", mode="fast", nx=1024, ny=512, bed="shoal", wall=True,
             manning=0.0),
        # configuration 1: the adaptive loop on the small periodic mesh
        dict(name="steps_small", kind="steps", mode="fast", nx=128, ny=64, bed="flat", wall=False,
             manning=0.0, steps=20),
        # the drop-in default through its adaptive loop, partial tiles
        dict(name="steps_exact", kind="steps", mode="exact", nx=250, ny=131, bed="bump", wall=True,
             manning=0.0, steps=8),
        # configuration 2, the benchmark: waves over the elliptic shoal at full size
        dict(name="steps_large", kind="steps", mode="fast", nx=2048, ny=1024, bed="shoal",
             wall=True, manning=0.0, steps=4),
        # the mixed-precision loop on a large mesh
        dict(name="steps_mixed", kind="steps", mode="mixed", nx=1024, ny=512, bed="shoal",
             wall=True, manning=0.0, steps=5),
        # configuration 4: a sweep of uneven instances in one batch, FP64 and mixed
        dict(name="batch_fast", kind="batch", mode="fast", n=24, sizes=4, steps=5),
        dict(name="batch_mixed", kind="batch", mode="mixed", n=24, sizes=14, steps=5),
        # configuration 5: gauge records of a frozen trajectory and their gradient
        dict(name="adjoint", kind="adjoint", mode="fast", nx=256, ny=128, steps=12, every=5,
             gauges=16),
        # one mesh split into slabs (all on this device), the multi-GPU solver's path
        dict(name="slabs", kind="slabs", mode="fast", nx=1024, ny=512, bed="shoal", wall=True,
             manning=0.0, steps=4, slabs=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, lo, hi):
    """Nx in [lo, hi] spread over its logarithm, Ny about half of it; half of the meshes
    are whole numbers of 8 x 4 element tiles, the others take any size."""
    nx = _log_int(rng, lo, hi)
    ny = max(16, min(int(nx * rng.uniform(0.35, 0.65)), hi // 2))
    if rng.random() < 0.5:
        nx, ny = max(8, nx // 8 * 8), max(4, ny // 4 * 4)
    return nx, ny


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "rhs", "steps", "steps", "steps", "steps", "batch", "batch",
                       "adjoint", "slabs"])
    bed = rng.choice(["flat", "bump", "shoal"])
    if kind == "rhs":
        mode = rng.choice(["fast", "fast", "exact"])
        nx, ny = _mesh(rng, 96, 1200)
        return dict(kind=kind, mode=mode, nx=nx, ny=ny, bed=bed, wall=rng.random() < 0.6,
                    manning=rng.choice([0.0, 0.0, 0.025]) if bed != "flat" else 0.0)
    if kind == "steps":
        mode = rng.choice(["fast", "fast", "exact", "mixed"])
        nx, ny = _mesh(rng, 96, 1400)
        return dict(kind=kind, mode=mode, nx=nx, ny=ny, bed=bed, wall=rng.random() < 0.6,
                    manning=0.0, steps=rng.randint(3, 10))
    if kind == "batch":
        return dict(kind=kind, mode=rng.choice(["fast", "mixed"]), n=rng.randint(6, 24),
                    sizes=rng.randint(100, 10000), steps=rng.randint(3, 6))
    if kind == "adjoint":
        nx, ny = _mesh(rng, 96, 280)
        return dict(kind=kind, mode="fast", nx=nx, ny=ny, steps=rng.randint(6, 12),
                    every=rng.randint(2, 6), gauges=rng.randint(4, 20))
    nx, ny = _mesh(rng, 256, 1100)
    return dict(kind=kind, mode="fast", nx=nx, ny=ny, bed=bed, wall=rng.random() < 0.6,
                manning=0.0, steps=rng.randint(3, 6), slabs=rng.randint(2, 5))


# ---------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------
_BEDS = {"flat": (sgnb.BATHY_CONST, (1.0,)),
         "bump": (sgnb.BATHY_GAUSS, (1.0, 0.4, 11.0, 5.0, 6.0)),
         "shoal": (sgnb.BATHY_SHOAL, (0.45, 0.15, 20.0, 10.0, 4.0, 3.0))}


def _solver_args(case):
    """Solver arguments: the flat and bump beds on configuration 1's 20 x 10 domain, the
    shoal on configuration 2's 40 x 20 one."""
    kind, par = _BEDS[case["bed"]]
    Lx, Ly = (40.0, 20.0) if case["bed"] == "shoal" else (20.0, 10.0)
    b = int(case["wall"])
    return dict(P=4, Nx=case["nx"], Ny=case["ny"], Lx=Lx, Ly=Ly, g=G, c=ALPHA * math.sqrt(G * par[0]),
                gamma=GAMMA, nManning=case["manning"], bc_x=b, bc_y=b, bathy_kind=kind, bathy_par=par)


def _sweep_args(case):
    """The sweep's instances: sizes, dispersion and shoal crest drawn as configuration 4
    draws them."""
    rng = np.random.default_rng(case["sizes"])
    out = []
    for _ in range(case["n"]):
        nx, ny = int(rng.integers(64, 513)), int(rng.integers(32, 257))
        alpha, crest = float(rng.uniform(1.5, 6.0)), float(rng.uniform(0.3, 0.9))
        out.append(dict(P=4, Nx=nx, Ny=ny, Lx=20.0, Ly=10.0, g=G, c=alpha * math.sqrt(G), gamma=GAMMA,
                        bc_x=1, bc_y=1, bathy_kind=sgnb.BATHY_SHOAL,
                        bathy_par=(1.0, crest, 12.0, 5.0, 4.0, 3.0)))
    return out


_S = math.sqrt(3.0 / 7.0)
_XI = (-1.0, -_S, 0.0, _S, 1.0)


def _axis(n, L):
    """Node coordinates of one direction, [n, 5]."""
    h = L / n
    e = torch.arange(n, device=DEV, dtype=torch.float64)
    xi = torch.tensor(_XI, device=DEV, dtype=torch.float64)
    return e[:, None] * h + 0.5 * h * (xi[None, :] + 1.0)


def _coords(kw):
    """x and y of every node, broadcastable to [Ny, Nx, 5 (y node), 5 (x node)]."""
    x = _axis(kw["Nx"], kw["Lx"])[None, :, None, :]
    y = _axis(kw["Ny"], kw["Ly"])[:, None, :, None]
    return x, y


def _waves(rng, x, y, Lx, Ly, n, amp, periodic):
    """Sum of n sine waves with random phase and amplitude; whole wave numbers of the
    domain when it is periodic."""
    out = torch.zeros(torch.broadcast_shapes(x.shape, y.shape), dtype=torch.float64, device=DEV)
    for _ in range(n):
        a, ph = amp * rng.uniform(0.25, 1.0), rng.uniform(0.0, 2 * math.pi)
        lam, th = rng.uniform(2.0, 6.0), rng.uniform(0.0, 2 * math.pi)
        kx, ky = 2 * math.pi / lam * math.cos(th), 2 * math.pi / lam * math.sin(th)
        if periodic:
            kx = 2 * math.pi / Lx * round(kx * Lx / (2 * math.pi))
            ky = 2 * math.pi / Ly * round(ky * Ly / (2 * math.pi))
        out += a * torch.sin(kx * x + ky * y + ph)
    return out


def _state(kw, rng):
    """A moving sea: surface waves over the bed and small smooth velocities (vanishing at
    walls) and non-hydrostatic fields; [5, Ny, Nx, 5, 5]."""
    x, y = _coords(kw)
    H = _depth(kw, x, y)
    per = kw["bc_x"] == 0
    Lx, Ly = kw["Lx"], kw["Ly"]
    U = torch.empty((5, kw["Ny"], kw["Nx"], 5, 5), dtype=torch.float64, device=DEV)
    U[0] = H + _waves(rng, x, y, Lx, Ly, 4, 0.01, per)
    at_wall = (1.0, 1.0) if per else (torch.sin(math.pi / Lx * x), torch.sin(math.pi / Ly * y))
    for v, amp in ((1, 0.03), (2, 0.03), (3, 0.01), (4, 0.01)):
        U[v] = U[0] * _waves(rng, x, y, Lx, Ly, 2, amp, per)
        if v < 3:
            U[v] *= at_wall[v - 1]
    return U


def _adjoint_inputs(case, seed):
    """Configuration 5: noisy element means of a shoal, a hump of the free surface, gauges
    and the cotangent of their records; the frozen steps stay below the stability limit."""
    rng = np.random.default_rng(seed)
    nx, ny, Lx, Ly = case["nx"], case["ny"], 20.0, 10.0
    X, Y = np.meshgrid((np.arange(nx) + 0.5) * Lx / nx, (np.arange(ny) + 0.5) * Ly / ny)
    q = np.clip(1.0 - ((X - 12.0) / 4.0) ** 2 - ((Y - 5.0) / 3.0) ** 2, 0.0, None)
    means = (1.0 - 0.5 * q ** 3 + 0.005 * rng.standard_normal(X.shape)).reshape(-1)
    kw = dict(P=4, Nx=nx, Ny=ny, Lx=Lx, Ly=Ly, g=G, c=ALPHA * math.sqrt(G), gamma=GAMMA, bc_x=1,
              bc_y=1, bathy_kind=sgnb.BATHY_CELLS, bathy_par=np.concatenate([[nx, ny, Lx, Ly], means]))
    x, y = (np.broadcast_to(t.cpu().numpy(), (ny, nx, 5, 5)) for t in _coords(kw))
    x0 = rng.uniform(5.0, 7.0)
    eta0 = (0.05 * np.exp(-((x - x0) ** 2 + (y - 5.0) ** 2) / 0.5)).reshape(-1)
    # gauges in the water that the hump moves within the run
    near = np.flatnonzero(np.maximum(np.abs(x - x0), np.abs(y - 5.0)).reshape(-1) < 1.0)
    gauges = np.sort(rng.choice(near, case["gauges"], replace=False)).astype(np.int64)
    lam = math.sqrt(G * 1.1 + kw["c"] ** 2) + 0.5
    dt = 0.4 * min(Lx / nx, Ly / ny) / 9.0 / lam
    dts = dt * rng.uniform(0.8, 1.0, case["steps"])
    eta_bar = rng.standard_normal((case["steps"], case["gauges"]))
    return kw, means, eta0, gauges, dts, eta_bar


def _start_dt(kw):
    """The step a program starts with and, as the loop's dtMax, never exceeds: 0.2 of the
    element-wise CFL step of the rest state. (The error control alone lets the step grow to
    the edge of linear stability, where the last bit of a state decides what is accepted.)"""
    H0 = kw["bathy_par"][0]
    lam = math.sqrt(G * 1.1 * H0 + kw["c"] ** 2) + 0.1
    return 0.2 * min(kw["Lx"] / kw["Nx"], kw["Ly"] / kw["Ny"]) / 9.0 / lam


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "adjoint":
        kw, means, eta0, gauges, dts, eta_bar = _adjoint_inputs(case, seed)
        solver = sgnb.SGN2DB200(precision=PRECISION[case["mode"]], **kw)
        return dict(kind=kind, solver=solver, adj=SGNAdjoint(solver, dts, gauges, case["every"]),
                    means=means, eta0=eta0, eta_bar=eta_bar)
    if kind == "batch":
        args = _sweep_args(case)
        U = [_state(kw, rng).reshape(-1) for kw in args]
        dt = [_start_dt(kw) for kw in args]
        return dict(kind=kind, batch=sgnb.SGNBatch(args, precision=PRECISION[case["mode"]]),
                    U=U, out=[torch.empty_like(u) for u in U],
                    dt=dt, opt=sgnb.AdaptiveRKOptions(dtMax=min(dt)), steps=case["steps"])
    kw = _solver_args(case)
    U = _state(kw, rng).reshape(-1)
    dt = _start_dt(kw)
    opt = sgnb.AdaptiveRKOptions(dtMax=dt)
    if kind == "slabs":
        return dict(kind=kind, slabs=SlabSolver(dict(kw, precision=PRECISION[case["mode"]]),
                                                nslabs=case["slabs"]),
                    U=U, dt=dt, opt=opt, steps=case["steps"])
    solver = sgnb.SGN2DB200(precision=PRECISION[case["mode"]], **kw)
    if kind == "rhs":
        return dict(kind=kind, solver=solver, U=U, dU=torch.empty_like(U))
    return dict(kind=kind, solver=solver, U=U, out=torch.empty_like(U), dt=dt, opt=opt,
                steps=case["steps"])


def run(state):
    kind = state["kind"]
    if kind == "rhs":
        state["solver"].rhs_device(state["U"].data_ptr(), state["dU"].data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
        return {"dU": state["dU"]}
    if kind == "steps":
        s = state["solver"]
        s.upload_tensor(state["U"])
        st = s.integrate_steps(0.0, state["dt"], state["steps"], state["opt"])
        # into the program's own tensor: the view ends with the solver
        state["out"].copy_(s.state_tensor())
        return {"U": state["out"], "t": st.tReached, "dt": st.dtLast,
                "accepted": st.accepted, "rejected": st.rejected}
    if kind == "batch":
        b = state["batch"]
        for i, U in enumerate(state["U"]):
            b[i].upload_tensor(U)
        sts = b.integrate_steps(state["dt"], state["steps"], state["opt"])
        for i, out in enumerate(state["out"]):
            out.copy_(b[i].state_tensor())
        return {"U": state["out"],
                "t": np.array([st.tReached for st in sts]),
                "accepted": np.array([st.accepted for st in sts]),
                "rejected": np.array([st.rejected for st in sts])}
    if kind == "adjoint":
        eta = state["adj"].forward(state["means"], state["eta0"])
        gm, ge = state["adj"].vjp(state["eta_bar"])
        return {"eta": eta, "grad_means": gm, "grad_eta0": ge}
    s = state["slabs"]
    s.upload_tensor(state["U"])
    st = s.integrate_steps(0.0, state["dt"], state["steps"], state["opt"])
    return {"U": s.download_tensor(), "t": st.tReached, "dt": st.dtLast,
            "accepted": st.accepted, "rejected": st.rejected}


# ---------------------------------------------------------------------------------------
# The work a pass cannot do without
# ---------------------------------------------------------------------------------------
def work(case):
    """Bytes per node. A right-hand side reads the five fields and the depth (nodal, and
    0.4 face values) and writes five derivatives. A BS3(2) step's three stages depend on
    one another across the whole mesh, so each is a pass of its own: u, k in, k out (twice),
    then u, k1, k2, k3 in, the new state and k4 out; derivatives are four bytes wide in the
    mixed mode. The adjoint: the forward, one more forward for the states between
    checkpoints, and per step three reverse right-hand sides (state and cotangent in,
    cotangent out) and the two recomputed stages.
    Operations: about 600 per node and right-hand side."""
    stat = 8 * 1.4
    k = 20 if case["mode"] == "mixed" else 40
    rhs = 80 + stat
    step = 2 * (40 + 2 * k + stat) + (2 * 40 + 4 * k + stat)
    kind = case["kind"]
    if kind == "batch":
        nodes = sum(25 * kw["Nx"] * kw["Ny"] for kw in _sweep_args(case))
    else:
        nodes = 25 * case["nx"] * case["ny"]
    if kind == "rhs":
        return {"bytes": nodes * rhs, "flops": nodes * 600}
    n = case["steps"]
    if kind == "adjoint":
        back = 2 * (40 + 2 * k + stat) + 3 * (120 + stat)
        return {"bytes": nodes * n * (2 * step + back), "flops": nodes * n * 600 * 16}
    return {"bytes": nodes * (rhs + n * step), "flops": nodes * 600 * (1 + 3 * n)}


# ---------------------------------------------------------------------------------------
# The same discretisation in plain torch, 64 bits
# ---------------------------------------------------------------------------------------
def _tables():
    """Differentiation matrix of the GLL points, derivatives of the two g_DG correction
    functions (the left one is the reflected right one)."""
    n = 5
    xi = np.array(_XI)
    w = np.array([1.0 / np.prod([xi[j] - xi[k] for k in range(n) if k != j]) for j in range(n)])
    D = np.zeros((n, n))
    for i in range(n):
        for j in range(n):
            if i != j:
                D[i, j] = w[j] / w[i] / (xi[i] - xi[j])
        D[i, i] = -D[i].sum()
    leg = np.polynomial.legendre.Legendre
    d4, d5 = leg.basis(4).deriv()(xi), leg.basis(5).deriv()(xi)
    return tuple(torch.tensor(a, dtype=torch.float64, device=DEV)
                 for a in (D, 0.5 * (d4 - d5), 0.5 * (d4 + d5)))


def _depth(kw, x, y, means=None):
    """Still depth at points (x, y)."""
    kind, p = kw["bathy_kind"], kw["bathy_par"]
    if kind == sgnb.BATHY_CONST:
        return p[0] + 0.0 * (x + y)
    if kind == sgnb.BATHY_GAUSS:
        return p[0] - p[1] * torch.exp(-((x - p[2]) ** 2 + (y - p[3]) ** 2) / p[4])
    if kind == sgnb.BATHY_SHOAL:
        q = torch.clamp(1.0 - (((x - p[2]) / p[4]) ** 2 + ((y - p[3]) / p[5]) ** 2), min=0.0)
        return p[0] - (p[0] - p[1]) * q ** 3
    # bilinear interpolant of cell means, periodic
    nx, ny = kw["Nx"], kw["Ny"]
    sx, sy = x / (kw["Lx"] / nx) - 0.5, y / (kw["Ly"] / ny) - 0.5
    fx, fy = torch.floor(sx), torch.floor(sy)
    tx, ty = sx - fx, sy - fy
    i0, j0 = fx.long() % nx, fy.long() % ny
    i1, j1 = (i0 + 1) % nx, (j0 + 1) % ny
    m = means.view(-1)
    a = m[i0 + nx * j0] + tx * (m[i1 + nx * j0] - m[i0 + nx * j0])
    b = m[i0 + nx * j1] + tx * (m[i1 + nx * j1] - m[i0 + nx * j1])
    return a + ty * (b - a)


class _Plain:
    """R(U) and the BS3(2) loop in torch; U is [5, Ny, Nx, 5 (y node), 5 (x node)]."""

    def __init__(self, kw, means=None):
        self.kw = kw
        self.D, self.gL, self.gR = _tables()
        self.J = (0.5 * kw["Lx"] / kw["Nx"], 0.5 * kw["Ly"] / kw["Ny"])
        x, y = _coords(kw)
        self.H = _depth(kw, x, y, means)
        self.Hg = (self._diff(self.H, 0) / self.J[0], self._diff(self.H, 1) / self.J[1])
        # face depths: left / bottom face of each element, and the domain's far edge
        xe = torch.arange(kw["Nx"], device=DEV, dtype=torch.float64) * (kw["Lx"] / kw["Nx"])
        ye = torch.arange(kw["Ny"], device=DEV, dtype=torch.float64) * (kw["Ly"] / kw["Ny"])
        fx = _depth(kw, xe[None, :, None], _axis(kw["Ny"], kw["Ly"])[:, None, :], means)
        fy = _depth(kw, _axis(kw["Nx"], kw["Lx"])[None, :, :], ye[:, None, None], means)
        endx = _depth(kw, torch.full_like(xe[:1, None], kw["Lx"]), _axis(kw["Ny"], kw["Ly"]), means)
        endy = _depth(kw, _axis(kw["Nx"], kw["Lx"]), torch.full_like(ye[:1, None], kw["Ly"]), means)
        hix, hiy = torch.roll(fx, -1, 1), torch.roll(fy, -1, 0)
        if kw["bc_x"]:
            hix = torch.cat([hix[:, :-1], endx[:, None, :]], 1)
        if kw["bc_y"]:
            hiy = torch.cat([hiy[:-1], endy[None]], 0)
        self.Hf = ((fx, hix), (fy, hiy))

    def _diff(self, f, d):
        return torch.einsum("mk,...k->...m", self.D, f) if d == 0 else \
            torch.einsum("mk,...kx->...mx", self.D, f)

    def _flux(self, U, H, d):
        kw = self.kw
        h, q = U[0], U[1 + d]
        vn, p = q / h, U[4] / h
        F = [q, q * U[1] / h, q * U[2] / h, q * U[3] / h, q * (p + kw["c"] ** 2)]
        F[1 + d] = q * vn + 0.5 * kw["g"] * (h - H) * (h + H) + U[4]
        return torch.stack(F)

    def _speed(self, U, d):
        kw = self.kw
        return torch.abs(U[1 + d] / U[0]) + torch.sqrt(kw["g"] * U[0] + U[4] / U[0] + kw["c"] ** 2)

    def _faces(self, U, d):
        """Own traces at the low and high face, and the neighbours' across them."""
        lo, hi = (U[..., 0], U[..., 4]) if d == 0 else (U[..., 0, :], U[..., 4, :])
        ax = 2 if d == 0 else 1
        nlo, nhi = torch.roll(hi, 1, ax), torch.roll(lo, -1, ax)
        if self.kw["bc_x" if d == 0 else "bc_y"]:
            sign = torch.ones(5, device=DEV, dtype=torch.float64)
            sign[1 + d] = -1.0
            sign = sign.view(5, 1, 1, 1)
            n = U.shape[ax]
            mlo, mhi = sign * lo.narrow(ax, 0, 1), sign * hi.narrow(ax, n - 1, 1)
            nlo = torch.cat([mlo, nlo.narrow(ax, 1, n - 1)], ax)
            nhi = torch.cat([nhi.narrow(ax, 0, n - 1), mhi], ax)
        return lo, hi, nlo, nhi

    def _jump(self, own, other, H, d, side):
        """Rusanov flux minus the own one; side +1: the own state is on the low side."""
        Fo, Fn = self._flux(own, H, d), self._flux(other, H, d)
        lam = torch.maximum(self._speed(own, d), self._speed(other, d))
        return 0.5 * (Fn - Fo) - 0.5 * side * lam * (other - own)

    def rhs(self, U):
        kw = self.kw
        h, w, p = U[0], U[3] / U[0], U[4] / U[0]
        vel = (U[1] / h, U[2] / h)
        out = torch.zeros_like(U)
        hp = 0.0
        for d in (0, 1):
            lo, hi, nlo, nhi = self._faces(U, d)
            jl = self._jump(lo, nlo, self.Hf[d][0], d, -1.0)
            jh = self._jump(hi, nhi, self.Hf[d][1], d, 1.0)
            def lift(a, b):
                return a[..., None] * self.gL + b[..., None] * self.gR if d == 0 else \
                    a[..., None, :] * self.gL[:, None] + b[..., None, :] * self.gR[:, None]
            out = out - (self._diff(self._flux(U, self.H, d), d) + lift(jl, jh)) / self.J[d]
            dh = (self._diff(h, d) + lift(0.5 * (nlo[0] - lo[0]), 0.5 * (nhi[0] - hi[0]))) / self.J[d]
            hp = hp + kw["c"] ** 2 * vel[d] * dh
        src = kw["g"] * (h - self.H) + kw["gamma"] * p
        s1, s2 = src * self.Hg[0], src * self.Hg[1]
        if kw.get("nManning", 0.0):
            cf = kw["nManning"] ** 2 * kw["g"] * torch.sqrt(vel[0] ** 2 + vel[1] ** 2) / h ** (1.0 / 3.0)
            s1, s2 = s1 - cf * vel[0], s2 - cf * vel[1]
        hp = hp - 2 * kw["c"] ** 2 * (w + vel[0] * self.Hg[0] + vel[1] * self.Hg[1])
        return out + torch.stack([torch.zeros_like(h), s1, s2, kw["gamma"] * p, hp])

    def bs3(self, u, dt):
        k1 = self.rhs(u)
        k2 = self.rhs(u + 0.5 * dt * k1)
        k3 = self.rhs(u + 0.75 * dt * k2)
        return u + dt * (2.0 / 9.0 * k1 + 1.0 / 3.0 * k2 + 4.0 / 9.0 * k3)

    def adaptive(self, u, dt, nsteps, dtmax, atol=1e-8, rtol=1e-6):
        """nsteps accepted BS3(2) steps with the PI controller (safety 0.9, factors in
        [0.2, 5], exponents 0.7 / 3 and 0.4 / 3). Returns u, t, the last step."""
        t, prev, n, dt, k1 = 0.0, 1.0, 0, min(dt, dtmax), self.rhs(u)
        while True:
            k2 = self.rhs(u + 0.5 * dt * k1)
            k3 = self.rhs(u + 0.75 * dt * k2)
            new = u + dt * (2.0 / 9.0 * k1 + 1.0 / 3.0 * k2 + 4.0 / 9.0 * k3)
            k4 = self.rhs(new)
            r = dt * (-5.0 / 72.0 * k1 + 1.0 / 12.0 * k2 + 1.0 / 9.0 * k3 - 0.125 * k4)
            r /= atol + rtol * torch.maximum(u.abs(), new.abs())
            err = max(math.sqrt(float(r.square().mean())), 1e-300)
            if err <= 1.0:
                t, n, u, k1 = t + dt, n + 1, new, k4
                last, prev = dt, err
                if n == nsteps:
                    return u, t, last
            dt = min(dtmax, dt * min(5.0, max(0.2, 0.9 * err ** (-0.7 / 3) * prev ** (0.4 / 3))))


def _exact_adjoint(case, seed):
    kw, means, eta0, gauges, dts, eta_bar = _adjoint_inputs(case, seed)
    m = torch.tensor(means, device=DEV, requires_grad=True)
    e0 = torch.tensor(eta0, device=DEV, requires_grad=True)
    solver = _Plain(kw, m)
    g = torch.tensor(gauges, device=DEV)
    shape = solver.H.shape
    u = torch.cat([(solver.H + e0.view(shape))[None], torch.zeros((4,) + shape, dtype=torch.float64,
                                                                 device=DEV)])
    eta = []
    for dt in dts:
        u = torch.utils.checkpoint.checkpoint(solver.bs3, u, float(dt), use_reentrant=False)
        eta.append((u[0] - solver.H).reshape(-1)[g])
    eta = torch.stack(eta)
    gm, ge = torch.autograd.grad((eta * torch.tensor(eta_bar, device=DEV)).sum(), (m, e0))
    return {"eta": eta.detach(), "grad_means": gm, "grad_eta0": ge}


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    rng = np.random.default_rng(seed)
    if kind == "batch":
        Us, ts = [], []
        args = _sweep_args(case)
        dtmax = min(_start_dt(kw) for kw in args)
        for kw in args:
            u, t, _ = _Plain(kw).adaptive(_state(kw, rng), _start_dt(kw), case["steps"], dtmax)
            Us.append(u.reshape(-1))
            ts.append(t)
        return {"U": Us, "t": np.array(ts)}
    kw = _solver_args(case)
    U = _state(kw, rng)
    plain = _Plain(kw)
    if kind == "rhs":
        return {"dU": plain.rhs(U).reshape(-1)}
    u, t, dt = plain.adaptive(U, _start_dt(kw), case["steps"], _start_dt(kw))
    return {"U": u.reshape(-1), "t": t, "dt": dt}
