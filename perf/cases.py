"""The work a user of phd_gb300 has it do, as timed cases.

Each case is one call (or the few calls of one time step) of the public entry
points on inputs made from a seed.  A case is a dict of plain values:

  kind    "iterate"  solvers.iterator for `steps` steps (1D or 2D)
          "step"     boundaries + solvers.ader_stepper, one step of a caller's
                     own loop, at Gauss order N (order.for_order(3) for N = 3)
          "stages"   the three stages called one by one (weno_launcher,
                     predictor, fv_launcher)
          "batch"    phd_gb300.batch.Batch.step: many uneven 1D grids
          "adjoint"  phd_gb300.adjoint.solve and its backward pass
          "bubble"   solvers.iterator with two materials (ghost fluid)
  problem "tube" (Riemann problem) or "vortex" (Taylor-Green), smoothly
          perturbed from the seed
  nx, ny  cells (ny = 0: 1D)        nvar   17 (heat conduction) or 14
  flux    0 Rusanov, 1 Roe, 2 Osher
  cfl, mu, split, steps, count as the entry points take them

`exact` evaluates the same step with plain torch in float64 (`_Scheme`,
`_step`), for the stiffened-gas Newtonian fluids that the cases use.
"""
import math

import numpy as np
import torch

import phd_gb300 as gpr
from phd_gb300 import adjoint as gadj
from phd_gb300 import order as gorder
from phd_gb300.batch import Batch
from phd_gb300.params import Cvec, material_params
from phd_gb300.problems import shock_bubble

TRANSMISSIVE, PERIODIC = 0, 1
DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the one-dimensional shock tube of the reference's first example:
        # the smallest grid in use, where launches and latency count
        dict(name="tube200", kind="iterate", problem="tube", nx=200, ny=0, nvar=17, flux=0,
             cfl=0.8, mu=1e-2, split=False, steps=4),
        # the same tube with the Osher flux (an eigen-problem per face point)
        dict(name="tube200_osher", kind="iterate", problem="tube", nx=200, ny=0, nvar=17, flux=2,
             cfl=0.8, mu=1e-2, split=False, steps=2),
        # the split scheme (analytic relaxation) on a fine 1D grid
        dict(name="tube2048_split", kind="iterate", problem="tube", nx=2048, ny=0, nvar=17,
             flux=0, cfl=0.8, mu=1e-3, split=True, steps=4),
        # a small 2D grid of odd sides, one step of a caller's own loop
        dict(name="vortex67x131", kind="step", problem="vortex", nx=67, ny=131, nvar=17, flux=0,
             cfl=0.4, mu=5e-2, order=2, stiff=False),
        # the headline workload: Taylor-Green 512 x 512
        dict(name="vortex512", kind="step", problem="vortex", nx=512, ny=512, nvar=17, flux=0,
             cfl=0.4, mu=1e-2, order=2, stiff=False),
        # the same flow at the production CFL, where most cells need the
        # stiff-source Newton pass
        dict(name="vortex256_cfl08", kind="step", problem="vortex", nx=256, ny=256, nvar=17,
             flux=0, cfl=0.8, mu=2e-2, order=2, stiff=False),
        # Roe's flux in 2D
        dict(name="vortex64_roe", kind="step", problem="vortex", nx=64, ny=64, nvar=17, flux=1,
             cfl=0.4, mu=8e-2, order=2, stiff=False),
        # third order (N = 3)
        dict(name="vortex128_order3", kind="step", problem="vortex", nx=128, ny=128, nvar=17,
             flux=0, cfl=0.4, mu=4e-2, order=3, stiff=False),
        # a fluid without heat conduction, its stages called one by one on a
        # ragged grid
        dict(name="stages301x203_v14", kind="stages", problem="vortex", nx=301, ny=203, nvar=14,
             flux=0, cfl=0.4, mu=2e-2),
        # 512 independent tubes of 128 .. 2048 cells in one batch
        dict(name="batch512", kind="batch", count=512, nmin=128, nmax=2048, steps=1),
        # gradients of a final state with respect to the initial states and
        # (mu, cs, calpha, gamma)
        dict(name="adjoint400", kind="adjoint", count=1, nx=400, tf=0.05),
        # shock-bubble interaction, two materials and a level set
        dict(name="bubble800x400", kind="bubble", nx=800, ny=400, steps=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges; costs at most what the largest
    listed case does."""
    kind = rng.choice(["iterate", "iterate", "step", "step", "step", "stages", "batch", "adjoint",
                       "bubble"])
    nvar = rng.choice([14, 17, 17])
    if kind == "iterate":
        flux = rng.choice([0, 0, 0, 1, 2])
        split = rng.random() < 0.4
        nx = _log(rng, 50, 1000 if flux else 4096)
        return dict(kind=kind, problem="tube", nx=nx, ny=0, nvar=nvar, flux=flux,
                    cfl=rng.choice([0.5, 0.8]), mu=rng.choice([1e-2, 1e-3]), split=split,
                    steps=rng.randint(1, 4))
    if kind == "step":
        order = rng.choice([2, 2, 2, 3])
        flux = rng.choice([0, 0, 0, 1, 2])
        hi = 512 if order == 2 else 180
        if flux:
            hi = 64 if order == 2 else 24
        nx, ny = _log(rng, 17, hi), _log(rng, 17, hi)
        # the relaxation time follows the cell size, as in a resolved flow
        mu = 1e-2 * 512 / max(nx, ny)
        cfl = 0.8 if flux == 0 and order == 2 and max(nx, ny) <= 256 and rng.random() < 0.3 \
            else 0.4
        return dict(kind=kind, problem="vortex", nx=nx, ny=ny, nvar=nvar, flux=flux, cfl=cfl,
                    mu=mu, order=order, stiff=False)
    if kind == "stages":
        nx, ny = _log(rng, 17, 400), _log(rng, 17, 400)
        return dict(kind=kind, problem="vortex", nx=nx, ny=ny, nvar=nvar, flux=0, cfl=0.4,
                    mu=1e-2 * 512 / max(nx, ny))
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 4, 500), nmin=_log(rng, 32, 128),
                    nmax=_log(rng, 200, 2048), steps=1)
    if kind == "adjoint":
        nx = _log(rng, 50, 400)
        return dict(kind=kind, count=rng.randint(1, 6), nx=nx, tf=0.05 * 400 / nx)
    ny = _log(rng, 60, 400)
    return dict(kind=kind, nx=2 * ny + rng.randint(-7, 0), ny=ny, steps=1)


# ---------------------------------------------------------------------------
# inputs

def _waves(shape, rng, amp, device):
    """A smooth random field: a few Fourier modes with seeded phases."""
    ax = [torch.arange(n, dtype=torch.float64, device=device) / n for n in shape]
    f = torch.zeros(shape, dtype=torch.float64, device=device)
    for _ in range(3):
        ph = torch.full(shape, float(rng.uniform(0, 2 * math.pi)), dtype=torch.float64,
                        device=device)
        for d, a in enumerate(ax):
            k = int(rng.integers(1, 4))
            ph = ph + 2 * math.pi * k * a.reshape([-1 if e == d else 1 for e in range(len(ax))])
        f = f + torch.sin(ph)
    return amp / 3 * f


def _conserved(rho, p, v, A, J, M):
    """Conserved states [rho, rho E, rho v, A, rho J] of a stiffened gas."""
    r = rho
    G = A.transpose(-1, -2) @ A
    D = G - torch.eye(3, dtype=G.dtype, device=G.device) * (
        torch.diagonal(G, dim1=-2, dim2=-1).sum(-1) / 3)[..., None, None]
    E = (p + M.gamma * M.pINF) / (r * (M.gamma - 1)) + 0.25 * M.b02 * (D * D).sum((-1, -2)) \
        + 0.5 * (v * v).sum(-1)
    cols = [r[..., None], (r * E)[..., None], r[..., None] * v, A.flatten(-2)]
    if J is not None:
        cols[1] = cols[1] + (0.5 * M.calpha2 * r * (J * J).sum(-1))[..., None]
        cols.append(r[..., None] * J)
    return torch.cat(cols, -1).contiguous()


def _flow(case, seed, device=DEV):
    """(u0, Par, dX, boundary code) of a "tube" or "vortex" case."""
    rng = np.random.default_rng([seed, 71])
    th = case["nvar"] == 17
    shape = (case["nx"],) if not case["ny"] else (case["nx"], case["ny"])

    def w(amp):
        return _waves(shape, rng, amp, device)

    eye = torch.eye(3, dtype=torch.float64, device=device)
    if case["problem"] == "tube":
        # density and pressure jump at x = 1/2 of the first workload, the
        # distortion at the density's compression
        M = material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=1.0, mu=case["mu"],
                            calpha=1.0 if th else None, Pr=2.0 / 3.0)
        dX = [1.0 / case["nx"]]
        left = torch.arange(case["nx"], device=device) * dX[0] < 0.5
        rho = torch.where(left, 1.0, 0.125).double() * (1 + w(0.02))
        p = torch.where(left, 1.0, 0.1).double() * (1 + w(0.02))
        v = torch.stack([w(0.02) for _ in range(3)], -1)
        A = eye + torch.stack([w(0.01) for _ in range(9)], -1).reshape(shape + (3, 3))
        bc = TRANSMISSIVE
    else:
        M = material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=10.0, mu=case["mu"],
                            calpha=1.0 if th else None, Pr=2.0 / 3.0)
        dX = [2 * math.pi / n for n in shape]
        X = [(torch.arange(n, dtype=torch.float64, device=device) + 0.5) * h
             + float(rng.uniform(0, 2 * math.pi)) for n, h in zip(shape, dX)]
        X, Y = torch.meshgrid(*X, indexing="ij")
        rho = 1 + w(1e-2)
        p = 100 / 1.4 + (torch.cos(2 * X) + torch.cos(2 * Y)) / 4 + w(1e-1)
        v = torch.stack([torch.sin(X) * torch.cos(Y), -torch.cos(X) * torch.sin(Y), w(1e-2)], -1)
        # a developed flow's strain and heat flux: of the size of the
        # relaxation time (6 mu / cs^2) times the velocity gradient, and of
        # Fourier's law
        A = eye + torch.stack([w(0.5 * 6e-2 * case["mu"]) for _ in range(9)], -1).reshape(
            shape + (3, 3))
        bc = PERIODIC
    # det A = rho / rho0, which the time loop keeps
    A = A * (rho / torch.linalg.det(A))[..., None, None] ** (1 / 3)
    aJ = 1e-2 * case["mu"] if case["problem"] == "vortex" else 1e-2
    J = torch.stack([w(aJ) for _ in range(3)], -1) if th else None
    return _conserved(rho, p, v, A, J, M), M, dX, bc


def _dt(case, u, M, dX):
    return case["cfl"] / float(_cfl(u, _Mat(M), dX))


class State:
    """What one case keeps between passes."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _batch_instances(case, seed):
    rng = np.random.default_rng([seed, 72])
    # the cell counts are the case's, the states and materials the seed's
    sizes = np.random.default_rng([case["count"], case["nmin"], case["nmax"]]).integers(
        case["nmin"], case["nmax"] + 1, case["count"])
    out = []
    for nx in sizes:
        rho, v = rng.uniform(0.1, 2.0, 2), rng.uniform(-0.5, 0.5, 2)
        p = np.exp(rng.uniform(math.log(0.1), math.log(10.0), 2))
        M = material_params("sg", 1.0, cv=2.5, gamma=float(rng.uniform(1.2, 1.67)),
                            b0=float(rng.uniform(0.5, 5.0)), calpha=1.0,
                            mu=float(np.exp(rng.uniform(math.log(1e-4), math.log(1e-1)))),
                            Pr=2.0 / 3.0)
        Q = [Cvec(rho[k], p[k], np.array([v[k], 0.0, 0.0]), M, rho[k] ** (1 / 3) * np.eye(3),
                  np.zeros(3)) for k in range(2)]
        x = np.arange(nx) / nx
        out.append((np.where((x < 0.5)[:, None], Q[0], Q[1]), M, [1.0 / nx], TRANSMISSIVE))
    return out


def _theta(case, seed):
    """(mu, cs, calpha, gamma) of every instance of an adjoint case."""
    rng = np.random.default_rng([seed, 73])
    return np.array([1e-2, 1.0, 1.0, 1.4]) * (1 + 0.05 * rng.uniform(-1, 1, (case["count"], 4)))


def _adjoint_par(theta):
    mu, cs, calpha, gamma = theta
    return material_params("sg", 1.0, cv=1.0, gamma=gamma, b0=cs, calpha=calpha, mu=mu, Pr=0.75)


def _adjoint_inputs(case, seed, device=DEV):
    """Initial states of the first problem of Stokes (a shear layer), smoothly
    perturbed, and a cotangent for each final state."""
    rng = np.random.default_rng([seed, 74])
    nx, eye = case["nx"], torch.eye(3, dtype=torch.float64, device=device)
    us = []
    for th in _theta(case, seed):
        M = _adjoint_par(th)

        def w(amp):
            return _waves((nx,), rng, amp, device)

        rho, p = 1 + w(0.02), (1 + w(0.02)) / M.gamma
        shear = torch.where(torch.arange(nx, device=device) * (2.0 / nx) < 1.0, 0.1, -0.1).double()
        v = torch.stack([w(0.02), shear + w(0.02), w(0.02)], -1)
        A = eye + torch.stack([w(0.02) for _ in range(9)], -1).reshape(nx, 3, 3)
        A = A * (rho / torch.linalg.det(A))[:, None, None] ** (1 / 3)
        us.append(_conserved(rho, p, v, A, torch.stack([w(0.02) for _ in range(3)], -1), M))
    u0 = torch.cat(us)
    return u0, torch.stack([_waves((u0.shape[0],), rng, 1.0, device) for _ in range(17)], -1)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = Batch(_batch_instances(case, seed), cfl=0.8, tf=0.2)
        return State(case=case, b=b, u0=b.u.clone(), clock0=b.clock.clone())
    if kind == "adjoint":
        u0, cot = _adjoint_inputs(case, seed)
        prob = gadj.Problem([case["nx"]] * case["count"], [2.0 / case["nx"]] * case["count"],
                            "transitive", _adjoint_par, cfl=0.8, tf=case["tf"])
        return State(case=case, prob=prob, u0=u0, cot=cot, theta=torch.tensor(_theta(case, seed)))
    if kind == "bubble":
        rng = np.random.default_rng([seed, 75])
        u, MPs, tf, dX, _ = shock_bubble(
            nx=case["nx"], ny=case["ny"], mach=1.22 + 0.05 * rng.uniform(-1, 1),
            radius=0.2 + 0.01 * rng.uniform(-1, 1), shear=1e-3 * rng.uniform(1, 2),
            centre=(0.6 + 0.02 * rng.uniform(-1, 1), 0.5 + 0.02 * rng.uniform(-1, 1)))
        u0 = torch.tensor(u, device=DEV)
        return State(case=case, u0=u0, u=u0.clone(), MPs=MPs, tf=tf, dX=dX,
                     nX=[case["nx"], case["ny"]], bcs=[TRANSMISSIVE] * 4)
    u0, M, dX, bc = _flow(case, seed)
    s = State(case=case, u0=u0, u=u0.clone(), MP=M, dX=dX, nX=list(u0.shape[:-1]),
              bcs=[bc] * (2 * len(dX)))
    if kind != "iterate":
        s.N = case.get("order", 2)
        s.G = gpr if s.N == 2 else gorder.for_order(s.N)
        s.dt = _dt(case, u0, M, dX)
        V = u0.shape[-1]
        ncb = int(np.prod([n + 2 for n in s.nX]))
        s.ub = torch.empty(int(np.prod([n + 2 * s.N for n in s.nX])) * V, dtype=torch.float64,
                           device=DEV)
        s.mask = torch.ones(ncb, dtype=torch.bool, device=DEV)
        if kind == "stages":
            ns = s.N ** len(s.nX)
            s.wh = torch.empty(ncb * ns * V, dtype=torch.float64, device=DEV)
            s.qh = torch.empty(ncb * s.N * ns * V, dtype=torch.float64, device=DEV)
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "batch":
        s.b.u.copy_(s.u0)
        s.b.clock.copy_(s.clock0)
        s.b.step(case["steps"])
        return [s.b.u, s.b.clock]
    if kind == "adjoint":
        u0 = s.u0.clone().requires_grad_()
        theta = s.theta.clone().requires_grad_()
        uN = gadj.solve(u0, theta, s.prob)
        uN.backward(s.cot)
        return [uN.detach(), u0.grad, theta.grad]
    s.u.copy_(s.u0)
    if kind == "bubble":
        return gpr.solvers.iterator(s.u, s.tf, s.nX, s.dX, 0.8, s.bcs, False, True, False, 0,
                                    s.MPs, max_steps=case["steps"])[99]
    if kind == "iterate":
        return gpr.solvers.iterator(s.u, 1.0, s.nX, s.dX, case["cfl"], s.bcs, case["split"], True,
                                    False, case["flux"], [s.MP], max_steps=case["steps"])[99]
    s.G.boundaries(s.u, s.ub, s.nX, s.bcs)
    if kind == "step":
        s.G.solvers.ader_stepper(s.u, s.ub, s.nX, s.dt, s.dX, case["stiff"], case["flux"], s.MP,
                                 s.mask)
        return s.u
    gpr.api.set_grid(s.nX)
    s.G.solvers.weno.weno_launcher(s.wh, s.ub, s.nX)
    s.G.solvers.dg.predictor(s.qh, s.wh, s.dt, s.dX, False, False, s.MP, s.mask)
    s.G.solvers.fv.fv_launcher(s.u, s.qh, s.nX, s.dt, s.dX, True, True, case["flux"], s.MP,
                               s.mask)
    return [s.wh, s.qh, s.u]


# ---------------------------------------------------------------------------
# work: floating-point operations of the scheme's own terms (a division, root
# or power counts one), with the derived quantities of a state computed once

_STATE, _FLUX, _WAVE, _SOURCE, _WENO = 85, 35, 150, 40, 44


def _cell_flops(nd, N, V, flux, ader=True, iters=2):
    nt = N if ader else 1
    pts = N ** (nd - 1) * nt          # quadrature points of a face
    nodes = N ** nd * nt              # space-time nodes of a cell
    side = 2 * N * V + _STATE + _FLUX + _WAVE
    face = 2 * side + 6 * V
    if flux:  # |M| (qL - qR): one matrix and eight products with it per path node
        face += (N if flux == 2 else 1) * 9 * 2 * V * 8
    weno = sum(N ** d for d in range(nd)) * V * _WENO * (1 if N == 2 else 2.5)
    node = _STATE + _SOURCE + nd * (_FLUX + 2 * N * V) + 2 * N * V
    pred = nodes * node * iters if ader else N ** nd * node
    return nd * pts * face + weno + pred + nodes * node + nd * _WAVE


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = int(np.random.default_rng([case["count"], case["nmin"], case["nmax"]]).integers(
            case["nmin"], case["nmax"] + 1, case["count"]).sum())
        return {"bytes": 16.0 * 17 * n * case["steps"],
                "flops": n * case["steps"] * _cell_flops(1, 2, 17, 0)}
    if kind == "adjoint":
        # forward and transposed steps until tf, the predictor to its fixed point
        n, steps = case["count"] * case["nx"], 32
        return {"bytes": 32.0 * 17 * n, "flops": 3.0 * n * steps * _cell_flops(1, 2, 17, 0,
                                                                              iters=8)}
    if kind == "bubble":
        n = case["nx"] * case["ny"]
        return {"bytes": 16.0 * 15 * n * case["steps"],
                "flops": case["steps"] * n * _cell_flops(2, 2, 15, 0)}
    nd = 2 if case["ny"] else 1
    n = case["nx"] * max(case["ny"], 1)
    V, N, steps = case["nvar"], case.get("order", 2), case.get("steps", 1)
    vals = 2 * V
    if kind == "stages":  # wh and qh are outputs too
        vals += V * N ** nd * (1 + N)
    return {"bytes": 8.0 * vals * n * steps,
            "flops": n * steps * _cell_flops(nd, N, V, case["flux"], not case.get("split"))}


# ---------------------------------------------------------------------------
# the same step in plain torch, float64

class _Mat:
    """Parameters of a stiffened-gas Newtonian fluid (floats or tensors)."""

    def __init__(self, M, theta=None):
        self.gamma, self.b02, self.calpha2 = M.gamma, M.b02, M.calpha2
        self.mu, self.kappa = M.mu, M.kappa
        self.rho0, self.cv, self.pINF = M.rho0, M.cv, M.pINF
        if theta is not None:  # (mu, cs, calpha, gamma) as differentiable numbers
            self.mu, self.gamma = theta[0], theta[3]
            self.b02, self.calpha2 = theta[1] ** 2, theta[2] ** 2
            self.kappa = theta[0] * theta[3] * M.cv / 0.75


class _Scheme:
    """Gauss-Legendre nodes, basis, WENO stencils and DG matrices for N nodes
    on [0, 1]."""

    def __init__(self, N, device):
        x, w = np.polynomial.legendre.leggauss(N)
        x, w = (x + 1) / 2, w / 2
        base = []
        for i in range(N):
            p = np.poly1d([1.0])
            for j in range(N):
                if j != i:
                    p = p * np.poly1d([1.0, -x[j]]) / (x[i] - x[j])
            base.append(p)
        I = [p.integ() for p in base]

        def stencil(shift):
            return np.linalg.inv([[P(i + shift + 1) - P(i + shift) for P in I] for i in range(N)])

        def t(a):
            return torch.tensor(np.asarray(a, dtype=np.float64), device=device)

        self.N, self.w, self.x = N, t(w), t(x)
        self.end = t([[p(0.0) for p in base], [p(1.0) for p in base]])
        der = np.array([[p.deriv()(xi) for p in base] for xi in x])
        self.der = t(der)
        # stencils ending at, starting at and (N = 3) around the cell, with
        # their first window row and linear weight
        self.sten = [(t(stencil(1 - N)), 0, 1.0), (t(stencil(0)), N - 1, 1.0)]
        if N == 3:
            self.sten.append((t(stencil(-1)), 1, 1e5))
        sig = np.zeros((N, N))
        for i in range(N):
            for j in range(N):
                for a in range(1, N):
                    q = (base[i].deriv(a) * base[j].deriv(a)).integ()
                    sig[i, j] += q(1.0) - q(0.0)
        self.sig = t(sig)
        dgder = w[:, None] * der
        self.dgder = t(dgder)
        mat = np.outer([p(1.0) for p in base], [p(1.0) for p in base]) - dgder.T
        self.mat, self.matinv = t(mat), t(np.linalg.inv(mat))


def _prims(Q, M):
    r = Q[..., 0]
    v = Q[..., 2:5] / r[..., None]
    A = Q[..., 5:14].unflatten(-1, (3, 3))
    G = A.transpose(-1, -2) @ A
    D = G - torch.eye(3, dtype=Q.dtype, device=Q.device) * (
        torch.diagonal(G, dim1=-2, dim2=-1).sum(-1) / 3)[..., None, None]
    e = Q[..., 1] / r - 0.5 * (v * v).sum(-1) - 0.25 * M.b02 * (D * D).sum((-1, -2))
    J = None
    if Q.shape[-1] == 17:
        J = Q[..., 14:17] / r[..., None]
        e = e - 0.5 * M.calpha2 * (J * J).sum(-1)
    p = (M.gamma - 1) * r * (e - M.pINF / r) - M.pINF
    T = (p + M.pINF) / (r * (M.gamma - 1) * M.cv)
    return r, v, A, G, D, J, p, T


def _flux(Q, d, M):
    r, v, A, G, D, J, p, T = _prims(Q, M)
    sg = -r[..., None] * M.b02 * (D @ G)[..., :, d]
    vd = v[..., d]
    F = [Q[..., 2 + d],
         vd * (Q[..., 1] + p) - (sg * v).sum(-1)]
    if J is not None:
        F[1] = F[1] + M.calpha2 * T * J[..., d]
    F += [vd * Q[..., 2 + i] - sg[..., i] + (p if i == d else 0.0) for i in range(3)]
    Av = (A @ v[..., None])[..., 0]
    zero = torch.zeros_like(vd)
    F += [Av[..., i] if j == d else zero for i in range(3) for j in range(3)]
    if J is not None:
        F += [vd * Q[..., 14 + i] + (T if i == d else 0.0) for i in range(3)]
    return torch.stack(F, -1)


def _source(Q, M):
    r, v, A, G, D, J, p, T = _prims(Q, M)
    det = torch.linalg.det(A)
    th = det * (det * det) ** (1 / 3) * M.rho0 / (2 * M.mu)  # det(A)^(5/3)
    S = [torch.zeros_like(Q[..., :5]), (-M.b02 * th[..., None, None] * (A @ D)).flatten(-2)]
    if J is not None:
        S.append(-(M.calpha2 / M.kappa) * T[..., None] * J)
    return torch.cat(S, -1)


def _bdot(Q, X, d):
    v = Q[..., 2:5] / Q[..., :1]
    x = X[..., 5:14].unflatten(-1, (3, 3))
    cols = []
    for c in range(3):
        if c == d:
            cols.append(-sum(v[..., k, None] * x[..., :, k] for k in range(3) if k != d))
        else:
            cols.append(v[..., d, None] * x[..., :, c])
    return torch.cat([torch.zeros_like(X[..., :5]), torch.stack(cols, -1).flatten(-2),
                      torch.zeros_like(X[..., 14:])], -1)


def _wave(Q, d, M):
    """|v_d| + the square root of the thermo-acoustic tensor's largest
    eigenvalue (Newton's iteration on its characteristic polynomial from an
    upper bound; the last step is differentiable)."""
    r, v, A, G, D, J, p, T = _prims(Q, M)
    S = D @ G
    g = G[..., :, d]
    X = S + g[..., :, None] * g[..., None, :] / 3 + g[..., d, None, None] * G
    dd = torch.zeros(3, 3, dtype=Q.dtype, device=Q.device)
    dd[d, d] = 1.0
    X = M.b02 * (X + dd @ S)
    e0 = torch.zeros(3, dtype=Q.dtype, device=Q.device)
    e0[0] = 1.0
    ed = torch.zeros(3, dtype=Q.dtype, device=Q.device)
    ed[d] = 1.0
    X = X + (M.b02 * S[..., :, d])[..., :, None] * e0          # - dsigma/drho
    gm = M.gamma - 1
    pp = p + M.pINF
    c2 = M.gamma * pp / r                                      # sound speed squared
    X = X + e0[:, None] * (c2[..., None] * ed)[..., None, :]
    if J is not None:
        h = M.calpha2 * T * gm
        tp = 1 / (r * r * gm * M.cv)
        right = (e0 * (h / r)[..., None])[..., :, None]
        low = e0 * (-pp / (r * r * gm * M.cv))[..., None] + ed * (tp * r * c2)[..., None]
        X = torch.cat([torch.cat([X, right], -1),
                       torch.cat([low, (tp * h)[..., None]], -1)[..., None, :]], -2)
    m = X.shape[-1]
    eye = torch.eye(m, dtype=Q.dtype, device=Q.device)
    c, P = [], eye
    for k in range(1, m + 1):  # Faddeev - Le Verrier
        XP = X @ P
        c.append(-torch.diagonal(XP, dim1=-2, dim2=-1).sum(-1) / k)
        P = XP + c[-1][..., None, None] * eye
    lam = X.detach().abs().sum(-1).amax(-1)
    cd = [x.detach() for x in c]
    for _ in range(60):
        f, df = torch.ones_like(lam), torch.zeros_like(lam)
        for x in cd:
            df = df * lam + f
            f = f * lam + x
        lam = lam - torch.where(df != 0, f / df, torch.zeros_like(f))
    f, df = torch.ones_like(lam), torch.zeros_like(lam)
    for x in cd:
        df = df * lam + f
        f = f * lam + x
    f = torch.ones_like(lam)
    for x in c:
        f = f * lam + x
    return v[..., d].abs() + torch.sqrt(lam - f / df)


def _jacobian(Q, d, M):
    """dF_d/dQ + B_d by complex steps."""
    V, cols = Q.shape[-1], []
    for k in range(V):
        z = Q.to(torch.complex128)
        z[..., k] += 1e-30j
        cols.append(_flux(z, d, M).imag / 1e-30)
    eye = torch.eye(V, dtype=Q.dtype, device=Q.device)
    B = torch.stack([_bdot(Q, eye[k].expand_as(Q), d) for k in range(V)], -1)
    return torch.stack(cols, -1) + B


def _abs_apply(J, dq):
    """|J| dq by eigen-decomposition."""
    lam, R = np.linalg.eig(J.cpu().numpy())
    y = np.linalg.solve(R, dq.cpu().numpy()[..., None].astype(complex))
    out = (R @ (np.abs(lam)[..., None] * y))[..., 0].real
    return torch.tensor(out, device=dq.device)


def _interface(ql, qr, d, M, flux, S):
    if flux == 0:
        f = torch.maximum(_wave(ql, d, M), _wave(qr, d, M))[..., None] * (ql - qr)
    else:
        dq = ql - qr
        Js = [_jacobian(qr + x * dq, d, M) for x in S.x]
        if flux == 2:
            f = sum(w * _abs_apply(J, dq) for w, J in zip(S.w, Js))
        else:
            f = _abs_apply(sum(w * J for w, J in zip(S.w, Js)), dq)
    f = f + _flux(ql, d, M) + _flux(qr, d, M)
    b = sum(w * _bdot(ql + x * (qr - ql), qr - ql, d) for w, x in zip(S.w, S.x))
    return f, b


def _ghosts(u, N, bc):
    for d in range(u.dim() - 1):
        n = u.shape[d]
        i = torch.arange(-N, n + N, device=u.device)
        u = u.index_select(d, i % n if bc == PERIODIC else i.clamp(0, n - 1))
    return u


def _weno(data, S, use):
    """Node values (a new leading axis) from 2N - 1 window rows; use[s]: where
    stencil s may be taken."""
    num, den = 0.0, 0.0
    for (m, r0, lam), on in zip(S.sten, use):
        w = torch.einsum("ab,b...->a...", m, torch.stack(data[r0:r0 + S.N]))
        t = (torch.einsum("a...,ab->b...", w, S.sig) * w).sum(0) + 1e-14
        o = on * lam / t ** 8
        num, den = num + w * o, den + o
    return num / den


def _reconstruct(ub, S):
    """WENO node values [cells...][nodes...][V] of the cells and one ghost
    layer around them."""
    N, dev = S.N, ub.device
    nxp = ub.shape[0] - 2 * N + 2
    rows = [ub[k:k + nxp] for k in range(2 * N - 1)]

    def use(i, n, gap):
        on = [i >= gap, i <= n - gap - 1]
        return [x.double() for x in (on + [i + 1 >= gap] if N == 3 else on)]

    i = torch.arange(nxp, device=dev)
    if ub.dim() == 2:
        return _weno(rows, S, [x[:, None] for x in use(i, nxp, 0)]).movedim(0, 1)
    nyb = ub.shape[1]
    j = torch.arange(nyb, device=dev)
    gap = torch.where((j < N) | (j >= nyb - N), N, 0)
    ux = _weno(rows, S, [x[..., None] for x in use(i[:, None], nxp, gap[None, :])])
    nyp = nyb - 2 * N + 2
    cols = [ux[:, :, k:k + nyp] for k in range(2 * N - 1)]   # [a][i][j][V]
    j = torch.arange(nyp, device=dev)
    gap = torch.where((i == 0) | (i == nxp - 1), 1, 0)
    wh = _weno(cols, S, [x[None, :, :, None] for x in use(j[None, :], nyp, gap[:, None])])
    return wh.permute(2, 3, 1, 0, 4)                         # [i][j][a][b][V]


def _along(m, q, ax):
    return torch.movedim(torch.tensordot(m, q, dims=([1], [ax])), 0, ax)


def _smooth_rhs(q, dX, M, S, source=True):
    """S(q) - B dq/dx - ... at the nodes of q [cells][t][nodes...][V]."""
    r = _source(q, M) if source else torch.zeros_like(q)
    for d, h in enumerate(dX):
        r = r - _bdot(q, _along(S.der, q, 2 + d) / h, d)
    return r


def _weighted(S, nd):
    """Quadrature weights of a cell's spatial nodes, shaped to broadcast over
    [cells][t][nodes...][V]."""
    w = S.w.reshape([1, 1, S.N] + [1] * nd)
    return w if nd == 1 else w * S.w.reshape(1, 1, 1, S.N, 1)


def _dg_map(q, w, dt, dX, M, S):
    """One application of the predictor's fixed-point map."""
    r = _smooth_rhs(q, dX, M, S)
    for d, h in enumerate(dX):
        r = r - _along(S.dgder / S.w[:, None], _flux(q, d, M), 2 + d) / h
    sh = [1, S.N] + [1] * (q.dim() - 2)
    r = r * S.w.reshape(sh) * dt + S.end[0].reshape(sh) * w[:, None]
    return _along(S.matinv, r, 1)


def _predict(wh, dt, dX, M, S, tol=6e-6, its=50):
    """Picard iteration with the reference's per-cell stop; cells that do not
    stop get the fixed point by a Newton iteration implicit in the sources."""
    q = wh[:, None].expand([wh.shape[0], S.N] + list(wh.shape[1:])).clone()
    live = torch.arange(q.shape[0], device=q.device)
    out = q.clone()
    for _ in range(its):
        if live.numel() == 0:
            break
        q0 = q[live]
        q1 = _dg_map(q0, wh[live], dt, dX, M, S)
        big = ((q1 - q0).abs() > tol * (1 + q0.abs())).flatten(1).any(1)
        out[live[~big]] = q1[~big]
        q[live[big]] = q1[big]
        live = live[big]
    if live.numel():
        out[live] = _newton(wh[live], dt, dX, M, S)
    return out


def _newton(w, dt, dX, M, S):
    """The predictor's fixed point, implicit in the relaxation sources."""
    N, V = S.N, w.shape[-1]
    q = w[:, None].expand([w.shape[0], N] + list(w.shape[1:])).clone()
    for _ in range(60):
        g = _dg_map(q, w, dt, dX, M, S) - q               # DG_MAT^-1 of the residual
        jac = torch.zeros(q.shape[:-1] + (V, V), dtype=q.dtype, device=q.device)
        for k in range(5, V):                             # dS/dq by complex steps
            z = q.to(torch.complex128)
            z[..., k] += 1e-30j
            jac[..., k] = _source(z, M).imag / 1e-30
        # (I - dt DG_MAT^-1 W dS/dq) delta = g, coupled over the time nodes
        js = jac.movedim(1, -3).reshape(-1, N, V, V)
        K = -dt * torch.einsum("tm,m,cmij->ctimj", S.matinv, S.w, js).reshape(-1, N * V, N * V)
        K = K + torch.eye(N * V, dtype=q.dtype, device=q.device)
        gs = g.movedim(1, -2)
        d = torch.linalg.solve(K, gs.reshape(-1, N * V, 1)).reshape(gs.shape).movedim(-2, 1)
        q = q + d
        if not (d.abs() > 1e-14 * (1 + q.abs())).any():
            break
    return q


def _update(u, qh, dt, dX, M, S, flux, sources=True):
    """u plus the finite-volume update from node values qh [cells incl. one
    ghost layer][t][nodes...][V]."""
    nd, N = len(dX), S.N
    nt = qh.shape[nd]
    wt = (S.w if nt > 1 else torch.ones(1, dtype=u.dtype, device=u.device)) * dt
    q = qh[(slice(1, -1),) * nd].flatten(0, nd - 1)
    vol = _smooth_rhs(q, dX, M, S, sources) * _weighted(S, nd)
    vol = vol * wt.reshape([1, -1] + [1] * (nd + 1))
    u = u + vol.sum(list(range(1, nd + 2))).reshape(u.shape)
    for d, h in enumerate(dX):
        inner = tuple(slice(None) if e == d else slice(1, -1) for e in range(nd))
        # the two traces at every face: [cells][t][transverse node][V]
        L = torch.tensordot(S.end[1], qh[inner], dims=([0], [nd + 1 + d]))
        R = torch.tensordot(S.end[0], qh[inner], dims=([0], [nd + 1 + d]))
        n = L.shape[d]
        f, b = _interface(L.narrow(d, 0, n - 1), R.narrow(d, 1, n - 1), d, M, flux, S)
        k = wt / (2 * h)
        if nd == 2:
            k = k[:, None] * S.w
        k = k[..., None]
        fl, fr = ((b + f) * k), ((b - f) * k)
        dims = list(range(nd, fl.dim() - 1))
        fl, fr = fl.sum(dims), fr.sum(dims)
        u = u - fl.narrow(d, 1, n - 2) - fr.narrow(d, 0, n - 2)
    return u


def _step(u, dt, dX, M, S, bc, flux, tol=6e-6, its=50, parts=False):
    nd = len(dX)
    wh = _reconstruct(_ghosts(u, S.N, bc), S)
    qh = _predict(wh.flatten(0, nd - 1), dt, dX, M, S, tol, its)
    qh = qh.unflatten(0, wh.shape[:nd])
    un = _update(u, qh, dt, dX, M, S, flux)
    return (wh, qh, un) if parts else un


def _ode(Q, dt, M):
    """The analytic relaxation step of the split scheme."""
    U, s, Vh = torch.linalg.svd(Q[..., 5:14].unflatten(-1, (3, 3)))
    det13 = s.prod(-1) ** (1 / 3)
    k = (s / det13[..., None]) ** 2
    m0 = k.sum(-1) / 3
    u0 = ((k[..., 0] - k[..., 1]) ** 2 + (k[..., 1] - k[..., 2]) ** 2
          + (k[..., 2] - k[..., 0]) ** 2) / 3
    tau = M.rho0 * M.b02 * det13 ** 7 / (3 * M.mu) * dt
    e6, e9 = torch.exp(-6 * tau), torch.exp(-9 * tau)
    a, b = 3 * m0 - u0 / 3 - 3, 2 * m0 - u0 / 3 - 2
    m = 1 + a * e6 - b * e9
    uu = (6 * a * e6 - 9 * b * e9).clamp(min=0)
    Dl = -2 * m ** 3 + m * uu + 2
    arg = (6 * uu ** 3 - 81 * Dl ** 2).clamp(min=0)
    safe = torch.where(Dl.abs() < 1e-12, torch.ones_like(Dl), Dl)
    th = torch.where(Dl.abs() < 1e-12, torch.full_like(Dl, math.pi / 2),
                     torch.atan(arg.sqrt() / (9 * safe)))
    x1 = (6 * uu).sqrt() / 3 * torch.cos(th / 3) + m
    cb = torch.sign(safe) * (54 * safe).abs() ** (1 / 3)
    x1 = torch.where((arg == 0) & (Dl.abs() >= 1e-12), cb / 6 + uu / cb + m, x1)
    t2 = 3 * m - x1
    x2 = 0.5 * (((x1 * t2 * t2 - 4).clamp(min=0) / x1).sqrt() + t2)
    x = torch.stack([x1, x2, 1 / (x1 * x2)], -1).sort(-1, descending=True)[0]
    An = (U * (det13[..., None] * x.sqrt())[..., None, :]) @ Vh
    An = torch.where((u0 < 1e-12)[..., None], Q[..., 5:14], An.flatten(-2))
    Q = torch.cat([Q[..., :5], An, Q[..., 14:]], -1)
    if Q.shape[-1] == 17:
        r, v, A, G, D, J, p, T = _prims(Q, M)
        c1 = Q[..., 1] / r - 0.25 * M.b02 * (D * D).sum((-1, -2)) - 0.5 * (v * v).sum(-1)
        k = 2 * M.calpha2 / (M.kappa * r * M.cv)
        ea = torch.exp(-c1 * k * dt / 2)
        den = 1 - (M.calpha2 / 2) / c1 * (1 - ea * ea) * (J * J).sum(-1)
        Q = torch.cat([Q[..., :14], Q[..., 14:] * (ea / den.sqrt())[..., None]], -1)
    return Q


def _split_step(u, dt, dX, M, S, bc, flux):
    nd = len(dX)
    ub = _ode(_ghosts(u, S.N, bc), dt / 2, M)
    u = _ode(u, dt / 2, M)
    wh = _reconstruct(ub, S)
    w = wh.flatten(0, nd - 1)[:, None]
    inc = -_smooth_rhs(w, dX, M, S, False)
    for d, h in enumerate(dX):
        inc = inc + _along(S.der, _flux(w, d, M), 2 + d) / h
    w = (w - dt / 2 * inc).unflatten(0, wh.shape[:nd])
    return _ode(_update(u, w, dt, dX, M, S, flux, False), dt / 2, M)


def _cfl(u, M, dX):
    return sum(_wave(u, d, M) / h for d, h in enumerate(dX)).max()


def _renorm(u, M):
    A = u[..., 5:14]
    f = (u[..., 0] / (M.rho0 * torch.linalg.det(A.unflatten(-1, (3, 3))))) ** (1 / 3)
    return torch.cat([u[..., :5], A * f[..., None], u[..., 14:]], -1)


def _num(x):
    return float(x.detach()) if isinstance(x, torch.Tensor) else float(x)


def _loop(u, M, dX, bc, S, cfl, tf, flux=0, split=False, steps=10 ** 9, renorm=True, tol=6e-6,
          its=50):
    """The time loop: CFL step (a fifth of it for the first six), scheme,
    renormalised distortion.  Returns the state and its time."""
    t = 0.0
    for n in range(steps):
        if not _num(t) < tf:
            break
        dt = cfl / _cfl(u, M, dX) * (0.2 if n <= 5 else 1.0)
        if _num(t + dt) > tf:
            dt = tf - t
        u = _split_step(u, dt, dX, M, S, bc, flux) if split else \
            _step(u, dt, dX, M, S, bc, flux, tol, its)
        if renorm:
            u = _renorm(u, M)
        t = t + dt
    return u, dt, t, n + 1


def exact(case, seed, device=DEV):
    kind = case["kind"]
    S = _Scheme(case.get("order", 2), device)
    if kind == "bubble":
        return None  # Riemann star states and the marched level set: no plain form
    if kind == "batch":
        if case["count"] > 40:
            return None  # one grid after another: minutes
        us, clk = [], []
        for u, M, dX, bc in _batch_instances(case, seed):
            u, dt, t, n = _loop(torch.tensor(u, device=device), _Mat(M), dX, bc, S, 0.8, 0.2,
                                steps=case["steps"])
            us.append(u.flatten())
            clk += [float(t), float(dt), 0.2, 0.8, float(n)]
        return [torch.cat(us), torch.tensor(clk, dtype=torch.float64)]
    if kind == "adjoint":
        if case["count"] > 1:
            return None  # about ten seconds an instance
        u0, cot = _adjoint_inputs(case, seed, device)
        u0.requires_grad_()
        theta = torch.tensor(_theta(case, seed), device=device, requires_grad=True)
        nx, us = case["nx"], []
        for k in range(case["count"]):
            M = _Mat(_adjoint_par(theta[k].detach().cpu().numpy()), theta[k])
            us.append(_loop(u0[k * nx:(k + 1) * nx], M, [2.0 / nx], TRANSMISSIVE, S, 0.8,
                            case["tf"], tol=1e-13, its=300)[0])
        uN = torch.cat(us)
        uN.backward(cot)
        return [uN.detach(), u0.grad, theta.grad]
    if case["nx"] * max(case["ny"], 1) * case["flux"] > 5000 and case["ny"]:
        return None  # a host eigen-decomposition per face point: minutes
    u, M, dX, bc = _flow(case, seed, device)
    if kind == "iterate":
        return _loop(u, _Mat(M), dX, bc, S, case["cfl"], 1.0, case["flux"], case["split"],
                     case["steps"])[0].flatten()
    wh, qh, un = _step(u, _dt(case, u, M, dX), dX, _Mat(M), S, bc, case["flux"], parts=True)
    return un if kind == "step" else [wh.flatten(), qh.flatten(), un]
