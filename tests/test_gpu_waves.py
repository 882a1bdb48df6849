"""Wave speeds by the short root iteration and the Osher dissipation in closed
form, at the states where their branches meet: isotropic distortion (equal
shear speeds), distortions from rounding level to O(0.1), sub- and supersonic
flow, a heat wave 1e-4 of the sound speed, and the states that the general
routines take (heat conduction with a density-dependent shear speed).

Bars.  Along x the acoustic tensor is similar to a symmetric matrix, so its
largest eigenvalue is determined to a few roundings: 1e-13.  Along y and z
the reference's tensor is not symmetric (its pressure and density entries
stay in row and column 0) and an eigenvalue moves by the rounding times
about c0^2 / cs^2 and the inverse relative gap: 1e-11 for distortions up to
1e-3, where the dominant root is real and separated.  A 17 x 17
eigen-decomposition carries its eigenvectors' conditioning, about 1e3
roundings at these scales: 1e-11 of the largest flux entry.  Two are compared
with, along x on states with the axes exchanged (the system is invariant), and
each state is held to the nearer: the oracle's, and numpy's of the balanced
system matrix.  Either can lose more where eigenvalues coincide (against 40
digits: the oracle's 2e-11 in the fast smg flow and 1e-3 along z at an
isotropic distortion, numpy's 7e-11 in a fluid at rest; the closed form
stays within 1e-12)."""
import numpy as np
import pytest
import torch
from scipy.linalg import matrix_balance

from phd_gb300.params import Cvec, material_params

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _material(name, th):
    ca = 1.0 if th else None
    if name == "gas":
        return material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=1.0, mu=1e-2, calpha=ca, Pr=0.67), 1.0
    if name == "slow_heat":
        return material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=1.0, mu=1e-2,
                               calpha=1e-4 if th else None, Pr=0.67), 1.0
    if name == "smg":
        return material_params("smg", 8.9, cv=4e-4, c0=0.394, Gamma0=2, s=1.48, b0=0.22, tau0=1.0,
                               sigmaY=9e-4, n=10, calpha=0.1 if th else None, kappa=1e-3), 0.3
    return material_params("gr", 2.7, cv=9e-4, c0=0.5, alpha=1, beta=3.577, gamma=2.0, b0=0.3,
                           tau0=1.0, sigmaY=9e-4, n=10, calpha=0.1 if th else None, kappa=1e-3), 0.3


def _states(MP, p0, V, amp, jump, mach, n, seed):
    rng = np.random.default_rng(seed)
    out = []
    v0 = rng.standard_normal((n, 3)) * mach * np.sqrt(MP.b02)
    for side in range(2):
        Q = np.zeros((n, V))
        for i in range(n):
            rho = MP.rho0 * (1 + jump * rng.uniform(-1, 1))
            A = (rho / MP.rho0) ** (1 / 3) * (np.eye(3) + amp * rng.standard_normal((3, 3)))
            c = Cvec(rho, p0 * (1 + jump * rng.uniform(-1, 1)),
                     v0[i] * (1 + jump * rng.uniform(-1, 1)), MP, A,
                     0.1 * amp * rng.standard_normal(3) if V == 17 else None)
            Q[i, :len(c)] = c
        out.append(Q)
    return out


@pytest.mark.parametrize("V", [17, 14])
@pytest.mark.parametrize("name", ["gas", "slow_heat", "smg"])
@pytest.mark.parametrize("amp", [0.0, 1e-12, 1e-6, 1e-3, 0.1])
def test_wave_speed(V, name, amp):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import phd_gb300 as G
    from oracle import Oracle
    MP, p0 = _material(name, V == 17)
    O = Oracle(thermal=V == 17)
    Q = _states(MP, p0, V, amp, 0.1, 0.5, 65, 1)[0]
    for d in range(3):
        if d and amp > 1e-3:
            continue
        got = G.system.max_abs_eigs(torch.tensor(Q, device=DEV), d, MP).cpu().numpy()
        ref = np.array([O.max_abs_eigs(q, d, MP) for q in Q])
        err = np.max(np.abs(got - ref) / np.abs(ref))
        assert err < (1e-13 if d == 0 else 1e-11), (d, err)


def _exchange(V, d):
    """The state entries with the axes 0 and d exchanged."""
    def s(a):
        return d if a == 0 else (0 if a == d else a)
    idx = list(range(V))
    for k in range(3):
        idx[2 + k] = 2 + s(k)
        if V == 17:
            idx[14 + k] = 14 + s(k)
        for c in range(3):
            idx[5 + 3 * k + c] = 5 + 3 * s(k) + s(c)
    return idx


def _osher(O, ql, qr, MP):
    """D_OSH along x: two Gauss nodes of |M| (qL - qR), plus both fluxes, by
    numpy's decomposition of the balanced system matrix (None where it has no
    eigenvector basis)."""
    f = O.flux(ql, 0, MP) + O.flux(qr, 0, MP)
    dq = ql - qr
    for x in (0.5 - 0.5 / np.sqrt(3), 0.5 + 0.5 / np.sqrt(3)):
        M, (D, _) = matrix_balance(O.system_matrix(qr + x * dq, 0, MP), permute=False,
                                   separate=True)
        lam, R = np.linalg.eig(M)
        if not np.linalg.cond(R) <= 1e6:
            return None
        f = f + 0.5 * D * (R @ (np.abs(lam) * np.linalg.solve(R, dq / D + 0j))).real
    return f


@pytest.mark.parametrize("V", [17, 14])
@pytest.mark.parametrize("name", ["gas", "slow_heat", "smg", "gr"])
@pytest.mark.parametrize("amp,jump,mach", [(0.0, 0.1, 0.0), (0.0, 0.1, 0.5), (1e-9, 1e-2, 0.3),
                                           (1e-3, 1e-2, 1.0), (0.03, 0.3, 3.0)])
def test_osher_closed_form(V, name, amp, jump, mach):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import phd_gb300 as G
    from oracle import Oracle
    MP, p0 = _material(name, V == 17)
    O = Oracle(thermal=V == 17)
    QL, QR = _states(MP, p0, V, amp, jump, mach, 33, 2)
    for d in range(3):
        got = G.solvers.fv.D_OSH(torch.tensor(QL, device=DEV), torch.tensor(QR, device=DEV), d,
                                 MP).cpu().numpy()
        ix = _exchange(V, d)
        for i in range(len(QL)):
            ql, qr = QL[i, ix].copy(), QR[i, ix].copy()
            refs = [r for r in (_osher(O, ql, qr, MP), O.D(2, ql, qr, 0, MP)) if r is not None]
            err = min(np.max(np.abs(got[i, ix] - r)) / np.max(np.abs(r)) for r in refs)
            assert err < 1e-11, (d, i, err)


@pytest.mark.parametrize("flux", [1, 2])
@pytest.mark.parametrize("nx", [1, 7, 8, 33])
def test_1d_step_flux_edges(flux, nx):
    """The 1D face kernels at the edges of their lane groups and blocks, with
    flat faces (qL = qR) among the others."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import phd_gb300 as G
    from oracle import Oracle
    MP, p0 = _material("gas", True)
    u0 = _states(MP, p0, 17, 0.02, 0.2, 0.3, nx, 3)[0]
    u0[nx // 2:] = u0[nx // 2]
    nX = np.array([nx], dtype=np.int32)
    dX, dt = [1.0 / nx], 0.05 / nx
    u = torch.tensor(u0.ravel(), device=DEV)
    ub = torch.empty((nx + 4) * 17, dtype=torch.float64, device=DEV)
    mask = torch.ones(nx + 2, dtype=torch.bool, device=DEV)
    G.boundaries(u, ub, nX, [0, 0])
    G.solvers.ader_stepper(u, ub, nX, dt, dX, False, flux, MP, mask)
    O = Oracle()
    ref = u0.ravel().copy()
    O.ader_stepper(ref, O.boundaries(u0, nX, [0, 0]), nX, dt, dX, MP, flux=flux)
    assert np.max(np.abs(u.cpu().numpy() - ref) / (1 + np.abs(ref))) < 1e-11
