"""The Osher faces that the closed form declines: marked by k_faces1d_osher and
evaluated by k_faces1d_eigw, per thread in k_faces2d_osher, and all of them
where heat conduction meets a density-dependent shear speed (no closed form).

Face stages (interfs1 / interfs2) against the oracle.  Negative pressures give an
acoustic eigenvalue that is not positive (a pair of complex wave speeds), which
the closed form refuses; the declining cells lie at each place of the four-lane
groups and 32-lane warps, beside cells that it takes.  Bar: the oracle's and
numpy's decompositions of these states agree to 1e-14 of the largest entry and
a stage moves by 1e-13 when its nodes move by 1e-15; 1e-10 of a cell's largest
entry leaves three digits for another decomposition, and a face that is left
out, stale or taken from a neighbour is off by more than 1e-3."""
import numpy as np
import pytest
import torch

from oracle import Oracle
from phd_gb300.params import Cvec, material_params

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def _default_layout():
    yield
    from phd_gb300 import api
    api.set_nvar(17)


def _material(name, th):
    ca = 1.0 if th else None
    if name == "gas":
        return material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=1.0, mu=1e-2, calpha=ca, Pr=0.67)
    return material_params("gr", 2.7, cv=9e-4, c0=0.5, alpha=1, beta=3.577, gamma=2.0, b0=0.3,
                           tau0=1.0, sigmaY=9e-4, n=10, calpha=0.1 if th else None, kappa=1e-3)


def _values(MP, V, n, neg, seed):
    """n states; those with neg have a negative pressure."""
    rng = np.random.default_rng(seed)
    Q = np.zeros((n, V))
    for i in range(n):
        A = np.eye(3) + 0.06 * rng.standard_normal((3, 3))
        rho = MP.rho0 * np.linalg.det(A)
        p = rng.uniform(-4.0, -3.0) if neg[i] else rng.uniform(0.8, 1.2)
        c = Cvec(rho, p, 0.3 * rng.standard_normal(3), MP, A,
                 0.05 * rng.standard_normal(3) if V == 17 else None)
        Q[i, :len(c)] = c
    return Q


def _declines(O, q, MP):
    """A system matrix whose eigenvalues along x are not all real."""
    lam = np.linalg.eigvals(O.system_matrix(q, 0, MP))
    return np.any(np.abs(lam.imag) > 1e-2)


def _rel(a, b, V):
    """Largest difference over the largest entry, cell by cell."""
    a, b = a.reshape(-1, V), b.reshape(-1, V)
    return np.max(np.max(np.abs(a - b), axis=1) / np.max(np.abs(b), axis=1))


def _stage(O, qh, nX, MP, time, mask, dX, dt):
    from phd_gb300 import api
    import phd_gb300 as G
    V = O.V
    u0 = np.zeros(int(np.prod(nX)) * V)
    ref = O.fv_parts(u0.copy(), qh, nX, dt, dX, MP, 2, mask=mask, time=time, flux=2)
    api.set_nvar(V)
    api.set_grid(nX)
    u, q = torch.tensor(u0, device=DEV), torch.tensor(qh, device=DEV)
    m = torch.tensor(mask, device=DEV)
    if len(nX) == 1:
        G.solvers.fv.interfs1(u, q, int(nX[0]), dt, dX[0], time, 2, MP, m)
    else:
        G.solvers.fv.interfs2(u, q, int(nX[0]), int(nX[1]), dt, dX[0], dX[1], time, 2, MP, m)
    return u.cpu().numpy(), ref


def _nodes(Q, NS, nt, seed):
    """Node values of each cell: its state, varied a little from node to node."""
    rng = np.random.default_rng(seed)
    n, V = Q.shape
    return np.ascontiguousarray(
        Q[:, None, :] * (1 + 1e-3 * rng.standard_normal((n, nt * NS, V)))).ravel()


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("time", [True, False])
@pytest.mark.parametrize("V", [17, 14])
@pytest.mark.parametrize("nx", [1, 8, 70])
def test_marked_faces_1d(cuda_ok, nx, V, time, masked):
    O, MP = Oracle(thermal=V == 17), _material("gas", V == 17)
    nX = np.array([nx], np.int32)
    neg = (np.arange(nx + 2) * 7 % 11) < 3
    Q = _values(MP, V, nx + 2, neg, 31)
    gone = [_declines(O, Q[i + 1] + x * (Q[i] - Q[i + 1]), MP) for i in range(nx + 1)
            for x in (0.2113, 0.7887)]
    assert any(gone) and not all(gone)
    mask = np.ones(nx + 2, np.uint8)
    if masked:
        mask[::5] = 0
    got, ref = _stage(O, _nodes(Q, 2, 2 if time else 1, 32), nX, MP, time, mask, [1.0 / nx],
                      0.1 / nx)
    on = np.any(ref.reshape(-1, V) != 0, axis=1)
    assert np.all(got.reshape(-1, V)[~on] == 0)
    if on.any():
        assert _rel(got.reshape(-1, V)[on], ref.reshape(-1, V)[on], V) < 1e-10


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("V,time", [(17, True), (17, False), (14, True)])
@pytest.mark.parametrize("nx,ny", [(1, 3), (9, 6)])
def test_declined_points_2d(cuda_ok, nx, ny, V, time, masked):
    O, MP = Oracle(thermal=V == 17), _material("gas", V == 17)
    nX = np.array([nx, ny], np.int32)
    n = (nx + 2) * (ny + 2)
    neg = (np.arange(n) * 7 % 11) < 3
    Q = _values(MP, V, n, neg, 33)
    assert any(_declines(O, q, MP) for q in Q) and not all(_declines(O, q, MP) for q in Q)
    mask = np.ones(n, np.uint8)
    if masked:
        mask[::5] = 0
    got, ref = _stage(O, _nodes(Q, 4, 2 if time else 1, 34), nX, MP, time, mask, [0.1, 0.13],
                      0.01)
    on = np.any(ref.reshape(-1, V) != 0, axis=1)
    assert np.all(got.reshape(-1, V)[~on] == 0)
    if on.any():
        assert _rel(got.reshape(-1, V)[on], ref.reshape(-1, V)[on], V) < 1e-10


@pytest.mark.parametrize("nX", [(9,), (5, 4)])
def test_conduction_with_a_density_dependent_shear_speed(cuda_ok, nX):
    """No closed form for any point of this material."""
    O, MP = Oracle(), _material("gr", True)
    nX = np.array(nX, np.int32)
    n = int(np.prod(nX + 2))
    Q = _values(MP, 17, n, np.zeros(n, bool), 35)
    got, ref = _stage(O, _nodes(Q, 2 ** len(nX), 2, 36), nX, MP, True, np.ones(n, np.uint8),
                      [0.1, 0.13][:len(nX)], 0.01)
    assert _rel(got, ref, 17) < 1e-10
