"""The 2D Roe faces at the edges of their lane groups, warps and blocks (a point per
lane, four to a face, 64 to a block): the face stage against the oracle, with
masks, without time nodes, and the sums it leaves in the caller's buffer.  Bar:
as test_gpu_osher_handover's, 1e-10 of a cell's largest entry."""
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


def _nodes(MP, V, ncb, nt):
    rng = np.random.default_rng(41)
    Q = np.zeros((ncb, V))
    for i in range(ncb):
        A = np.eye(3) + 0.06 * rng.standard_normal((3, 3))
        c = Cvec(MP.rho0 * np.linalg.det(A), rng.uniform(0.8, 1.2), 0.3 * rng.standard_normal(3), MP,
                 A, 0.05 * rng.standard_normal(3) if V == 17 else None)
        Q[i, :len(c)] = c
        if V == 15:
            Q[i, 14] = rng.uniform(-1, 1)
    return np.ascontiguousarray(
        Q[:, None, :] * (1 + 1e-3 * rng.standard_normal((ncb, nt * 4, V)))).ravel()


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("V,time", [(17, True), (17, False), (15, True), (14, True)])
@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 3), (3, 3), (9, 6), (5, 17)])
def test_roe_faces(cuda_ok, nx, ny, V, time, masked):
    from phd_gb300 import api
    import phd_gb300 as G
    MP = material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=1.0, mu=1e-2,
                         calpha=1.0 if V == 17 else None, Pr=0.67)
    O = Oracle(thermal=V == 17, lset=int(V == 15))
    nX, ncb, dX, dt = np.array([nx, ny], np.int32), (nx + 2) * (ny + 2), [0.1, 0.13], 0.01
    qh = _nodes(MP, V, ncb, 2 if time else 1)
    mask = np.ones(ncb, np.uint8)
    if masked:
        mask[::5] = 0
    ref = O.fv_parts(np.zeros(nx * ny * V), qh, nX, dt, dX, MP, 2, mask=mask, time=time,
                     flux=1).reshape(-1, V)
    api.set_nvar(V)
    api.set_grid(nX)
    u = torch.zeros(nx * ny * V, dtype=torch.float64, device=DEV)
    G.solvers.fv.interfs2(u, torch.tensor(qh, device=DEV), nx, ny, dt, dX[0], dX[1], time, 1, MP,
                          torch.tensor(mask, device=DEV))
    got = u.cpu().numpy().reshape(-1, V)
    scale = np.max(np.abs(ref), axis=1)
    assert np.all(got[scale == 0] == 0)
    err = np.max(np.abs(got - ref), axis=1)[scale > 0] / scale[scale > 0]
    assert err.size == 0 or err.max() < 1e-10, err.max()


def _mirrored(MP, V, n):
    """States, and what a symmetric wall along x makes of them (bc code 5)."""
    rng = np.random.default_rng(43)
    Q = np.zeros((n, V))
    for i in range(n):
        A = np.eye(3) + 0.05 * rng.standard_normal((3, 3))
        c = Cvec(np.linalg.det(A), rng.uniform(0.8, 1.2), 0.2 * rng.standard_normal(3), MP, A)
        Q[i, :len(c)] = c
        if V == 15:
            Q[i, 14] = rng.uniform(-1, 1)
    W = Q.copy()
    W[:, 2] *= -1
    for k in range(5, 14):
        if ((k - 5) // 3 == 0) != ((k - 5) % 3 == 0):
            W[:, k] *= -1
    return Q, W


def _share(got, ref):
    """The share of rows within 1e-10 of their largest entry."""
    return np.mean(np.max(np.abs(got - ref), axis=1) < 1e-10 * np.max(np.abs(ref), axis=1))


@pytest.mark.parametrize("V", [14, 15])
def test_roe_at_a_symmetric_wall(cuda_ok, V):
    """Between a state and its mirror image Roe's average matrix has a zero
    eigenvalue that is not semisimple: |M| has one value for v -> 0+ and another
    for v -> 0-, and the sign of a rounding error must not choose (mass would
    cross the wall, 1e-5 .. 1e-3 of the jump).  The reference's value is that
    of independent vectors; the oracle's own moves by more than 1e-10 in an
    eighth of these faces when the states move by 1e-15, so three quarters
    of them have to agree to 1e-10, and all have to hold the mass back.
    Pointwise (the 2D kernel's routine) and in the 1D kernel."""
    from phd_gb300 import api
    import phd_gb300 as G
    MP = material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=1.0, mu=1e-2)
    O = Oracle(thermal=False, lset=int(V == 15))
    Q, W = _mirrored(MP, V, 64)
    for d in (0, 1):
        ix = list(range(V))
        if d:  # the same wall along y: axes 0 and 1 exchanged
            ix[2], ix[3] = 3, 2
            for k in range(9):
                ix[5 + k] = 5 + 3 * [1, 0, 2][k // 3] + [1, 0, 2][k % 3]
        ql, qr = Q[:, ix], W[:, ix]
        got = G.solvers.fv.D_ROE(torch.tensor(ql, device=DEV), torch.tensor(qr, device=DEV), d,
                                 MP).cpu().numpy()
        ref = np.array([O.D(1, a, b, d, MP) for a, b in zip(ql, qr)])
        assert np.mean(np.abs(got[:, 0]) < 1e-12) > 0.75
        assert _share(got, ref) > 0.75
    # 1D: cells q0, its image, q1, its image, ...; every other face is a wall
    cells = np.stack([Q, W], 1).reshape(-1, V)
    nX, dX, dt = np.array([len(cells) - 2], np.int32), [0.1], 0.01
    qh = np.ascontiguousarray(np.repeat(cells, 4, axis=0).ravel())
    api.set_nvar(V)
    api.set_grid(nX)
    u = torch.zeros(nX[0] * V, dtype=torch.float64, device=DEV)
    mask = np.zeros(len(cells), np.uint8)
    for first in (0, 2):  # one wall face beside each unmasked cell
        mask[:] = 0
        mask[first::4] = mask[first + 1::4] = 1
        u.zero_()
        G.solvers.fv.interfs1(u, torch.tensor(qh, device=DEV), int(nX[0]), dt, dX[0], True, 1, MP,
                              torch.tensor(mask, device=DEV))
        got = u.cpu().numpy().reshape(-1, V)
        ref = O.fv_parts(np.zeros(nX[0] * V), qh, nX, dt, dX, MP, 2, mask=mask, time=True,
                         flux=1).reshape(-1, V)
        on = np.max(np.abs(ref), axis=1) > 0
        assert on.sum() >= 60 and np.all(got[~on] == 0)
        assert np.mean(np.abs(got[on, 0]) < 1e-12) > 0.75
        assert _share(got[on], ref[on]) > 0.75
