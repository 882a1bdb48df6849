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
