"""The resident loop on masks: it reconstructs only the masked-on cells and
leaves whole warps of the others out, so its steps are compared with the
stages called one by one, whose reconstruction covers every cell (the same
kernels on the same inputs: 1e-13 of the largest entry for the clock's
roundings), with the scratch filled by NaN beforehand.  Masks: nothing,
everything, single cells at the corners, a disc, columns that end inside a
reconstruction block, noise."""
import numpy as np
import pytest
import torch

from phd_gb300 import problems

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _masks(nxp, nyp):
    i, j = np.meshgrid(np.arange(nxp), np.arange(nyp), indexing="ij")
    rng = np.random.default_rng(5)
    corner = np.zeros((nxp, nyp), bool)
    corner[[0, 0, -1, -1, 3], [0, -1, 0, -1, 61 % nyp]] = True
    return {"none": i < 0, "all": i >= 0, "corners": corner,
            "disc": (i - nxp / 2) ** 2 + (j - nyp / 2) ** 2 < (min(nxp, nyp) / 3) ** 2,
            "columns": (j % 61 < 30) & (i % 5 < 4), "noise": rng.uniform(size=i.shape) < 0.4}


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("nx,ny", [(11, 7), (19, 131)])
@pytest.mark.parametrize("kind", ["none", "all", "corners", "disc", "columns", "noise"])
def test_masked_loop(cuda_ok, kind, nx, ny, split):
    from phd_gb300 import _lib, api
    lib = _lib.load()
    u0, MP, _, dX, _ = problems.taylor_green(n=nx, ny=ny, cs=10.0, mu=0.5)
    nX, bcs, V, steps = np.array([nx, ny], np.int32), [1] * 4, 17, 3
    api.set_nvar(V)
    mask = torch.tensor(_masks(nx + 2, ny + 2)[kind].astype(np.uint8).ravel(), device=DEV)
    a = torch.tensor(u0.ravel(), dtype=torch.float64, device=DEV)
    b = a.clone()
    (nXa, pn), (dXa, pd), (bca, pb) = api._i32(nX), api._f64(dX), api._i32(bcs)
    c, pp = api._par(MP)
    scr = torch.full((int(lib.gpr_iterate_scratch_doubles(pn, 2, V)),), float("nan"),
                     dtype=torch.float64, device=DEV)
    clk = torch.tensor([0.0, 0.0, 10.0, 0.3, 0.0], dtype=torch.float64, device=DEV)
    pm, tol = api._dev(mask, "mask", torch.uint8), float("inf")
    if split:
        rc = lib.gpr_iterate_split(api._dev(a, "u"), pn, 2, pd, pb, 0, 1, pp, pm,
                                   api._dev(clk, "c"), steps, api._dev(scr, "s"), tol, V, None)
    else:
        rc = lib.gpr_iterate(api._dev(a, "u"), pn, 2, pd, pb, 0, pp, pm, api._dev(clk, "c"),
                             steps, api._dev(scr, "s"), None, tol, V, None)
    _lib.check(rc, "iterate")
    dt = torch.empty(1, dtype=torch.float64, device=DEV)
    ub = torch.empty(int(np.prod(nX + 4)) * V, dtype=torch.float64, device=DEV)
    t = 0.0
    for k in range(steps):
        h = float(api.timestep_device(b, dX, 0.3, t, 10.0, k, MP, out=dt).item())
        api.boundaries(b, ub, nX, bcs)
        if split:
            wh = torch.empty((nx + 2) * (ny + 2) * 4 * V, dtype=torch.float64, device=DEV)
            api.ode_launcher(b, h / 2, MP)
            api.ode_launcher(ub, h / 2, MP)
            api.weno_launcher(wh, ub, nX)
            api.midstepper(wh, h, dX, MP, mask, nX=nX)
            api.fv_launcher(b, wh, nX, h, dX, False, False, 0, MP, mask)
            api.ode_launcher(b, h / 2, MP)
        else:
            api.ader_stepper(b, ub, nX, h, dX, False, 0, MP, mask)
        api.renorm_distortion(b, [MP])
        t += h
    assert torch.isfinite(a).all()
    assert float((a - b).abs().max() / b.abs().max()) < 1e-13
