"""The one-call step of `solvers.iterator`: its NaN flag at the edges of the
kernel's blocks, the loop against the same stages called one by one (the same
kernels on the same inputs: equal to the last bit but for the roundings that
the clock's two forms may differ in, 1e-13 of the largest entry), its early
exit on a NaN and the arguments that it refuses."""
import numpy as np
import pytest
import torch

from phd_gb300.params import Cvec, material_params

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _gas():
    return material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=1.0, mu=1e-2, calpha=1.0, Pr=0.67)


def _tube(nX, MP):
    n = int(np.prod(nX))
    left, right = (np.asarray(Cvec(r, p, np.zeros(3), MP, r ** (1 / 3) * np.eye(3), np.zeros(3)))
                   for r, p in ((1.0, 1.0), (0.8, 0.7)))
    u = np.where(np.arange(n)[:, None] // max(n // nX[0], 1) < nX[0] // 2, left, right)
    return torch.tensor(u, dtype=torch.float64, device=DEV)


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 152 * 4 * 256 + 1, 1000003])
def test_any_nan(cuda_ok, n):
    from phd_gb300 import _lib, api
    lib = _lib.load()

    def flag(u, start=0.0):
        f = torch.full((1,), start, dtype=torch.float64, device=DEV)
        _lib.check(lib.gpr_any_nan(api._dev(u, "u"), u.numel(), api._dev(f, "f"), api._stream()),
                   "any_nan")
        return f.item()

    u = torch.zeros(n, dtype=torch.float64, device=DEV)
    u[n // 2], u[n - 1] = float("inf"), -float("inf")
    assert flag(u) == 0.0 and flag(u, 1.0) == 1.0
    for i in {0, n // 2, n - 1}:
        for bad in (float("nan"), -float("nan")):
            v = u.clone()
            v[i] = bad
            assert flag(v) == 1.0
    assert lib.gpr_any_nan(api._dev(u, "u"), 0, api._dev(u, "f"), None) < 0


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("nX", [(1,), (67,), (9, 5)])
def test_loop_against_stages(cuda_ok, nX, split):
    from phd_gb300 import api, driver
    MP = _gas()
    dX, bcs = [1.0 / n for n in nX], [0] * (2 * len(nX))
    a, b = _tube(nX, MP), _tube(nX, MP)
    steps, tf = 8, 10.0
    driver.iterate(a, tf, nX, dX, 0.6, bcs, SPLIT=split, MPs=MP, max_steps=steps)
    st, t = driver.Stepper(nX, 17, device=DEV), 0.0
    for count in range(steps):
        dt = float(api.timestep_device(b.view(-1), dX, 0.6, t, tf, count, MP, out=st.dt).item())
        st.step(b.view(-1), dt, dX, bcs, MP, split=split, contorted_tol=1.0)
        t += dt
    assert float((a - b).abs().max() / b.abs().max()) < 1e-13


def test_loop_stops_at_a_nan_and_refuses(cuda_ok):
    from phd_gb300 import driver
    MP = _gas()
    u = _tube((40,), MP)
    u[7, 3] = float("nan")
    before = u.clone()
    ret = driver.iterate(u.view(-1), 1.0, [40], [0.025], 0.6, [0, 0], MPs=MP)
    assert torch.equal(torch.nan_to_num(ret[0].view(40, 17)), torch.nan_to_num(before))
    assert ret[1] is not None and all(r is None for r in ret[2:])
    with pytest.raises(ValueError):
        driver.iterate(torch.zeros(40 * 17 + 3, dtype=torch.float64, device=DEV), 1.0, [40],
                       [0.025], 0.6, [0, 0], MPs=MP)
    with pytest.raises(ValueError):
        driver.iterate(_tube((40,), MP).view(-1), 1.0, [40], [0.025], 0.6, [0], MPs=MP)
