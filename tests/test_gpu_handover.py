"""Which cells the Picard pass hands to the Newton pass early: vortices and
shock tubes from the relaxation time well above the step to well below it,
where cells converge in 4 to 50 iterations, grow, or settle into
oscillations.  Every cell that the oracle's iteration converges has to
converge on the device with the oracle's count (one more or less where an
update meets its threshold within rounding), and no cell that the oracle
gives up may be called converged (but for the last iteration, for the same
reason)."""
import numpy as np
import pytest
import torch

from oracle import Oracle
from phd_gb300 import problems

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

CASES = [("vortex", mu) for mu in (0.05, 0.1, 0.2, 0.4)] + \
        [("tube", mu) for mu in (1e-5, 1e-4, 1e-3)]


def _reconstruction(kind, mu):
    O = Oracle()
    if kind == "vortex":
        u0, MP, _, dX, _ = problems.taylor_green(n=24, cs=10.0, mu=mu)
        nX, bcs = [24, 24], [1] * 4
    else:
        u0, MP, _, dX, _ = problems.shock_tube(nx=200, mu=mu)
        nX, bcs = [200], [0, 0]
    u, _, _ = O.run(u0, MP, 1e9, dX, bcs, cfl=0.3, max_steps=3)
    nX = np.array(nX, np.int32)
    wh = O.weno_launcher(O.boundaries(u, nX, bcs), nX)
    dt1 = O.timestep(u, dX, 1.0, 0.0, 1e9, 10, MP)
    return O, wh, dt1, nX, dX, MP


@pytest.mark.parametrize("kind,mu", CASES)
def test_handover_against_oracle(cuda_ok, kind, mu):
    from phd_gb300 import api
    O, wh, dt1, nX, dX, MP = _reconstruction(kind, mu)
    ncb = int(np.prod(nX + 2))
    mask = torch.ones(ncb, dtype=torch.uint8, device=DEV)
    api.set_nvar(17)
    api.set_grid(nX)
    for cfl in (0.3, 0.5, 0.7, 0.8, 0.95):
        _, ref = O.predictor(wh, cfl * dt1, dX, nX, MP, newton_fallback=False)
        qh = torch.empty(ncb * 2 ** (len(nX) + 1) * 17, dtype=torch.float64, device=DEV)
        status = torch.full((ncb,), -1, dtype=torch.int32, device=DEV)
        api.predictor(qh, torch.tensor(wh, device=DEV), cfl * dt1, dX, False, False, MP, mask,
                      status=status)
        st = status.cpu().numpy()
        picard, its = (st & 0xff) == 0, st >> 8
        sure = (ref > 0) & (ref < 49)
        assert picard[sure].all(), (cfl, ref[sure & ~picard], st[sure & ~picard])
        assert (np.abs(its - ref)[sure] <= 1).all(), cfl
        assert (its[picard & (ref <= 0)] >= 50).all(), cfl
