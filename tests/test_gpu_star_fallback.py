"""The interface Riemann solver where the bulk sound speed is imaginary: the
reference takes c_0 = sqrt(...) (waves/speeds.cpp:8-18), so a negative square
makes the step NaN and the input is returned, although the shear part may keep
the acoustic tensor's spectrum real and positive.  Pressures on both sides of
-pINF (a stiffened gas has c_0^2 = gamma (p + pINF) / rho) and a solid in
strong tension, on the left, the right or both sides; decisions equal to the
oracle's; a solved state within 50 times what the oracle itself moves by when
its inputs move by 1e-15, and 1e-10 where that is less."""
import numpy as np
import pytest
import torch

from oracle import Oracle
from phd_gb300.params import Cvec, material_params

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
A0 = np.eye(3) + 0.03 * np.array([[1.0, 0.4, -0.2], [-0.3, -1.0, 0.5], [0.2, 0.1, 0.6]])

GAS = material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=1.0, mu=1e-2)
STIFF = material_params("sg", 1.0, cv=2.5, gamma=2.8, pINF=0.5, b0=0.8, mu=1e-2)
SOLID = material_params("smg", 8.9, cv=4e-4, c0=0.394, Gamma0=2, s=1.48, b0=0.22, tau0=1.0,
                        sigmaY=9e-4, n=10)
# material, pressures with c_0^2 < 0, pressures with c_0^2 > 0
CASES = {"gas": (GAS, (-0.3, -0.02, -1e-4), (1e-2, 0.2, 1.0)),
         "stiffened": (STIFF, (-0.8, -0.52), (-0.45, 0.1, 1.0)),
         "solid": (SOLID, (-2.5, -1.5), (-0.05, 0.1))}


def _state(MP, p, vx, phi):
    A = A0 if MP is not SOLID else A0 * 0.98
    rho = MP.rho0 * np.linalg.det(A)
    return np.concatenate([Cvec(rho, p, np.array([vx, 0.02, -0.01]), MP, A), [phi]])


def _bar(O, ref, ql, qr, ML, MR, dt, n):
    moved = O.left_star_state(ql * (1 + 1e-15), qr * (1 - 1e-15), ML, MR, dt, n)
    return max(1e-10, 50 * np.max(np.abs(moved - ref) / (1 + np.abs(ref))))


@pytest.mark.parametrize("dt", [0.0, 1e-3])
@pytest.mark.parametrize("name", list(CASES))
def test_star_state_with_imaginary_sound_speed(cuda_ok, name, dt):
    import phd_gb300 as G
    O = Oracle(N=2, thermal=False, lset=1)
    MP, neg, pos = CASES[name]
    pairs = [(a, b) for a in neg + pos for b in neg + pos]
    QL = np.stack([_state(MP, a, 0.03, -0.1) for a, _ in pairs])
    QR = np.stack([_state(MP, b, -0.02, 0.1) for _, b in pairs])
    ang = 0.3 + 0.1 * np.arange(len(pairs))
    n = np.stack([np.cos(ang), np.sin(ang)], 1)
    t = [torch.tensor(x, device=DEV) for x in (QL, QR, n)]
    out = G.system.multi.left_star_state(t[0], t[1], MP, MP, dt, t[2]).cpu().numpy()
    solved = 0
    for k, (a, b) in enumerate(pairs):
        ref = O.left_star_state(QL[k], QR[k], MP, MP, dt, n[k])
        back = np.array_equal(ref, QL[k])
        assert back or (a in pos and b in pos), (a, b)
        assert np.array_equal(out[k], QL[k]) == back, (a, b)
        if not back:
            solved += 1
            err = np.max(np.abs(out[k] - ref) / (1 + np.abs(ref)))
            assert err < _bar(O, ref, QL[k], QR[k], MP, MP, dt, n[k]), (a, b, err)
    assert solved > 0


def test_star_state_at_a_vacuum(cuda_ok):
    """One material only: the left side alone decides."""
    import phd_gb300 as G
    O = Oracle(N=2, thermal=False, lset=1)
    vac = material_params("vac", 1.0)
    ps = CASES["gas"][1] + CASES["gas"][2]
    QL = np.stack([_state(GAS, p, 0.03, -0.1) for p in ps])
    n = np.tile([0.6, 0.8], (len(ps), 1))
    t = [torch.tensor(x, device=DEV) for x in (QL, 0 * QL, n)]
    out = G.system.multi.left_star_state(t[0], t[1], GAS, vac, 1e-3, t[2]).cpu().numpy()
    for k, p in enumerate(ps):
        ref = O.left_star_state(QL[k], 0 * QL[k], GAS, vac, 1e-3, n[k])
        assert np.array_equal(ref, QL[k]) == np.array_equal(out[k], QL[k]), p
        err = np.max(np.abs(out[k] - ref) / (1 + np.abs(ref)))
        assert err < _bar(O, ref, QL[k], 0 * QL[k], GAS, vac, 1e-3, n[k]), (p, err)
