"""Wave speeds along y and z at O(0.1) distortions, and along every axis where the
shear speed depends on the density (beta != 0), with and without heat
conduction, against the oracle.

Bar: the largest root l of the tensor's characteristic polynomial, whose
coefficients are sums of principal minors, is determined to the rounding of
those sums' terms over |p'(l)|: with T = sum_k (sum of the permanents of |X|'s
principal minors of order k) l^(m - k), 64 roundings of T, halved by the root
that gives the speed; and 64 roundings of the speed itself."""
from itertools import combinations, permutations

import numpy as np
import pytest
import torch

from oracle import Oracle
from phd_gb300.params import Cvec, material_params

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _material(name, th):
    ca = 1.0 if th else None
    if name == "gas":
        return material_params("sg", 1.0, cv=2.5, gamma=1.4, b0=1.0, mu=1e-2, calpha=ca, Pr=0.67), 1.0
    if name == "smg":
        return material_params("smg", 8.9, cv=4e-4, c0=0.394, Gamma0=2, s=1.48, b0=0.22, tau0=1.0,
                               sigmaY=9e-4, n=10, calpha=0.1 if th else None, kappa=1e-3), 0.3
    return material_params("gr", 2.7, cv=9e-4, c0=0.5, alpha=1, beta=3.577, gamma=2.0, b0=0.3,
                           tau0=1.0, sigmaY=9e-4, n=10, calpha=0.1 if th else None, kappa=1e-3), 0.3


def _states(MP, p0, V, amp, n):
    rng = np.random.default_rng(17)
    out = []
    for _ in range(n):
        rho = MP.rho0 * rng.uniform(0.9, 1.1)
        A = (rho / MP.rho0) ** (1 / 3) * (np.eye(3) + amp * rng.standard_normal((3, 3)))
        out.append(Cvec(rho, p0 * rng.uniform(0.8, 1.2), 0.3 * rng.standard_normal(3) * np.sqrt(MP.b02),
                        MP, A, 0.1 * rng.standard_normal(3) if V == 17 else None))
    return np.array(out)


def _permanents(X):
    m = len(X)
    return [sum(sum(np.prod([X[s[i], s[p[i]]] for i in range(k)]) for p in permutations(range(k)))
                for s in combinations(range(m), k)) for k in range(m + 1)]


def _bar(X, lam, speed):
    m, l = len(X), lam * lam
    T = sum(e * l ** (m - k) for k, e in enumerate(_permanents(np.abs(X))))
    dp = abs(np.polyval(np.polyder(np.poly(X)), l))
    return 64 * 2.0 ** -53 * (0.5 * T / (dp * l) * lam + speed)


@pytest.mark.parametrize("V", [17, 14])
@pytest.mark.parametrize("name,amp", [("gas", 0.1), ("smg", 0.1), ("gr", 0.0), ("gr", 1e-6),
                                      ("gr", 1e-3), ("gr", 0.1)])
def test_wave_speed_along_each_axis(cuda_ok, name, V, amp):
    import phd_gb300 as G
    MP, p0 = _material(name, V == 17)
    O = Oracle(thermal=V == 17)
    Q = _states(MP, p0, V, amp, 65)
    for d in range(3):
        got = G.system.max_abs_eigs(torch.tensor(Q, device=DEV), d, MP).cpu().numpy()
        for q, s in zip(Q, got):
            ref = O.max_abs_eigs(q, d, MP)
            X = O.thermo_acoustic_tensor(q, d, MP)
            bar = _bar(X, ref - abs(q[2 + d] / q[0]), ref)
            assert bar < 1e-6 * ref and abs(s - ref) <= bar, (d, abs(s - ref) / ref, bar / ref)
