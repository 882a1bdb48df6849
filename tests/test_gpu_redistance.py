"""Re-distancing on 2D grids against the oracle's marcher bit for bit: grids
of a few cells, of one row of segments, with a last segment that is cut, with
more segments than one pass of a block reads, and with rows of a whole number
of segment groups; a smooth front (few points wait at a time) and noise (most
points do)."""
import numpy as np
import pytest
import torch

from oracle import Oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

SHAPES = [(3, 3), (3, 41), (41, 3), (15, 17), (16, 16), (17, 33), (5, 2433), (131, 67),
          (400, 399), (130, 1216)]


def _phi(nx, ny, kind, seed=7):
    rng = np.random.default_rng(seed)
    if kind == "noise":
        return rng.uniform(-1, 1, (nx, ny)) + 0.3
    x, y = np.meshgrid((np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / ny, indexing="ij")
    return np.minimum(np.hypot(x - 0.31, y - 0.57) - 0.23, 0.4 - x + 0.1 * np.sin(9 * y))


def _check(nx, ny, kind):
    import phd_gb300
    dX = [1.0 / max(nx, ny), 1.3 / max(nx, ny)]
    nX = np.array([nx, ny], np.int32)
    phi = np.ascontiguousarray(_phi(nx, ny, kind).ravel())
    st = torch.zeros(4, dtype=torch.int32, device=DEV)
    d = phd_gb300.system.multi.distance(torch.tensor(phi, device=DEV), dX, nX, status=st)
    d = d.cpu().numpy()
    assert st.cpu().numpy()[0] == 0
    ref = Oracle().distance(phi, dX, nX)
    assert np.array_equal(d, ref), np.max(np.abs(d - ref))


@pytest.mark.parametrize("kind", ["front", "noise"])
@pytest.mark.parametrize("nx,ny", SHAPES)
def test_distance(cuda_ok, nx, ny, kind):
    _check(nx, ny, kind)


def test_distance_of_a_large_grid(cuda_ok):
    _check(1300, 1101, "front")
