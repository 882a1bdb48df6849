"""MultiIterator.step's NaN report belongs to the step: an iterator that has met a
NaN reports none for a clean state stepped afterwards."""
import numpy as np
import pytest
import torch

from phd_gb300 import problems

pytestmark = pytest.mark.gpu


def test_nan_report_of_a_later_clean_step(cuda_ok):
    from phd_gb300.ghost import MultiIterator
    u0, MPs, _, dX, _ = problems.shock_bubble(nx=40, ny=20, mu=1e-2, shear=0.3)
    nX = np.array(u0.shape[:2], np.int32)
    clean = torch.tensor(u0.ravel(), device="cuda")
    it = MultiIterator(nX, dX, 0, MPs, 0.8, 1e9, device="cuda")
    start = it.clock.clone()
    u = clean.clone()
    assert it.step(u)[2] is False
    bad = clean.clone()
    bad.view(-1, 15)[7, 3] = float("nan")
    assert it.step(bad)[2] is True
    for _ in range(2):
        it.clock.copy_(start)
        v = clean.clone()
        t, dt, nan = it.step(v)
        assert nan is False and t == dt > 0
        assert torch.equal(v, u)
