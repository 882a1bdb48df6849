"""Scratch of the 2D calls: the face buffer holds the face sums of both directions
and nothing per quadrature point, whatever the flux."""
import ctypes

import numpy as np
import pytest

from phd_gb300 import _lib


@pytest.mark.parametrize("V", [14, 15, 17])
@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 5), (512, 512), (4096, 4096)])
def test_2d_face_scratch(nx, ny, V):
    lib = _lib.load()
    nX = np.array([nx, ny], np.int32)
    p = nX.ctypes.data_as(ctypes.c_void_p)
    faces, cells = (nx + 1) * (ny + 1), (nx + 2) * (ny + 2)
    fv = lib.gpr_fv_scratch_doubles(p, 2, V)
    assert fv == 2 * faces * 2 * V
    # the loops keep the predictor's deferred cells (2 doubles a cell) there too
    assert fv >= 2 * cells + 8
    total = lib.gpr_iterate_scratch_doubles(p, 2, V)
    states = (nx + 4) * (ny + 4) + 4 * cells + 8 * cells
    assert total <= states * V + max(fv, lib.gpr_weno_scratch_doubles(p, 2, V)) + 64
