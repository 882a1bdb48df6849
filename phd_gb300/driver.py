"""Time loop of the reference's `solvers.iterator` (code/cpp/src/solvers/
iterator.cpp:85-170) for one material, on the GPU: CFL time step ->
boundaries -> ADER step (or the split scheme, SPLIT = True) -> distortion
renormalisation -> contortion reset (solvers/utils.cpp:44-85), with the
reference's 100-snapshot return convention and NaN early exit."""
import numpy as np
import torch

from . import api

N = api.N


class Stepper:
    """Device buffers for repeated steps of one grid (no per-step allocation)."""

    def __init__(self, nX, V, device="cuda"):
        from . import _lib
        self.lib = _lib.load()
        self.nX = np.asarray(nX, dtype=np.int32)
        self.nd = self.nX.size
        self.V = V
        ncb = int(np.prod(self.nX + 2))
        self.ub = torch.empty(int(np.prod(self.nX + 2 * N)) * V, dtype=torch.float64,
                              device=device)
        self.mask = torch.ones(ncb, dtype=torch.uint8, device=device)
        self.status = torch.zeros(ncb, dtype=torch.int32, device=device)
        self.dt = torch.empty(1, dtype=torch.float64, device=device)
        self.flag = torch.zeros(1, dtype=torch.int32, device=device)

    def step(self, u, dt, dX, bcs, MP, flux=0, stiff=False, split=False, half_step=True,
             contorted_tol=None):
        api.boundaries(u, self.ub, self.nX, bcs)
        if split:
            api.split_stepper(u, self.ub, self.nX, dt, dX, half_step, flux, MP, self.mask)
        else:
            api.ader_stepper(u, self.ub, self.nX, dt, dX, stiff, flux, MP, self.mask,
                             status=self.status)
        api.renorm_distortion(u, [MP])
        if contorted_tol is not None:
            api.reset_contorted(u, contorted_tol, [MP], flag=self.flag)
        return u


def iterate(u, tf, nX, dX, CFL, boundaryTypes, SPLIT=False, HALF_STEP=True, STIFF=False,
            FLUX=0, MPs=None, max_steps=None, contorted_tol=1.0):
    MP = MPs[0] if isinstance(MPs, (list, tuple)) else MPs
    nXa = np.asarray(nX, dtype=np.int32)
    V = u.numel() // int(np.prod(nXa))
    api.set_nvar(V)
    uf = u.view(-1)
    uprev, step = torch.empty_like(uf), None
    ret = [None] * 100
    t, count, push = 0.0, 0, 0
    while t < tf:
        if step is None:
            step = (_staged_step if STIFF and not SPLIT else _resident_step)(
                uf, tf, nXa, V, dX, CFL, boundaryTypes, SPLIT, HALF_STEP, FLUX, MP, contorted_tol)
        uprev.copy_(uf)
        t, nan = step(t, count)
        count += 1
        if t >= (push + 1) / 100.0 * tf:
            ret[push] = uf.clone()
            push += 1
        if nan:
            ret[push] = uprev
            if push + 1 < 100:
                ret[push + 1] = uf.clone()
            return ret
        if max_steps is not None and count >= max_steps:
            break
    ret[99] = uf.clone()
    return ret


def _resident_step(uf, tf, nXa, V, dX, CFL, boundaryTypes, SPLIT, HALF_STEP, FLUX, MP,
                   contorted_tol):
    """A step of the loop body in one call of the library (gpr_iterate,
    gpr_iterate_split) on a device clock, and one read of {t, dt, tf, cfl, count,
    NaN flag} back: the arguments are packed once per loop, and the host waits
    once per step."""
    from . import _lib
    lib = _lib.load()
    nXa, pn = api._i32(nXa)
    dXa, pd = api._f64(dX)
    bca, pb = api._i32(boundaryTypes)
    nd = nXa.size
    if bca.size != 2 * nd:
        raise ValueError("expected %d boundary codes" % (2 * nd))
    api.set_grid(nXa)
    api._nvar(uf, int(np.prod(nXa)))  # refuses a size that is no multiple of the cells
    c, pp = api._par(MP)
    n = lib.gpr_iterate_scratch_doubles(pn, nd, V)
    _lib.check(n, "iterate")
    scr = api._scratch(n, uf)
    ctl = torch.tensor([0.0, 0.0, float(tf), float(CFL), 0.0, 0.0], dtype=torch.float64,
                       device=uf.device)
    pu, ps, pclk = api._dev(uf, "u"), api._dev(scr, "s"), api._dev(ctl, "clock")
    pflag = api.ctypes.c_void_p(ctl.data_ptr() + 5 * 8)
    tol = float("inf") if contorted_tol is None else float(contorted_tol)
    size = uf.numel()

    def step(t, count):
        st = api._stream()
        if SPLIT:
            rc = lib.gpr_iterate_split(pu, pn, nd, pd, pb, int(FLUX), int(bool(HALF_STEP)), pp,
                                       None, pclk, 1, ps, tol, V, st)
        else:
            rc = lib.gpr_iterate(pu, pn, nd, pd, pb, int(FLUX), pp, None, pclk, 1, ps, None, tol,
                                 V, st)
        _lib.check(rc, "iterate")
        _lib.check(lib.gpr_any_nan(pu, size, pflag, st), "any_nan")
        c = ctl.tolist()
        return c[0], c[5] != 0.0

    step.keep = (nXa, dXa, bca, c, scr, ctl)  # what the pointers point to
    return step


def _staged_step(uf, tf, nXa, V, dX, CFL, boundaryTypes, SPLIT, HALF_STEP, FLUX, MP,
                 contorted_tol):
    """The same step by its stages, for STIFF (every cell through the Newton
    pass), which the resident loop does not take."""
    st = Stepper(nXa, V, device=uf.device)

    def step(t, count):
        dt = float(api.timestep_device(uf, dX, CFL, t, tf, count, MP, out=st.dt).item())
        st.step(uf, dt, dX, boundaryTypes, MP, flux=FLUX, stiff=True, contorted_tol=contorted_tol)
        return t + dt, bool(torch.isnan(uf).any())

    return step
