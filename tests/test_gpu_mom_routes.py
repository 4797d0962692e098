"""The routes of the momentum right-hand side's viscous pass: one viscosity (told by the cells' codes), one viscosity
but for a cell, a rest term of -0, velocities that are huge or not finite, no viscosity.  Every value bit for bit the
oracle's (NaN as NaN): the routes differ in what they read, not in what they compute."""
import numpy as np
import pytest

import xflow_gb300 as xf
from oracle import oracle as O
from xflow_gb300 import workloads as wl_step
from test_gpu_step import grids, momentum_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["one", "cell", "minus_zero", "huge", "inf", "nan", "none"])
@pytest.mark.parametrize("axis", [1, 2, 3])
def test_viscous_routes(what, axis):
    ctx = xf.Context(0)
    cs = wl_step.staggered_channel()
    gp, gu, gv, gw = grids(ctx, cs)
    vis, comps, extra = momentum_case(cs)
    _, codes, hs = comps[axis - 1]
    g = (gu, gv, gw)[axis - 1]
    border, force = extra[axis][0], np.zeros(g.shape)
    vis = np.full_like(vis, 0.0371)
    u, v, w = (np.array(cs[k]) for k in "uvw")
    mid = tuple(n // 2 for n in vis.shape)
    if what == "cell":
        vis[mid] *= 1.5
    elif what == "minus_zero":
        force[:] = -0.0
    elif what in ("huge", "inf", "nan"):
        v[mid] = {"huge": 1e200, "inf": np.inf, "nan": np.nan}[what]
    vis = None if what == "none" else vis
    out = xf.momentum_rhs(axis, g, gu.vec(u), gv.vec(v), gw.vec(w), vis=gp.vec(vis) if vis is not None else None,
                          border=g.vec(border), force=g.vec(force))
    with np.errstate(all="ignore"):
        want, st, _ = O.momentum_rhs(axis, codes, u, v, w, *hs, vis=vis, border=border, force=force)
    assert st == 0
    for name, o, w_ in zip(("uTr", "vTr", "wTr", "visTr", "rp"), out, want):
        got = o.download()
        np.testing.assert_array_equal(got, w_, err_msg=name)
        ok = ~np.isnan(w_)
        np.testing.assert_array_equal(np.signbit(got[ok]), np.signbit(w_[ok]), err_msg=name)
    ctx.close()
