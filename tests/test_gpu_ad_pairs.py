"""The advection-diffusion table rows by pairs of cells (even rows) and cell by cell (odd rows): rows, the untouched
inactive cells of a plain apply and the dot, against the oracle's rows.

Tolerance: the seven products of a fast row in another order than the oracle's, 7 units of 2^-53 of the largest term,
below 1e-13 of the largest |y| (the bound of the fast rows elsewhere); the dot the same, summed over the cells."""
import numpy as np
import pytest

import xflow_gb300 as xf
from oracle import oracle as O
from xflow_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


# the shortest rows, rows whose pairs hold a border cell and an inner one, a box of one and of several blocks, odd rows
@pytest.mark.parametrize("shape", [(5, 6, 4), (6, 5, 6), (12, 11, 14), (40, 21, 34), (9, 8, 17)])
@pytest.mark.parametrize("flags", [3, 7])
def test_pair_rows(shape, flags):
    rng = np.random.default_rng(sum(shape) + flags)
    codes, nrm = wl.poisson_cube(*shape)
    seps = [np.diff(wl.random_nodes(n, rng)) for n in shape]
    vel = [rng.uniform(-2, 2, shape) for _ in range(3)]
    ctx = xf.Context(0)
    g = xf.Grid(ctx, codes, *seps, nrm)
    A = xf.Operator(g, xf.XF_OP_ADVDIFF)
    A.set_advection(*(g.vec(v) for v in vel), 1e-2, 0.05, flags)
    og = O.Grid(codes, nrm, *seps)
    sm = og.smask.astype(bool)
    x = rng.standard_normal(shape)
    want = O.apply_advdiff(og, x, *vel, 1e-2, 0.05, flags)
    top = np.abs(want[sm]).max()
    y = g.vec(np.full(shape, 7.0))
    dot = A.apply(g.vec(x), y, want_dot=True)
    got = y.download()
    assert np.abs(got[sm] - want[sm]).max() <= 1e-13 * top
    assert np.all(got[~sm] == 7.0)
    assert abs(dot - (x[sm] * want[sm]).sum()) <= 1e-13 * np.abs(x[sm] * want[sm]).sum() * 4
    A.apply(g.vec(x), y, flags=xf.XF_ZERO_INACTIVE)
    assert np.all(y.download()[~sm] == 0.0)
    ctx.close()
