"""The two-level preconditioner's transfers cell by cell: with right-hand sides of small whole numbers the block sums are
exact, so the network of the mixed path sees the bits that the general FP64 path's network sees, and the first iterates
x_1 = alpha M b differ by FP32 rounding only.

Bar, in the maximum norm over the cells: 2e-5 of the largest value, 170 FP32 roundings (the open-face differences, the
smoother's two to four passes of two rows each and the combination); one cell's wrong face moves that cell by percent."""
import numpy as np
import pytest

import xflow_gb300 as xf
from xflow_gb300 import capi
from xflow_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F,n,degree", [(4, (32, 32, 32), 2), (4, (32, 48, 64), 4), (4, (80, 32, 144), 8),
                                        (4, (48, 80, 64), 4), (4, (64, 128, 32), 4), (2, (16, 24, 32), 4)])
def test_first_iterate_cell_by_cell(F, n, degree):
    rng = np.random.default_rng(sum(n) + F)
    codes = np.zeros([v + 2 for v in n], np.int32)
    inner = codes[1:-1, 1:-1, 1:-1]
    inner[:] = (rng.random(n) > 0.1) * wl.ACTUAL                 # holes: closed faces of every kind
    inner[:F, :2 * F, 3:2 * F + 1] = 0                            # whole blocks and parts of blocks
    inner[-1] = wl.ACTUAL
    seps = [np.full(v + 1, 1.0 / n[2]) for v in n]
    b = np.where(codes == wl.ACTUAL, rng.integers(-2, 3, codes.shape), 0).astype(float)
    ctx = xf.Context(0)
    g = xf.Grid(ctx, codes, *seps)
    gc = xf.Grid(ctx, *wl.coarse_grid(codes, seps[0], F)[:1], *[np.full(v // F + 1, F / n[2]) for v in n])
    net = xf.UNet(gc, seed=3)
    A = xf.Operator(g)
    xs = []
    for prec in (xf.XF_PREC_FP64, xf.XF_PREC_MIXED):
        x, bv = g.vec(np.zeros(g.shape)), g.vec(b)
        st = xf.solve_fcg(A, x, bv, unet=net, precond=capi.XF_PRECOND_UNET2, precision=prec, maxit=1, window=1,
                          degree=degree, ratio=30, rtol=1e-12)
        assert st.iterations == 1
        xs.append(x.download())
    assert np.abs(xs[1] - xs[0]).max() <= 2e-5 * np.abs(xs[0]).max()
    ctx.close()
