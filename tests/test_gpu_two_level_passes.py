"""The two-level preconditioner's transfers (open-face counts, omega, r - omega A P zc, y in the smoother's last pass)
against the general path, which prolongates, multiplies and combines FP64 boxes in separate launches: the first
iterate x_1 = alpha M b of the mixed solve is that of the FP64 solve.

Tolerance: the two networks see the same input up to FP32 rounding, so at most a few of its BF16 values and of each
layer's differ by one unit (2^-8 relative); everything else is FP32.  5 units in the l2 norm, 2e-2; a wrong face, block
or omega changes x_1 by tens of percent."""
import numpy as np
import pytest

import xflow_gb300 as xf
from xflow_gb300 import capi
from xflow_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


# the smallest boxes a network takes, planes of one and several tiles, chunks that end inside a block; F = 2 stores A y
@pytest.mark.parametrize("F,n,degree", [(4, (32, 32, 32), 2), (4, (32, 48, 64), 4), (4, (80, 32, 144), 8),
                                        (4, (48, 80, 64), 4), (2, (16, 24, 32), 4)])
def test_first_iterate_is_the_general_paths(F, n, degree):
    rng = np.random.default_rng(sum(n) + F)
    codes = np.zeros([v + 2 for v in n], np.int32)
    inner = codes[1:-1, 1:-1, 1:-1]
    inner[:] = (rng.random(n) > 0.1) * wl.ACTUAL                 # holes: closed faces of every kind
    inner[:F, :2 * F, 3:2 * F + 1] = 0                            # whole blocks and parts of blocks
    inner[-1] = wl.ACTUAL
    seps = [np.full(v + 1, 1.0 / n[2]) for v in n]
    b = np.where(codes == wl.ACTUAL, rng.standard_normal(codes.shape), 0.0)
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
    assert np.linalg.norm(xs[1] - xs[0]) <= 2e-2 * np.linalg.norm(xs[0])
    ctx.close()
