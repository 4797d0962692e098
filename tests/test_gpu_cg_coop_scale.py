"""The resident CG on right-hand sides of any magnitude.  A system times a power of two is the same arithmetic unless
something under- or overflows, so the iterates of 2^k b are 2^k times those of b, bit for bit, as long as (b, b) and A x
stay in FP64's range; mixed solves at every k, although the squares of FP32 leave its range at |k| above 60."""
import numpy as np
import pytest

import xflow_gb300 as xf
from xflow_gb300 import capi
from xflow_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warm", [False, True])
@pytest.mark.parametrize("precision", [xf.XF_PREC_FP64, xf.XF_PREC_MIXED])
@pytest.mark.parametrize("shape", [(40, 36, 44), (13, 11, 12), (75, 40, 33)])
def test_any_magnitude(shape, precision, warm):
    ctx = xf.Context(0)
    rng = np.random.default_rng(sum(shape))
    codes, _ = wl.neumann_box(*[n + 2 for n in shape])
    codes[1:-1, 1:-1, 1:-1][rng.random(shape) < 0.03] = 0
    wl._drop_isolated(codes)
    g = xf.Grid(ctx, codes, *[np.full(n + 1, 1.0 / n) for n in shape])
    A = xf.Operator(g)
    act = codes == 1
    y = g.vec(None)
    A.apply(g.vec(np.where(act, rng.standard_normal(g.shape), 0.0)), y, flags=xf.XF_ZERO_INACTIVE)
    b = y.download()
    x0 = np.where(act, rng.standard_normal(g.shape), 0.0) * warm
    want = None
    for k in (0, -40, -48, -60, -75, -140, -480, 40, 60, 120, 470, 478):
        x = g.vec(np.ldexp(x0, k))
        st = xf.solve(A, x, g.vec(np.ldexp(b, k)), method=xf.XF_CG, precision=precision, rtol=1e-10)
        assert st.reserved[0] == 2 and st.status == capi.XF_OK and st.rel_resid <= 1e-10, (k, st.status, st.rel_resid)
        got = np.ldexp(x.download(), -k)
        if want is None:
            want, its = got, st.iterations
        assert st.iterations == its, k
        np.testing.assert_array_equal(got, want, err_msg=str(k))
    ctx.close()


@pytest.mark.parametrize("precision", [xf.XF_PREC_FP64, xf.XF_PREC_MIXED])
def test_start_far_from_the_right_hand_side(precision):
    """b of 2^-120 against a start of 1, on a system with Defined neighbours (no null space): (r, r) falls from one scale
    to the other within the solve, the mixed one's by replaced residuals.  No NaN, and the residual the solve reports is
    that of the iterate it leaves."""
    ctx = xf.Context(0)
    shape = (20, 18, 22)
    rng = np.random.default_rng(3)
    codes, _ = wl.neumann_box(*[n + 2 for n in shape])
    codes[1:-1, 1:-1, 1:-1][rng.random(shape) < 0.05] = 3
    g = xf.Grid(ctx, codes, *[np.full(n + 1, 1.0 / n) for n in shape])
    A = xf.Operator(g)
    act = codes == 1
    b = np.where(act, rng.standard_normal(g.shape), 0.0) * 2.0 ** -120
    x = g.vec(np.where(act, rng.standard_normal(g.shape), 0.0))
    st = xf.solve(A, x, g.vec(b), method=xf.XF_CG, precision=precision, rtol=1e-8, maxit=3000)
    got = x.download()
    r = g.vec(None)
    A.apply(x, r, s=g.vec(b), sign=-1, flags=xf.XF_ZERO_INACTIVE)
    rel = np.linalg.norm(r.download()) / np.linalg.norm(b)
    assert np.isfinite(got).all() and st.status in (capi.XF_OK, capi.XF_STALL, capi.XF_MAXIT)
    assert abs(st.rel_resid - rel) <= 1e-6 * rel and rel <= 1e24   # the start's is 2^120 times the coefficients, 1e40
    assert precision == xf.XF_PREC_FP64 or st.status == capi.XF_OK
    ctx.close()
