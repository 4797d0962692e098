"""The resident CG (one cooperative launch a solve) against the CPU oracle, at
the sizes where its split can go wrong: one block, bricks of unequal extents,
a single layer of cells, every count of cells a thread, and the largest grid
that it takes beside the first one that it leaves to the kernel chain.

Bars: the true relative residual, recomputed by the oracle, meets the
tolerance, and the solution (zero mean, the systems are all-Neumann) agrees
with the oracle's CG to 1e-6 of its range where that is run.  At rtol 1e-9 both
errors are below cond * rtol; cond is at most 4 (n / pi)^2 < 3e2 at the
compared sizes."""
import numpy as np
import pytest

import xflow_gb300 as xf
from oracle import oracle as O
from xflow_gb300 import capi
from xflow_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = xf.Context(0)
    yield c
    c.close()


def case(shape, seed, holes):
    """A uniform box with Fictive holes and inactive Defined cells (their values enter their neighbours' rows)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    codes, _ = wl.neumann_box(*[n + 2 for n in shape])
    inner = codes[1:-1, 1:-1, 1:-1]
    if holes:
        inner[rng.random(shape) < 0.04] = 0
        inner[rng.random(shape) < 0.01] = 3
    wl._drop_isolated(codes)
    seps = [np.full(n + 1, 1.0 / n) for n in shape]
    act = codes == 1
    b = np.where(act, rng.standard_normal(codes.shape), 0.0)
    b[act] -= b[act].mean()
    x0 = np.zeros(codes.shape)
    if holes:   # a warm start with values on the inactive cells too
        x0 = rng.standard_normal(codes.shape) * 1e-3
    return codes, seps, b, x0


def check(ctx, shape, seed, precision, holes, compare):
    codes, seps, b, x0 = case(shape, seed, holes)
    g = xf.Grid(ctx, codes, *seps)
    A = xf.Operator(g)
    x = g.vec(x0)
    st = xf.solve(A, x, g.vec(b), method=xf.XF_CG, precision=precision, rtol=1e-9)
    got = x.download()
    assert st.status == capi.XF_OK and st.rel_resid <= 1e-9, (st.status, st.rel_resid)
    og = O.Grid(codes, None, *seps)
    O.set_threads(8)
    act = codes == 1
    r = O.apply(O.LAPLACE, og, got, b, -1)
    assert np.linalg.norm(r[act]) <= 1.01e-9 * np.linalg.norm(b[act])
    np.testing.assert_array_equal(got[~act], x0[~act])
    if compare:
        xo, _ = O.cg_plain(O.LAPLACE, og, np.zeros(codes.shape), b, 1e-11)
        d, ref = got - xo, xo - xo[act].mean()
        assert np.abs(d[act] - d[act].mean()).max() <= 1e-6 * np.abs(ref[act]).max()
    O.set_threads(1)


@pytest.mark.parametrize("precision", [xf.XF_PREC_FP64, xf.XF_PREC_MIXED])
@pytest.mark.parametrize("shape", [(2, 3, 2), (8, 8, 8), (1, 40, 37), (23, 1, 50), (31, 33, 1), (30, 41, 29),
                                   (75, 61, 83), (200, 20, 12)])
def test_sizes(ctx, precision, shape):
    check(ctx, shape, sum(shape), precision, holes=False, compare=max(shape) <= 50)


@pytest.mark.parametrize("precision", [xf.XF_PREC_FP64, xf.XF_PREC_MIXED])
@pytest.mark.parametrize("shape", [(17, 19, 23), (64, 48, 33)])
def test_holes_and_warm_start(ctx, precision, shape):
    check(ctx, shape, sum(shape), precision, holes=True, compare=False)


@pytest.mark.parametrize("precision", [xf.XF_PREC_FP64, xf.XF_PREC_MIXED])
@pytest.mark.parametrize("shape", [(256, 64, 64), (104, 108, 104), (110, 108, 110)])
def test_the_largest_grids(ctx, precision, shape):
    check(ctx, shape, 3, precision, holes=False, compare=False)


@pytest.mark.parametrize("precision", [xf.XF_PREC_FP64, xf.XF_PREC_MIXED])
def test_zero_right_hand_side_and_caps(ctx, precision):
    codes, seps, b, _ = case((12, 9, 10), 5, False)
    g = xf.Grid(ctx, codes, *seps)
    A = xf.Operator(g)
    x = g.vec(np.zeros(g.shape))
    st = xf.solve(A, x, g.vec(np.zeros(g.shape)), method=xf.XF_CG, precision=precision)
    assert st.status == capi.XF_OK and st.iterations == 0 and not x.download().any()
    for cap in (1, 7):
        st = xf.solve(A, g.vec(np.zeros(g.shape)), g.vec(b), method=xf.XF_CG, precision=precision, rtol=1e-13, maxit=cap)
        assert st.status == capi.XF_MAXIT and st.iterations == cap
    b2 = np.where(codes == 1, 1.0, 0.0)   # not in the range: no solver can meet the tolerance
    st = xf.solve(A, g.vec(np.zeros(g.shape)), g.vec(b2), method=xf.XF_CG, precision=precision, maxit=200)
    assert st.status != capi.XF_OK
