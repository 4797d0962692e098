"""The resident mixed CG where its FP32 recursion runs to its own rounding before the true residual meets the tolerance:
smooth right-hand sides near the floor of FP64, and right-hand sides of a few eigenvectors.

Bars: smooth ones at 1e-12, above the FP64 floor of these boxes (5e-13, the rounding of A x), in at most twice the
iterations of FP64 CG.  Of a few eigenvectors nothing is left after as many iterations but the rounding of FP32, which
is noise: at most the iterations of a right-hand side of noise more."""
import numpy as np
import pytest

import xflow_gb300 as xf
from xflow_gb300 import capi
from xflow_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def box(ctx, shape, holes=False):
    rng = np.random.default_rng(1)
    codes, _ = wl.neumann_box(*[n + 2 for n in shape])
    if holes:
        codes[1:-1, 1:-1, 1:-1][rng.random(shape) < 0.03] = 0
        wl._drop_isolated(codes)
    g = xf.Grid(ctx, codes, *[np.full(n + 1, 1.0 / n) for n in shape])
    return g, xf.Operator(g), codes == 1, rng


def run(A, g, b, rtol, maxit=100000, precision=xf.XF_PREC_MIXED, every=50):
    st = xf.solve(A, g.vec(np.zeros(g.shape)), g.vec(b), method=xf.XF_CG, precision=precision, rtol=rtol, maxit=maxit,
                  replace_every=every)
    assert st.reserved[0] == 2   # the resident kernel
    assert st.status == capi.XF_OK and st.rel_resid <= rtol, (st.status, st.iterations, st.rel_resid)
    return st.iterations


@pytest.mark.parametrize("every", [50, 200])
@pytest.mark.parametrize("shape,holes", [((100, 100, 100), False), ((128, 64, 64), False), ((128, 64, 64), True),
                                         ((96, 96, 96), True), ((40, 36, 44), True)])
def test_smooth(shape, holes, every):
    ctx = xf.Context(0)
    g, A, act, _ = box(ctx, shape, holes)
    t = [np.linspace(0, 1, n) for n in g.shape]
    b = np.where(act, np.sin(3 * t[0])[:, None, None] * np.cos(5 * t[1])[None, :, None] * np.exp(t[2])[None, None], 0)
    b[act] -= b[act].mean()
    plain = run(A, g, b, 1e-12, precision=xf.XF_PREC_FP64)
    run(A, g, b, 1e-12, maxit=2 * plain, every=every)
    ctx.close()


@pytest.mark.parametrize("rtol", [1e-6, 1e-9])
@pytest.mark.parametrize("modes", [1, 2, 3, 5, 7])
@pytest.mark.parametrize("shape", [(24, 20, 28), (40, 41, 39), (64, 64, 64)])
def test_few_modes(shape, modes, rtol):
    ctx = xf.Context(0)
    g, A, act, rng = box(ctx, shape)
    cs = [np.pad(np.cos(np.pi * np.outer(np.arange(n), np.arange(n) + 0.5) / n), ((0, 0), (1, 1))) for n in shape]
    b = np.zeros(g.shape)
    for m in range(modes):   # eigenvectors of the all-Neumann box
        b += (1 + 0.3 * m) * np.einsum("i,j,k->ijk", cs[0][2 + 2 * m], cs[1][1 + 2 * m], cs[2][3 + m])
    noise = np.where(act, rng.standard_normal(g.shape), 0.0)
    noise[act] -= noise[act].mean()
    run(A, g, b, rtol, maxit=modes + run(A, g, noise, rtol))
    ctx.close()
