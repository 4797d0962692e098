"""Jacobi BiCGStab on the scaled transport rows (boxes from half a million cells on): the manufactured solution from
a start that is not zero, on even rows (pairs of cells) and odd ones, with semi-sum, normal-difference and oblique
border rows; and the rows themselves again after the solve.

Tolerances: the solver's stop rule on the true residual, recomputed by the oracle (1e-9 of the largest |b|, and the
rounding of x += D^-1 y, another 1e-13 of the largest |A||x| that stands in a row); the solution's error is the
residual's times the inverse's norm, below tau (1e-3) times the largest diagonal over the smallest, 1e-5 as in the
small boxes."""
import numpy as np
import pytest

import xflow_gb300 as xf
from oracle import oracle as O
from xflow_gb300 import capi
from test_gpu_advdiff import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(82, 80, 82), (80, 84, 81)])
@pytest.mark.parametrize("flags", [3, 7])
def test_scaled_bicgstab(shape, flags):
    ctx = xf.Context(0)
    g, A, og, vel, rng = case(ctx, shape=shape, seed=sum(shape), tau=1e-3, D=0.02, flags=flags)
    sm = og.smask.astype(bool)
    xt = np.where(sm, rng.standard_normal(g.shape), 0.0)
    b = O.apply_advdiff(og, xt, *vel, 1e-3, 0.02, flags)
    top = np.abs(b).max()
    x0 = np.where(sm, rng.standard_normal(g.shape), 0.0)
    its = []
    for rep in range(2):   # the second solve finds the table made
        x = g.vec(x0)
        st = xf.solve(A, x, g.vec(b), method=xf.XF_BICGSTAB, precond=capi.XF_PRECOND_JACOBI, atol=1e-9 * top)
        assert st.status == capi.XF_OK
        got = x.download()
        r = O.apply_advdiff(og, got, *vel, 1e-3, 0.02, flags) - b
        assert np.abs(r[sm]).max() <= 1.001e-9 * top
        assert np.abs(got[sm] - xt[sm]).max() <= 1e-5 * np.abs(xt[sm]).max()
        its.append(st.iterations)
    assert its[0] == its[1]
    y = g.vec(None)
    A.apply(g.vec(xt), y, flags=xf.XF_ZERO_INACTIVE)
    assert np.abs(y.download()[sm] - b[sm]).max() <= 1e-13 * top
    ctx.close()
