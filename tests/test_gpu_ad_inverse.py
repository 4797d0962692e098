"""The Jacobi preconditioner's inverse row diagonals are 1 / d correctly rounded.  A box with one Actual cell makes the
solve scalar: every sum of an iteration is one product, so BiCGStab's first iterate follows bit for bit from the row's
diagonal (read by a unit vector) and the right-hand side, in rational arithmetic rounded where the device rounds.
Diagonals from 1e-295 to 1e295 (the outermost by the division, the others by Newton steps); no tolerance."""
from fractions import Fraction as Q

import numpy as np
import pytest

import xflow_gb300 as xf
from xflow_gb300 import capi

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    return float(Q(a) * Q(b) + Q(c))


def first_iterate(d, b):
    """One iteration from 0 on d x = b."""
    inv = 1.0 / d
    ph = inv * b
    v = d * ph
    an = (b * b) / (b * v)
    s = fma(-an, v, b)
    sh = inv * s
    t = d * sh
    tt = t * t
    if tt == 0.0:   # an exact first half: the device's omega is 0 / 0
        return None
    wn = (t * s) / tt
    return fma(an, ph, fma(wn, sh, 0.0))


@pytest.mark.parametrize("k", [0, -900, 900, -980, 980])
def test_inverse_diagonals(k):
    ctx = xf.Context(0)
    rng = np.random.default_rng(5)
    codes = np.full((3, 3, 3), 3, np.int32)   # Defined around one Actual cell
    codes[1, 1, 1] = 1
    g = xf.Grid(ctx, codes, *[np.ones(2)] * 3)
    A = xf.Operator(g, xf.XF_OP_ADVDIFF)
    zero, unit, y, x = g.vec(None), np.zeros(g.shape), g.vec(None), g.vec(None)
    unit[1, 1, 1] = 1.0
    scale = np.ldexp(1.0, k)
    seen = 0
    for _ in range(300):
        A.set_advection(zero, zero, zero, float(rng.uniform(0.5, 2.0)) / scale, 0.0, 3)   # 1 / tau is the diagonal
        A.apply(g.vec(unit), y, flags=xf.XF_ZERO_INACTIVE)
        d = float(y.download()[1, 1, 1])
        b = float(rng.uniform(0.5, 2.0))
        want = first_iterate(d, b)
        if want is None:
            continue
        x.fill(0.0)
        xf.solve(A, x, g.vec(unit * b), method=xf.XF_BICGSTAB, precond=capi.XF_PRECOND_JACOBI, atol=1e-300, maxit=1)
        assert float(x.download()[1, 1, 1]) == want, (d.hex(), b.hex())
        seen += 1
    assert seen >= 30
    ctx.close()
