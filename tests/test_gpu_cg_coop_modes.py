"""Right-hand sides of a few eigenvectors: FP64 CG ends after as many iterations, the last of which takes (r, r) down by
all that the arithmetic carries.  The resident CG forms the next (r, r) from (r, r), (r, q) and (q, q), a difference
that says nothing below their rounding, so it has to measure it there, as the kernel chain always does.

Bar: no more iterations than the chain."""
import numpy as np
import pytest

import xflow_gb300 as xf
from xflow_gb300 import capi
from xflow_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rtol", [1e-6, 1e-9, 1e-12])
@pytest.mark.parametrize("modes", [1, 2, 3, 5])
@pytest.mark.parametrize("shape", [(24, 20, 28), (40, 41, 39)])
def test_few_modes(monkeypatch, shape, modes, rtol):
    ctx = xf.Context(0)
    codes, _ = wl.neumann_box(*[n + 2 for n in shape])
    g = xf.Grid(ctx, codes, *[np.full(n + 1, 1.0 / n) for n in shape])
    A = xf.Operator(g)
    cs = [np.pad(np.cos(np.pi * np.outer(np.arange(n), np.arange(n) + 0.5) / n), ((0, 0), (1, 1))) for n in shape]
    b = np.zeros(codes.shape)
    for m in range(modes):   # eigenvectors of the all-Neumann box
        b += (1 + 0.3 * m) * np.einsum("i,j,k->ijk", cs[0][2 + 3 * m], cs[1][1 + 2 * m], cs[2][3 + m])
    its = []
    for chain in (True, False):
        if chain:
            monkeypatch.setenv("XF_PQT", "0")   # names a kernel of the chain
        else:
            monkeypatch.delenv("XF_PQT")
        x = g.vec(np.zeros(codes.shape))
        st = xf.solve(A, x, g.vec(b), method=xf.XF_CG, rtol=rtol)
        assert st.status == capi.XF_OK and st.rel_resid <= rtol
        assert (st.reserved[0] == 2) == (not chain)
        its.append(st.iterations)
    ctx.close()
    assert its[1] <= its[0], its
