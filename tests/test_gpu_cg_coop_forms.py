"""Every form of the resident CG's kernel (2 to 16 cells a column, those that the other tests' sizes do not reach), a
last brick that is shorter on each axis, and the route: the resident solve is two launches, the kernel chain hundreds.
The split takes 16 cells a column, 512 columns a brick and a brick an SM at most: on 152 SMs 102^3 and 128 x 152 x 64 go
to the resident kernel, 104 x 108 x 104 and 110 x 108 x 110 do not.

Bar: the true relative residual, recomputed by the oracle, meets the tolerance."""
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


def check(ctx, shape, precision, resident, holes=False):
    rng = np.random.default_rng(sum(shape))
    codes, _ = wl.neumann_box(*[n + 2 for n in shape])
    if holes:
        codes[1:-1, 1:-1, 1:-1][rng.random(shape) < 0.03] = 0
        wl._drop_isolated(codes)
    seps = [np.full(n + 1, 1.0 / n) for n in shape]
    g = xf.Grid(ctx, codes, *seps)
    A = xf.Operator(g)
    act = codes == 1
    y = g.vec(None)
    A.apply(g.vec(np.where(act, rng.standard_normal(g.shape), 0.0)), y, flags=xf.XF_ZERO_INACTIVE)
    b = y.download()   # in the range, whatever the holes cut off
    x = g.vec(np.zeros(g.shape))
    st = xf.solve(A, x, g.vec(b), method=xf.XF_CG, precision=precision, rtol=1e-9)
    assert st.status == capi.XF_OK and st.rel_resid <= 1e-9, (st.status, st.rel_resid)
    assert (st.reserved[0] == 2) == resident, st.reserved[0]
    og = O.Grid(codes, None, *seps)
    O.set_threads(8)
    r = O.apply(O.LAPLACE, og, x.download(), b, -1)
    O.set_threads(1)
    assert np.linalg.norm(r[act]) <= 1.01e-9 * np.linalg.norm(b[act])


PRECISIONS = [xf.XF_PREC_FP64, xf.XF_PREC_MIXED]


# cells a column: 6, 6, 10, 12, 16 (of 15), 16, 16 (of 15)
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("shape", [(72, 72, 72), (53, 64, 64), (88, 88, 88), (96, 96, 96), (90, 90, 90), (128, 128, 64),
                                   (102, 102, 102)])
def test_forms(ctx, precision, shape):
    check(ctx, shape, precision, resident=True, holes=shape in ((53, 64, 64), (90, 90, 90)))


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("shape,resident", [((128, 152, 64), True), ((104, 108, 104), False), ((110, 108, 110), False)])
def test_the_limit(ctx, precision, shape, resident):
    if ctx_sms() != 152:
        pytest.skip("the limit of 152 SMs")
    check(ctx, shape, precision, resident)


def ctx_sms():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count
