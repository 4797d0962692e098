"""Lines along the memory in staged tiles of 16 steps: lengths on both sides of a tile's edge, from one to nine tiles,
lines that do not fill a block of 64, lines of one index, strides wider than a line, and divisors whose reciprocal is
not a normal number (they take the IEEE division).  Bit for bit the oracle's recurrences, elements outside the lines
untouched; no tolerance."""
import numpy as np
import pytest

import xflow_gb300 as xf
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def lines(ctx, M, nl1, nl2, ls1, ls2, size, extreme=False):
    rng = np.random.default_rng(M + nl1 + nl2)
    a, c = rng.uniform(-1, 0, size), rng.uniform(-1, 0, size)
    b, f, u = 2.5 + rng.uniform(0, 1, size), rng.standard_normal(size), rng.standard_normal(size)
    if extreme:   # rows from the denormals to the top of the range, and zeros
        s = np.ldexp(1.0, rng.integers(-1070, 1015, size))
        a, b, c, f = (np.where(rng.random(size) < 0.02, 0.0, t * s) for t in (a, b, c, f))
    dev = [torch.from_numpy(t.copy()).cuda() for t in (u, a, b, c, f)]
    torch.cuda.synchronize()
    xf.thomas_lines(ctx, M, *(t.data_ptr() for t in dev), nl1, nl2, ls1, ls2, 1)
    ctx.synchronize()
    want = u.copy()
    with np.errstate(all="ignore"):
        for l1 in range(nl1):
            for l2 in range(nl2):
                at = slice(l1 * ls1 + l2 * ls2, l1 * ls1 + l2 * ls2 + M + 1)
                want[at] = O.thomas(M, want[at], a[at], b[at], c[at], f[at])
    np.testing.assert_array_equal(dev[0].cpu().numpy(), want)


@pytest.fixture(scope="module")
def ctx():
    c = xf.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("M", [1, 2, 15, 16, 17, 18, 32, 33, 34, 49, 129, 130])
@pytest.mark.parametrize("nl1,nl2", [(1, 1), (3, 21), (8, 8), (5, 13), (129, 1), (1, 70)])
def test_lengths_and_blocks(ctx, M, nl1, nl2):
    lines(ctx, M, nl1, nl2, nl2 * (M + 1), M + 1, nl1 * nl2 * (M + 1))


def test_strides_wider_than_a_line(ctx):
    lines(ctx, 40, 7, 11, 11 * 47 + 5, 47, 7 * (11 * 47 + 5))


@pytest.mark.parametrize("M", [2, 17, 50])
def test_divisors_at_the_ends_of_the_range(ctx, M):
    lines(ctx, M, 40, 20, 20 * (M + 1), M + 1, 800 * (M + 1), extreme=True)


@pytest.mark.parametrize("shape", [(20, 5, 37), (34, 18, 16)])
@pytest.mark.parametrize("axis", [1, 2, 3])
def test_right_hand_side_in_place(ctx, axis, shape):
    """f and u the same array: every f[m] is read before u[m] is written."""
    rng = np.random.default_rng(axis)
    a, c = rng.uniform(-1, 0, shape), rng.uniform(-1, 0, shape)
    b, u = 2.5 + rng.uniform(0, 1, shape), rng.standard_normal(shape)
    dev = [torch.from_numpy(t.copy()).cuda() for t in (u, a, b, c)]
    torch.cuda.synchronize()
    M, *where = xf.box_lines(shape, axis)
    pu, pa, pb, pc = (t.data_ptr() for t in dev)
    xf.thomas_lines(ctx, M, pu, pa, pb, pc, pu, *where)
    ctx.synchronize()
    want = u.copy()
    W, A, B, C, F = (np.moveaxis(t, axis - 1, -1) for t in (want, a, b, c, u))
    for at in np.ndindex(W.shape[:-1]):
        W[at] = O.thomas(M, W[at], A[at], B[at], C[at], F[at])
    np.testing.assert_array_equal(dev[0].cpu().numpy(), want)
