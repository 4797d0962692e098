"""The convolution's operand copies by the length of a box's rows: slabs that overlap and come as one copy (rows shorter
than a tile's 128 cells) and slabs of their own (128 and longer), at the edges, with resident and streamed weights and
every number of CTAs an SM.

Tolerance: BF16 products are exact in FP32 and 27 ci of them are summed, 27 * 96 * 2^-24 relative at worst, below 2e-4 of
the sum of magnitudes and, with signs at random, below 1e-5 of the largest output (the bound of the other layers' test)."""
import numpy as np
import pytest

from test_gpu_conv import case, conv_ref, ctx, run_conv   # noqa: F401 (ctx is a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3", [3, 126, 127, 128, 129, 140])
@pytest.mark.parametrize("ci,co", [(16, 16), (48, 16), (64, 64), (96, 32)])
def test_row_lengths(ctx, n3, ci, co):   # noqa: F811
    x, W, bias, mask = case((4, 5, n3), ci, co, ci + co + n3)
    got = run_conv(ctx, x, W, bias, mask, 1, True)
    want = conv_ref(x, W, bias, mask, 1)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
