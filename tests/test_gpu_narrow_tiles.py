"""The 128 x 128 tiles of the two-plane bf16 product (kernel code 2064), which
orders up to one wave of them run on: the accumulation order over K and the plane
products is that of the 256-wide kernels, so the results are the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 256, 257, 520, 1536, 1537, 2048])
def test_narrow_tiles_are_bit_exact(ctx, n):
    rng = np.random.default_rng(n)
    A = rng.uniform(-1, 1, (n, n))
    X = 0.5 * (A + A.T)
    C = ctx.symsq_split(X, 2, 2064)
    assert np.array_equal(C, ctx.symsq_split(X, 2, 64))
    assert np.array_equal(C, ctx.symsq_split(X, 2, 1064))
