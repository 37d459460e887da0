"""The slicing kernels and the choice of product kernel by size, at the sizes
where they change: the row slicer in shared memory up to padded order 1536 and
the tiled one above, 128 x 64 tiles up to padded order 1024 and CTA pairs above.

A product with the identity hands the digits back: with f = 1 for the rows of I
(one digit, 64 / 128) every digit pair of weight above 2^(-7S) is kept, and the
sums of one row's digits are exact in FP64, so the result is exactly
trunc(A 2^(7S - e)) 2^(e - 7S) with |row max| < 2^e.
"""
import numpy as np
import pytest

from oracle import ptb_oracle as O
from ptb_b200 import synth

pytestmark = pytest.mark.gpu


def cut(M, S):
    """Rows of M as S truncated base-128 digits; a NaN has no digits."""
    F = np.where(np.isnan(M), 0.0, M)
    _, e = np.frexp(np.max(np.abs(F), axis=1, keepdims=True))
    return np.ldexp(np.trunc(np.ldexp(F, 7 * S - e)), e - 7 * S)


@pytest.mark.parametrize("S", [4, 6, 7, 8])
@pytest.mark.parametrize("n", [1, 31, 129, 300, 1536, 1537])
def test_slices_hold_the_truncated_rows(ctx, n, S):
    rng = np.random.default_rng(100 * n + S)
    A = rng.standard_normal((n, n)) * np.exp2(rng.integers(-30, 30, (n, 1)))
    A *= np.exp2(-rng.integers(0, 3 * S, (n, n)).astype(float))   # short and long digit strings
    A[rng.random((n, n)) < 0.1] = 0.0
    if n > 30:
        A[7] = 0.0
        A[3, 5] = np.nan
    eye = np.eye(n)
    for tri, mask in ((0, np.ones((n, n))), (1, np.tri(n)), (2, np.tri(n).T)):
        want = cut(np.where(mask > 0, A, 0.0), S)
        # A as the row operand (rows contiguous), its transpose as the column one
        assert np.array_equal(ctx.oz_gemm(A, eye, slices=S, tri_a=tri), want)
        tb = (0, 2, 1)[tri]
        assert np.array_equal(ctx.oz_gemm(eye, np.ascontiguousarray(A.T), slices=S, tri_b=tb), want.T)


@pytest.mark.parametrize("nmol", [44, 45])
def test_product_on_both_sides_of_one_wave(ctx, nmol):
    """ndim 1012 (128 tiles of 128 x 64) and 1035 (CTA pairs): diag(s2 P s1) against
    FP64 within the bound of six slices, 3 K 2^-42 2^(e_i + f_j) per element of P s1."""
    s = synth.water_cluster(nmol, seed=2)
    n = s.ndim
    sh = synth.shell2ao(s.aoat)
    rng = np.random.default_rng(nmol)
    P = rng.standard_normal((n, n))
    P += P.T
    s1 = rng.standard_normal((n, n)).astype(np.float32)
    s2 = rng.standard_normal((n, n)).astype(np.float32)
    q, qsh, _ = ctx.mlpop2(s.nat, n, O.packsym(P), s1, s2, s.aoat, sh)
    q64, qsh64 = O.mlpop2(s.nat, n, O.packsym(P), s1, s2, s.aoat, sh, dtype=np.float64)
    e = np.frexp(np.max(np.abs(P), axis=1))[1]
    f = np.frexp(np.max(np.abs(s1), axis=0))[1]
    # an atom has at most n of the n diagonal elements, each a sum over n rows of P s1
    tol = n * 3.0 * n * 2.0 ** (-42) * 2.0 ** (e.max() + f.max()) * np.max(np.sum(np.abs(s2), axis=1)) / n
    assert np.max(np.abs(q - q64)) < tol
    assert np.max(np.abs(qsh - qsh64)) < tol
