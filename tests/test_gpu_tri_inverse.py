"""The triangular inverse by doubling (the orthogonalisation's L^-1) and, in FP64, the
tile products with it, at the orders where their blocks change: a density step's
tr(PS) and P feel every element of L^-1, so both precisions are compared with LAPACK's
projector on systems whose order is one 64-row block, a ragged second one, and levels
with a short or a missing last block."""
import numpy as np
import pytest
import scipy.linalg as sl

from oracle import ptb_oracle as O
from ptb_b200 import PREC_FP64, PREC_MIXED, Options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 63, 64, 65, 127, 128, 129, 192, 193, 320, 449, 577, 1025, 1100])
@pytest.mark.parametrize("precision,tol", [(PREC_MIXED, 1e-6), (PREC_FP64, 1e-9)])
def test_density_step_through_the_inverse(ctx, n, precision, tol):
    rng = np.random.default_rng(n)
    # a gap of 1 between the halves of the spectrum, and an overlap of condition ~ 10
    nocc = n // 2
    A = rng.standard_normal((n, n))
    S = A @ A.T / n * 0.9 + 0.4 * np.eye(n)
    L = np.linalg.cholesky(S)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    e = np.concatenate([-1.0 - rng.random(nocc), 0.0 + rng.random(n - nocc)])
    H = L @ (Q * e) @ Q.T @ L.T
    H = 0.5 * (H + H.T)
    P, st = ctx.tc_purify(n, 2 * nocc, O.packsym(H), O.packsym(S), Options(filter=0.0, precision=precision))
    _, U = sl.eigh(H, S)
    ref = 2.0 * U[:, :nocc] @ U[:, :nocc].T
    assert np.max(np.abs(O.blowsym(n, P) - ref)) <= tol
    assert abs(np.sum(O.blowsym(n, P) * S) - 2 * nocc) <= 1e-8
