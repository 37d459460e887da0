"""The dense step with an overlap of condition 1e6.  A and P are formed with L^-1, so the
condition enters as it does for LAPACK's solves: P, the electron count and idempotency
within n eps cond(S) (of max|P| where they scale with it), in FP64 and with the FP64
tile products of the mixed step."""
import numpy as np
import pytest
import scipy.linalg as sl

from oracle import ptb_oracle as O
from ptb_b200 import PREC_FP64, PREC_MIXED, Options

pytestmark = pytest.mark.gpu

COND, EPS = 1e6, 2.0 ** -52


@pytest.mark.parametrize("n", [65, 129, 320, 1025])
@pytest.mark.parametrize("precision,own", [(PREC_FP64, 0.0), (PREC_MIXED, 1e-6)])
def test_condition_of_the_overlap(ctx, n, precision, own):
    """own: what the step may be off by itself (the mixed step's tolerance)."""
    rng = np.random.default_rng(n)
    nocc = n // 2
    V, _ = np.linalg.qr(rng.standard_normal((n, n)))
    S = (V * np.logspace(0, -np.log10(COND), n)) @ V.T
    S = 0.5 * (S + S.T)
    L = np.linalg.cholesky(S)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    e = np.concatenate([-1.0 - rng.random(nocc), rng.random(n - nocc)])
    H = (L @ (Q * e)) @ (L @ Q).T
    H = 0.5 * (H + H.T)
    U = sl.eigh(H, S)[1][:, :nocc]
    ref = 2.0 * U @ U.T
    P, _ = ctx.tc_purify(n, 2 * nocc, O.packsym(H), O.packsym(S),
                         Options(filter=0.0, precision=precision, fp64_slices=0))
    P = O.blowsym(n, P)
    tol = n * EPS * COND
    assert np.max(np.abs(P - ref)) <= (tol + own) * np.max(np.abs(ref))
    assert abs(np.sum(P * S) - 2 * nocc) <= max(tol, 1e-8)
    if precision == PREC_FP64:
        assert np.max(np.abs(P @ S @ P - 2.0 * P)) <= 2.0 * tol * np.max(np.abs(ref))
