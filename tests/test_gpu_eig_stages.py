"""The eigensolver's stages at the orders where their shapes change, against LAPACK:
64-row blocks of the Cholesky factor and of the triangular solves, 64-reflector panels
(order - 2 a multiple of 64 and its neighbours), 32-column panels and 64- and
128-row strips of the tridiagonalisations, the last order of one CTA with 256 and with
512 threads (288, 800), cluster shapes above, and owned counts around one 64-vector
task.  Tolerances are those of the batched solver's own tests: eigenvalues to 1e-11
of the spectral range times sqrt(m), fe and P to 1e-10.
"""
import numpy as np
import pytest
import scipy.linalg as sl

from ptb_b200 import PtbGpuError

pytestmark = pytest.mark.gpu


def _problem(m, rng, nown):
    A = rng.standard_normal((m, m))
    S = A @ A.T / m + np.eye(m)                # SPD, condition ~ 5
    H = rng.uniform(-1, 1, (m, m))
    H = 0.5 * (H + H.T) + np.diag(rng.uniform(-2, 2, m))
    return H, S, np.sort(rng.choice(m, size=min(nown, m), replace=False))


def _check(prob, got, mu):
    H, S, own = prob
    e, fe, Pc = got
    m = H.shape[0]
    er, U = sl.eigh(H, S)
    order = np.argsort(e, kind="stable")
    assert np.max(np.abs(e[order] - er)) <= 1e-11 * max(1.0, np.max(np.abs(er))) * max(1.0, np.sqrt(m)), m
    assert np.max(np.abs(fe[order] - np.sum((S @ U)[own, :] * U[own, :], axis=0))) <= 1e-10, m
    occ = np.where(er < mu, 2.0, np.where(er == mu, 1.0, 0.0))
    assert np.max(np.abs(Pc - (U * occ) @ U[own, :].T)) <= 1e-10, m


@pytest.mark.parametrize("m", [2, 3, 4, 63, 64, 66, 67, 92, 128, 130, 131, 193, 287, 288, 289, 576, 737, 799, 800, 801,
                               1025, 1473])
def test_one_problem_at_the_edges(ctx, m):
    """Alone: tridiagonalised by the widest group of CTAs that pays."""
    rng = np.random.default_rng(m)
    prob = _problem(m, rng, (1, 64, 65, m)[m % 4])
    _check(prob, ctx.sygv_batched([prob], mu=0.05)[0], 0.05)


@pytest.mark.parametrize("top", [130, 289])
def test_more_problems_than_sms(ctx, top):
    """A batch that fills the SMs: one CTA each, two per SM up to order 288, the orders
    around the blocks, panels and strips side by side."""
    rng = np.random.default_rng(top)
    orders = [1, 2, 31, 32, 33, 34, 64, 65, 66, 67, 96, 97, 127, 128, 129, top - 1, top]
    probs = [_problem(orders[q % len(orders)], rng, 1 + q % 70) for q in range(320)]
    out = ctx.sygv_batched(probs, mu=0.05)
    for prob, got in list(zip(probs, out))[::7]:
        _check(prob, got, 0.05)


@pytest.mark.parametrize("m", [65, 200, 900])
def test_ill_conditioned_overlap(ctx, m):
    """Condition 1e6 of S: the solves with inverted 64 x 64 blocks keep LAPACK's backward
    error, m eps max|e|, on the eigenvalues, and sum fe = owned rows to m eps cond."""
    rng = np.random.default_rng(m)
    Q, _ = np.linalg.qr(rng.standard_normal((m, m)))
    S = (Q * np.logspace(0, -6, m)) @ Q.T
    S = 0.5 * (S + S.T)
    H, _, own = _problem(m, rng, 20)
    e, fe, _ = ctx.sygv_batched([(H, S, own)], mu=0.0)[0]
    er = sl.eigh(H, S, eigvals_only=True)
    assert np.max(np.abs(np.sort(e) - er)) <= 1e-11 * np.max(np.abs(er)) * np.sqrt(m)
    assert abs(np.sum(fe) - len(own)) <= m * 2.3e-16 * 1e6


@pytest.mark.parametrize("m,bad", [(40, 1), (130, 64), (130, 65), (200, 130), (900, 900)])
def test_first_non_positive_pivot_is_named(ctx, m, bad):
    """The order of the first non-positive pivot, in any 64-row block."""
    rng = np.random.default_rng(m + bad)
    H, S, own = _problem(m, rng, 3)
    S[bad - 1, bad - 1] = -1.0
    with pytest.raises(PtbGpuError, match=rf"leading minor {bad}\)"):
        ctx.sygv_batched([(H, S, own)], mu=0.0)
