"""Trace-correcting purification of systems with many states right above a small gap, the
highest occupied one among them.  On the way X^2 takes all of these down to a few hundredths
together, with an idempotency error far below one and the trace an electron short; the
occupied one then doubles its way back.  Every precision and the grouped entry against
LAPACK's projector, with the tolerances of the mixed step's own tests (1e-6; 1e-9 for
FP64; the electron count to 1e-8), and an impossible iteration limit refused.
"""
import numpy as np
import pytest
import scipy.linalg as sl

from oracle import ptb_oracle as O
from ptb_b200 import PREC_FP64, PREC_MIXED, Options, PtbGpuError, api

pytestmark = pytest.mark.gpu


def _system(n, near, gap, seed):
    """n // 4 occupied states, the highest at -gap, `near` empty ones within 8 gaps above."""
    rng = np.random.default_rng(seed)
    nocc = n // 4
    e = np.concatenate([-1.0 - 0.5 * rng.random(nocc - 1), [-gap], 8.0 * gap * rng.random(near),
                        0.5 + 0.5 * rng.random(n - nocc - near)])
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = rng.standard_normal((n, n))
    S = A @ A.T / n * 0.5 + 0.5 * np.eye(n)        # condition about 5
    L = np.linalg.cholesky(S)
    H = (L @ (Q * e)) @ (L @ Q).T
    H = 0.5 * (H + H.T)
    U = sl.eigh(H, S)[1][:, :nocc]
    return (n, 2 * nocc, O.packsym(H), O.packsym(S)), 2.0 * U @ U.T, S


def _check(n, nel, P, ref, S, tol):
    P = O.blowsym(n, P)
    assert np.max(np.abs(P - ref)) <= tol
    assert abs(np.sum(P * S) - nel) <= 1e-8


CASES = [(130, 10, 1e-2), (130, 60, 1e-2), (300, 30, 3e-3), (520, 60, 1e-2), (520, 10, 3e-3)]


@pytest.mark.parametrize("n,near,gap", CASES)
@pytest.mark.parametrize("precision,slices,tol", [(PREC_MIXED, 8, 1e-6), (PREC_MIXED, 0, 1e-6), (PREC_FP64, 8, 1e-9)])
def test_states_close_to_the_gap(ctx, n, near, gap, precision, slices, tol):
    (n, nel, H, S), ref, Sf = _system(n, near, gap, seed=n + near)
    P, _ = ctx.tc_purify(n, nel, H, S, Options(filter=0.0, precision=precision, fp64_slices=slices))
    _check(n, nel, P, ref, Sf, tol)


@pytest.mark.parametrize("precision,tol", [(PREC_MIXED, 1e-6), (PREC_FP64, 1e-9)])
def test_states_close_to_the_gap_grouped(ctx, precision, tol):
    made = [_system(n, near, gap, seed=n + near) for n, near, gap in CASES]
    Ps, _, _ = ctx.tc_purify_grouped([m[0] for m in made], Options(filter=0.0, precision=precision))
    for ((n, nel, _, _), ref, Sf), P in zip(made, Ps):
        _check(n, nel, P, ref, Sf, tol)


@pytest.mark.parametrize("precision", [PREC_MIXED, PREC_FP64])
def test_too_few_iterations_are_refused(ctx, precision):
    (n, nel, H, S), _, _ = _system(300, 30, 3e-3, seed=1)
    with pytest.raises(PtbGpuError) as ei:
        ctx.tc_purify(n, nel, H, S, Options(filter=0.0, precision=precision, max_iter=40))
    assert ei.value.code == api.EITER


@pytest.mark.parametrize("precision,tol", [(PREC_MIXED, 1e-6), (PREC_FP64, 1e-9)])
@pytest.mark.parametrize("pairs", [1, 2, -1, 0])
def test_few_electrons_and_few_holes(ctx, water8, pairs, precision, tol):
    """One or two occupied states, one empty one, none: the neighbours in energy are in the
    middle of a band there."""
    s = water8
    n = s.ndim
    nel = 2 * (pairs if pairs > 0 else n + pairs)
    H, S = O.blowsym(n, s.Hvec), O.blowsym(n, s.Svec)
    U = sl.eigh(H, S)[1][:, : nel // 2]
    opts = Options(filter=0.0, precision=precision)
    _check(n, nel, ctx.tc_purify(n, nel, s.Hvec, s.Svec, opts)[0], 2.0 * U @ U.T, S, tol)
    _check(n, nel, ctx.tc_purify_grouped([(n, nel, s.Hvec, s.Svec)], opts)[0][0], 2.0 * U @ U.T, S, tol)


@pytest.mark.parametrize("precision", [PREC_MIXED, PREC_FP64])
@pytest.mark.parametrize("nel", [2, 78, 80])
def test_exact_spectral_bounds(ctx, nel, precision):
    """Uncoupled states, for which the bounds of the spectrum are its ends."""
    n = 40
    e = np.sort(np.random.default_rng(1).random(n))
    H, S = O.packsym(np.diag(e)), O.packsym(np.eye(n))
    opts = Options(filter=0.0, precision=precision)
    ref = np.diag(2.0 * (np.arange(n) < nel // 2))
    _check(n, nel, ctx.tc_purify(n, nel, H, S, opts)[0], ref, np.eye(n), 1e-9)
    _check(n, nel, ctx.tc_purify_grouped([(n, nel, H, S)], opts)[0][0], ref, np.eye(n), 1e-9)


@pytest.mark.parametrize("nmol,seed", [(130, 31), (190, 27)])
def test_frontier_state_below_the_floor_of_pass_1(ctx, nmol, seed):
    """Boxes whose pass 1 ends with a frontier state a percent away from 0 or 1, under the
    rounding noise of the traces: one refinement round leaves more than refine_tol (1e-7, in
    the orthogonal basis) although its gain predicts half of that.  Against the library's
    FP64 dense diagonalisation."""
    from ptb_b200 import synth

    s = synth.water_cluster(nmol, seed=seed)
    n = s.ndim
    P, st = ctx.tc_purify(n, s.nel, s.Hvec, s.Svec, Options(filter=1e-5, precision=PREC_MIXED))
    ref, _, focc, _ = ctx.solve2(1, n, s.nel, 0, s.Hvec, s.Svec, Options(filter=1e-5))
    assert np.array_equal(np.sort(focc)[::-1][: s.nel // 2], np.full(s.nel // 2, 2.0))
    L = np.linalg.cholesky(O.blowsym(n, O.filter_matrix_sym(s.Svec, 1e-5)))
    d = L.T @ O.blowsym(n, P - ref) @ L
    assert np.max(np.abs(d)) / 2.0 <= 1e-7
    assert st.refine_rounds >= 2 and st.fp64_fallback == 0
