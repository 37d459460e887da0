"""The batch of independent systems in its parts (ptbgpu_eig_density_batch): systems above
order 800 go in two, three or four parts from 24, 72 and 96 of them on, the others beside
them.  Every part's results against LAPACK's dense projector, and the failure of a part
while others are on their way: the first failing system of the call is named whichever
part or group it is in, and the context serves the next call.
FP64 throughout: max|dP| <= 1e-8 as in the batch's other tests.
"""
import numpy as np
import pytest

from oracle import ptb_oracle as O
from ptb_b200 import PtbGpuError, api

pytestmark = pytest.mark.gpu


def _system(n, seed):
    """A gap of 1 at half filling and an overlap of condition about 5."""
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((n, n))
    S = A @ A.T / n + np.eye(n)
    L = np.linalg.cholesky(S)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    e = np.concatenate([-1.0 - rng.random(n // 2), rng.random(n - n // 2)])
    H = (L @ (Q * e)) @ (L @ Q).T
    H = 0.5 * (H + H.T)
    P, _ = O.dense_projector(H, S, 2 * (n // 2))
    return (n, 2 * (n // 2), O.packsym(H), O.packsym(S)), P


@pytest.fixture(scope="module")
def large():
    return [_system(801, 1), _system(834, 2)]


@pytest.fixture(scope="module")
def small():
    return _system(90, 3)


def _indefinite(system):
    n, nel, H, S = system
    bad = S.copy()
    bad[0] = -1.0                                   # S_11 < 0
    return (n, nel, H, bad)


def _check(made, Ps):
    for (system, ref), P in zip(made, Ps):
        assert np.max(np.abs(O.blowsym(system[0], P) - ref)) <= 1e-8


@pytest.mark.parametrize("count", [23, 24, 72, 96])
def test_every_part_is_solved(ctx, large, small, count):
    made = [large[(5 * k % 7) % 2] for k in range(count)]
    made.insert(count // 2, small)
    _check(made, ctx.eig_density_batch([m[0] for m in made])[0])


@pytest.mark.parametrize("bad,named", [([23], 24), ([3, 23], 4), ([23, 24], 24), ([24], 25), ([0, 24], 1)])
def test_the_first_failing_system_is_named(ctx, large, small, bad, named):
    """24 large systems (two parts), the small one after them."""
    made = [large[k % 2] for k in range(24)] + [small]
    systems = [_indefinite(m[0]) if k in bad else m[0] for k, m in enumerate(made)]
    with pytest.raises(PtbGpuError) as ei:
        ctx.eig_density_batch(systems)
    assert ei.value.code == api.ENOTSPD and f"system {named} not" in str(ei.value)
    _check(made, ctx.eig_density_batch([m[0] for m in made])[0])


def test_a_failure_in_the_last_of_four_parts(ctx, large):
    made = [large[k % 2] for k in range(96)]
    systems = [m[0] for m in made]
    systems[95] = _indefinite(systems[95])
    with pytest.raises(PtbGpuError, match="system 96 not positive definite"):
        ctx.eig_density_batch(systems)
    _check(made[:30], ctx.eig_density_batch([m[0] for m in made[:30]])[0])
