"""How many CTAs tridiagonalise a problem.

An uneven batch of orders up to 799 (none a multiple of 8, so that strips, chunks and
panels end raggedly) for which the clock model picks one CTA for its small problems and clusters of
2, 4 and 8 for the others, and a batch with an order above 5120, which no cluster's
shared memory holds.  Against projectors known by construction, max|dP| <= 1e-8 as in the batch's tests.
"""
import re

import numpy as np
import pytest
import scipy.linalg as sl

from oracle import ptb_oracle as O
from ptb_b200 import Options

pytestmark = pytest.mark.gpu


def _levels(n, rng):
    """A gap of 1 at half filling."""
    return np.concatenate([-1.0 - rng.random(n // 2), rng.random(n - n // 2)])


def _dense(n, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((n, n))
    S = A @ A.T / n + np.eye(n)                    # condition about 5
    L = np.linalg.cholesky(S)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    H = (L @ (Q * _levels(n, rng))) @ (L @ Q).T
    U = sl.solve_triangular(L.T, Q[:, : n // 2])
    return (n, 2 * (n // 2), O.packsym(0.5 * (H + H.T)), O.packsym(S)), 2.0 * U @ U.T


def _reflected(n, seed):
    """The same from three reflectors and a bidiagonal L, for an order where dense factors
    take the host too long."""
    rng = np.random.default_rng(seed)
    e = _levels(n, rng)
    A, B = np.diag(e), np.diag((np.arange(n) < n // 2).astype(float))
    for _ in range(3):
        v = rng.standard_normal(n)
        v /= np.linalg.norm(v)
        for M in (A, B):                           # M <- (I - 2 v v^T) M (I - 2 v v^T)
            w = M @ v
            M -= 2.0 * np.outer(v, w) + 2.0 * np.outer(w, v) - 4.0 * (v @ w) * np.outer(v, v)
    L = np.eye(n) + np.diag(np.full(n - 1, 0.3), -1)
    H, S = L @ A @ L.T, L @ L.T
    P = sl.solve_triangular(L.T, sl.solve_triangular(L.T, B).T).T
    return (n, 2 * (n // 2), O.packsym(0.5 * (H + H.T)), O.packsym(S)), P + P.T


def _groups(text):
    """(problems, CTAs) of every tridiagonalisation launch reported."""
    return [(int(a), int(b)) for a, b in re.findall(r"tridiagonalisation of (\d+) on (\d+) CTAs", text)]


def test_one_batch_on_groups_of_every_size(ctx, capfd):
    orders = [363 + (71 * i) % 437 for i in range(48)]
    orders = [n + 1 if n % 8 == 0 else n for n in orders]
    made = [_dense(n, n) for n in orders]
    Ps = ctx.eig_density_batch([m[0] for m in made], Options(filter=0.0, print_level=2))[0]
    groups = _groups(capfd.readouterr().out)
    assert {g for _, g in groups} >= {1, 2, 4, 8} and sum(c for c, _ in groups) == len(orders)
    for ((n, *_), ref), P in zip(made, Ps):
        assert np.max(np.abs(O.blowsym(n, P) - ref)) <= 1e-8, n


def test_order_beyond_every_clusters_shared_memory(ctx, capfd):
    made = [_reflected(5130, 1), _dense(130, 2)]
    Ps = ctx.eig_density_batch([m[0] for m in made], Options(filter=0.0, print_level=2))[0]
    assert sum(c for c, _ in _groups(capfd.readouterr().out)) == 2
    for ((n, *_), ref), P in zip(made, Ps):
        assert np.max(np.abs(O.blowsym(n, P) - ref)) <= 1e-8, n
