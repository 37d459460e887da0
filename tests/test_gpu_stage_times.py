"""Device times that a batch of the eigensolver reports at print level 2."""
import re

import numpy as np
import pytest

from ptb_b200 import Options, synth

pytestmark = pytest.mark.gpu

STAGES = ["Cholesky", "reduction", "tridiagonalisation", "panels", "divide and conquer", "vectors"]


def _weakly_coupled(n, seed):
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    d = i * (i + 3) // 2                           # packed position of (i, i)
    H = np.zeros(n * (n + 1) // 2)
    S = np.zeros_like(H)
    H[d] = np.where(i < n // 4, -1.0, 1.0) + 0.1 * rng.random(n)
    S[d] = 1.0
    H[d[1:] - 1] = 0.02 * rng.standard_normal(n - 1)
    S[d[1:] - 1] = 0.05
    return n, 2 * (n // 4), H, S


def test_stage_times_of_a_batch(ctx, capfd):
    """At print level 2 every stage of the submatrix method's batch and of each part of a
    host batch is reported with its device time."""
    s = synth.water_cluster(8, seed=5)
    _, st = ctx.sm_stupid_simple(s.ndim, s.nel, s.Hvec, s.Svec, s.nat, s.xyz, s.aoat, 2, 2, None,
                                 Options(filter=1e-4, print_level=2))
    large, small = _weakly_coupled(801, 1), _weakly_coupled(70, 2)
    _, _, wall = ctx.eig_density_batch([large] * 24 + [small], Options(filter=0.0, print_level=2))
    lines = re.findall(r"eigensolver stage (.+?) +([\d.]+) ms", capfd.readouterr().out)
    assert [name for name, _ in lines] == 4 * STAGES           # one batch, then two parts and the small system
    ms = np.array([float(t) for _, t in lines])
    assert np.all(ms > 0.0)
    assert np.sum(ms[:6]) <= st.ms_total and np.sum(ms[12:]) <= 2.0 * wall
