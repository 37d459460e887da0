"""Device memory that the library takes and keeps."""
import gc

import numpy as np
import pytest

from ptb_b200 import PREC_FP64, Context, Options

pytestmark = pytest.mark.gpu


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _gapped(n, seed=3):
    """Packed H and S of a weakly coupled gapped system: unit overlap but for one near diagonal."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    d = i * (i + 3) // 2                           # packed position of (i, i)
    H = np.zeros(n * (n + 1) // 2)
    S = np.zeros_like(H)
    H[d] = np.where(i < n // 4, -1.0, 1.0) + 0.1 * rng.random(n)
    S[d] = 1.0
    H[d[1:] - 1] = 0.02 * rng.standard_normal(n - 1)
    S[d[1:] - 1] = 0.05
    return H, S


def test_triangular_inverse_adds_no_matrix():
    """FP64 steps of orders on both sides of 64 * 2^6, where the inverse's last level has a
    short block of 64 rows: what the call takes grows with its arrays (three n x n, three
    packed: 19 MB in all), not by a scratch of 4096 x 4096 (128 MB)."""
    opts = Options(filter=0.0, precision=PREC_FP64)
    taken = []
    for n in (4096, 4160):
        gc.collect()
        H, S = _gapped(n)
        with Context(0) as c:
            before = _free()
            P, _ = c.tc_purify(n, 2 * (n // 4), H, S, opts)
            taken.append(before - _free())
        i = np.arange(n)
        d = i * (i + 3) // 2
        assert abs(np.sum(P[d]) + 2 * 0.05 * np.sum(P[d[1:] - 1]) - 2 * (n // 4)) <= 1e-7
    assert taken[1] - taken[0] <= 64 << 20
