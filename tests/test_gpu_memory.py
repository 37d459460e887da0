"""Device memory that the library takes and keeps."""
import gc

import numpy as np
import pytest

from oracle import ptb_oracle as O
from ptb_b200 import PREC_FP64, Context, Options, PurificationSettings, synth

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


@pytest.fixture(scope="module")
def medium():
    """One system of order 801 and its projector: a batch of many shares the host arrays."""
    n = 801
    H, S = _gapped(n)
    ref, _ = O.dense_projector(O.blowsym(n, H), O.blowsym(n, S), 2 * (n // 4))
    return (n, 2 * (n // 4), H, S), ref


def _solve(c, medium, count):
    system, ref = medium
    Ps = c.eig_density_batch([system] * count)[0]
    for P in Ps[:: max(1, count // 5)]:
        assert np.max(np.abs(O.blowsym(system[0], P) - ref)) <= 1e-8


def test_trim_gives_back_what_is_kept(medium):
    """A batch whose arrays (about 17 GB) exceed what may be kept: 1/16 of the device at most
    stays, trim returns it, and the next call is served."""
    import torch

    total = torch.cuda.mem_get_info()[1]
    with Context(0) as c:
        c.filter_matrix_sym(medium[0][2], medium[0][0], 0.0)
        _solve(c, medium, 420)
        before = _free()
        c.trim()
        kept = _free() - before
        assert 0 < kept <= total / 16
        c.trim()
        _solve(c, medium, 3)


def test_trim_between_the_phases_of_the_submatrix_method():
    s = synth.water_cluster(12, seed=4)
    opts = Options(filter=1e-4)
    with Context(0) as c:
        P, st = c.sm_stupid_simple(s.ndim, s.nel, s.Hvec, s.Svec, s.nat, s.xyz, s.aoat, 2, 2, None, opts)
        ids = np.arange(c.sm_plan(s.ndim, s.Hvec, s.Svec, s.nat, s.xyz, s.aoat, 2, 2, None, opts).shape[0])
        c.trim()
        c.sm_prepare(ids)
        c.trim()
        assert c.sm_nel(st.mu) == pytest.approx(st.nel, abs=1e-12)
        assert np.array_equal(c.sm_finish(s.ndim, st.mu), P)


def test_kept_blocks_make_room_for_another_context(medium):
    """With less free memory than a call needs, the blocks that another context keeps are
    freed for it."""
    import torch

    with Context(0) as a, Context(0) as b:
        _solve(b, medium, 2)
        _solve(a, medium, 200)                     # keeps several GB
        left = _free()
        hold = torch.empty(left - (3 << 30), dtype=torch.uint8, device="cuda")
        try:
            _solve(b, medium, 100)                 # about 4 GB
        finally:
            del hold
            torch.cuda.empty_cache()


def test_a_call_takes_what_its_arrays_need(medium):
    """419 systems of order 801: nine arrays of 2.15 GB and 0.5 GB of smaller ones, 19.9 GB in
    all, with 20.6 GB free.  (Just above a power of two: blocks rounded up by an eighth
    would come to 22.)"""
    import torch

    with Context(0) as c:
        _solve(c, medium, 2)
        c.trim()
        hold = torch.empty(_free() - int(20.6e9), dtype=torch.uint8, device="cuda")
        try:
            _solve(c, medium, 419)
        finally:
            del hold
            torch.cuda.empty_cache()


def test_trim_after_purification():
    s = synth.water_cluster(8, seed=5)
    pur = PurificationSettings(type=1, metric_type=1, cycles=100, prlvl=0, nel=s.nel)
    with Context(0) as c:
        P, _ = c.purification(pur, s.ndim, s.Hvec, s.Svec, Options(filter=1e-4))
        c.trim()
        Q, _ = c.purification(pur, s.ndim, s.Hvec, s.Svec, Options(filter=1e-4))
    assert np.array_equal(P, Q)
