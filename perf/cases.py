"""The density-matrix work a user of ptb_b200 has it do, as measurable cases.

A case names an entry point of the library, a system and the options of the call.  The systems are the synthetic
tight-binding pairs of ptb_b200.synth (same geometry, basis, H and S recipe), built on the GPU so that a large box
takes a fraction of a second: water boxes at 1 g/cm^3, all-trans alkanes and jittered cubic lattices.

Kinds of call:
  sm      Context.sm_stupid_simple: the submatrix method, one SCF iteration's density step (host arrays in and out)
  tc      Context.tc_purify_device / tc_purify: the dense trace-correcting purification, mixed precision or FP64
  solve2  Context.solve2: the dense diagonalisation with Fermi occupations
  purify  Context.purification: the full-matrix purification module with its chemical-potential search
  batch   Context.eig_density_batch: many independent molecules in one call
  mlpop2  Context.mlpop2_device: atomic and shell populations of a density left on the device
  xc      Context.xc_damping_device: the long-range damping term that the next iteration adds to H
"""
import math

import numpy as np
import torch

from ptb_b200 import PREC_FP64, PREC_MIXED, Context, Options, PurificationSettings, synth

DEV = "cuda:0"
BOHR = 1.0 / 0.52917721092
MOLECULES_PER_CLUSTER = 10          # columns mode 4: about this many molecules per cluster

_context = None


def context():
    """The one context a program keeps for its device."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


def listed():
    return [
        # the smallest job of the method: a water tetramer, where the call is launches and latency
        {"name": "sm_water4", "kind": "sm", "mol": "water", "size": 4, "columns": 2, "filter": 1e-4},
        # the standard cluster with per-atom columns, the method's default (ndim 736)
        {"name": "sm_water32", "kind": "sm", "mol": "water", "size": 32, "columns": 2, "filter": 1e-4},
        # a long chain: hundreds of small submatrices of a sparse system (ndim 4610)
        {"name": "sm_alkane200", "kind": "sm", "mol": "alkane", "size": 200, "columns": 2, "filter": 1e-4},
        # a large box with the columns grouped by the caller's clustering: tens of submatrices of 700 to 2800 (ndim 11776)
        {"name": "sm_clusters512", "kind": "sm", "mol": "water", "size": 512, "columns": 4, "filter": 1e-4},
        # the dense diagonalisation that check mode and small molecules use, odd order (ndim 1495)
        {"name": "solve2_water65", "kind": "solve2", "mol": "water", "size": 65, "filter": 1e-5},
        # the purification module, McWeeny with the mu search, on the standard cluster (ndim 736)
        {"name": "purify_mcweeny32", "kind": "purify", "mol": "water", "size": 32, "type": 1, "filter": 1e-4},
        # the dense step of the 512-molecule box with H, S and P kept on the device (ndim 11776)
        {"name": "tc_water512", "kind": "tc", "mol": "water", "size": 512, "mixed": True, "device": True, "filter": 1e-5},
        # the same step for a medium molecule from host arrays, odd order (ndim 1495)
        {"name": "tc_host_water65", "kind": "tc", "mol": "water", "size": 65, "mixed": True, "device": False,
         "filter": 1e-5},
        # the dense step where the caller asks for FP64 throughout (ndim 2208)
        {"name": "tc_fp64_water96", "kind": "tc", "mol": "water", "size": 96, "mixed": False, "device": True,
         "filter": 1e-5},
        # many uneven molecules in one call, as a screening run has them (ndim about 170 to 3060)
        {"name": "batch_lattice32", "kind": "batch", "size": 32, "atoms": 400},
        # populations after every density step, P and the powers of S on the device (ndim 5888)
        {"name": "mlpop2_water256", "kind": "mlpop2", "mol": "water", "size": 256},
        # the damping term of the second iteration on the large box (ndim 11776)
        {"name": "xc_water512", "kind": "xc", "mol": "water", "size": 512},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["sm", "sm", "sm", "sm4", "solve2", "purify", "tc", "tc", "batch", "mlpop2", "xc"])
    if kind == "sm":
        mol = rng.choice(["water", "alkane"])
        columns = rng.choice([1, 2, 2, 2, 3])
        top = {1: (24, 200), 2: (64, 200), 3: (64, 90)}[columns][mol == "alkane"]
        return {"kind": "sm", "mol": mol, "size": spread(3, top), "columns": columns, "filter": rng.choice([1e-4, 1e-5])}
    if kind == "sm4":
        return {"kind": "sm", "mol": "water", "size": spread(40, 400), "columns": 4, "filter": 1e-4}
    if kind == "solve2":
        return {"kind": "solve2", "mol": "water", "size": spread(3, 150), "filter": rng.choice([0.0, 1e-5])}
    if kind == "purify":
        return {"kind": "purify", "mol": "water", "size": spread(4, 48), "type": rng.choice([1, 2, 3, 4]), "filter": 1e-4}
    if kind == "tc":
        mixed = rng.choice([True, True, False])
        return {"kind": "tc", "mol": "water", "size": spread(4, 400 if mixed else 150), "mixed": mixed,
                "device": rng.choice([True, False]), "filter": 1e-5}
    if kind == "batch":
        return {"kind": "batch", "size": spread(2, 32), "atoms": spread(40, 400)}
    return {"kind": kind, "mol": "water", "size": spread(4, 400)}


# ---- inputs --------------------------------------------------------------------------------------------------

def packed_index(n):
    """Column and row of every packed element in storage order (column c, rows <= c)."""
    return torch.tril_indices(n, n, device=DEV)


class Molecule:
    """Geometry, basis layout and the packed H and S (unfiltered) of one system, on the GPU."""

    def __init__(self, symbols, xyz, seed, amp, matrices=True):
        self.xyz = np.ascontiguousarray(xyz, dtype=np.float64)
        self.aoat, self.slots, occ = synth.basis_layout(symbols)
        self.n, self.nat, self.nel = int(self.aoat.shape[0]), int(self.xyz.shape[0]), 2 * int(occ.sum())
        self.at = torch.from_numpy(self.aoat - 1).to(DEV)
        self.slot = torch.from_numpy(self.slots).to(DEV)
        x = torch.from_numpy(self.xyz).to(DEV)
        self.dist = (x[:, None, :] - x[None, :, :]).square().sum(-1).sqrt()
        self.gen = torch.Generator(device=DEV).manual_seed(seed)
        if not matrices:
            return
        c, r = packed_index(self.n)
        apart = self.dist[self.at[c], self.at[r]]
        same = (self.slot[c] == self.slot[r]) & (self.at[c] != self.at[r])
        self.S = torch.where(same, torch.exp(-0.5 * apart * apart), 0.0)
        del same
        self.H = torch.exp(-apart).mul_(amp)
        del apart
        self.H *= torch.rand(self.H.shape, generator=self.gen, device=DEV, dtype=torch.float64).mul_(2).sub_(1)
        diag = torch.arange(1, self.n + 1, device=DEV)
        diag = diag * (diag + 1) // 2 - 1
        level = torch.where(torch.from_numpy(occ).to(DEV), -0.5, 0.3).double()
        self.H[diag] = level + 0.1 * torch.randn(self.n, generator=self.gen, device=DEV, dtype=torch.float64)
        self.S[diag] = 1.0


def molecule(case, seed, matrices=True):
    if case["mol"] == "alkane":
        symbols, xyz = synth.alkane_geometry(case["size"], seed)
    else:
        symbols, xyz, _ = synth.water_cluster_geometry(case["size"], seed)
    return Molecule(symbols, xyz, seed, synth.MOLECULAR_AMP, matrices)


def lattices(case, seed):
    """The systems of a batch: 20 atoms up to the case's largest, in scattered order."""
    rng = np.random.default_rng(seed)
    made = []
    for k in range(case["size"]):
        nat = case["atoms"] - int((case["atoms"] - 20) * (0.6180339887 * k % 1.0))
        symbols, xyz = synth.lattice_geometry(nat, int(rng.integers(1 << 30)))
        made.append(Molecule(symbols, xyz, seed * 1009 + k, synth.LATTICE_AMP))
    return made


def clustering(m, molecules, seed):
    """Atom -> cluster ids (1-based) of whole water molecules: Lloyd's iterations on the oxygens."""
    rng = np.random.default_rng(seed)
    k = max(1, molecules // MOLECULES_PER_CLUSTER)
    o = m.xyz[::3]
    centre = o[rng.permutation(molecules)[:k]].copy()
    for _ in range(20):
        near = np.argmin(((o[:, None, :] - centre[None]) ** 2).sum(-1), axis=1)
        for j in range(k):
            if np.any(near == j):
                centre[j] = o[near == j].mean(0)
    _, near = np.unique(near, return_inverse=True)
    return np.repeat(near.reshape(-1).astype(np.int64) + 1, 3)


def pinned(t):
    """A page-locked host copy, as a program that calls the library on every iteration keeps its arrays."""
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()


def density_like(m):
    """A packed symmetric matrix with a density's size and decay with distance."""
    c, r = packed_index(m.n)
    p = torch.exp(-0.7 * m.dist[m.at[c], m.at[r]])
    p *= torch.randn(p.shape, generator=m.gen, device=DEV, dtype=torch.float64).mul_(0.2)
    diag = torch.arange(1, m.n + 1, device=DEV)
    p[diag * (diag + 1) // 2 - 1] = 2.0 * torch.rand(m.n, generator=m.gen, device=DEV, dtype=torch.float64)
    return p


def overlap_powers(m, x):
    """S^(1-x) and S^x in float32: S couples equal slots only, so its powers come from the atoms' kernels."""
    out = [torch.zeros(m.n, m.n, device=DEV, dtype=torch.float32) for _ in range(2)]
    done = {}
    for s in range(int(m.slots.max()) + 1):
        at = np.nonzero(m.slots == s)[0]
        key = tuple(m.aoat[at][:64]) + (len(at),)
        if key not in done:
            a = m.at[torch.from_numpy(at).to(DEV)]
            w, v = torch.linalg.eigh(torch.exp(-0.5 * m.dist[a][:, a].square()))
            powers = [(v * w.clamp_min(1e-12) ** y) @ v.T for y in (1.0 - x, x)]
            done[key] = [0.5 * (p + p.T) for p in powers]
        idx = torch.from_numpy(at).to(DEV)
        for o, p in zip(out, done[key]):
            o[idx[:, None], idx[None, :]] = p.float()
    return out


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "ctx": context()}
    if kind == "batch":
        state["systems"] = [(m.n, m.nel, m.H.cpu().numpy(), m.S.cpu().numpy()) for m in lattices(case, seed)]
        return state
    m = molecule(case, seed, matrices=kind not in ("mlpop2", "xc"))
    state.update(n=m.n, nat=m.nat, nel=m.nel, xyz=m.xyz, aoat=m.aoat)
    if kind == "sm":
        part = clustering(m, case["size"], seed) if case["columns"] == 4 else None
        out = torch.empty(m.H.shape, dtype=torch.float64, pin_memory=True).numpy()
        state.update(H=pinned(m.H), S=pinned(m.S), out=out, partition=part, opts=Options(filter=case["filter"]))
    elif kind == "tc":
        state["opts"] = Options(filter=case["filter"], precision=PREC_MIXED if case["mixed"] else PREC_FP64)
        if case["device"]:
            state.update(H=m.H, S=m.S, P=torch.empty_like(m.H))
        else:
            out = torch.empty(m.H.shape, dtype=torch.float64, pin_memory=True).numpy()
            state.update(H=pinned(m.H), S=pinned(m.S), out=out)
    elif kind in ("solve2", "purify"):
        state.update(H=m.H.cpu().numpy(), S=m.S.cpu().numpy(), opts=Options(filter=case["filter"]))
        if kind == "purify":
            # McWeeny works with S^-1, the sign solvers with S^-1/2
            state["settings"] = PurificationSettings(type=case["type"], metric_type=1 if case["type"] == 1 else 2,
                                                     cycles=100, prlvl=0, nel=m.nel)
    elif kind == "mlpop2":
        s34, s14 = overlap_powers(m, 1.0 / 3.0)
        state.update(P=density_like(m), s34=s34, s14=s14, shells=synth.shell2ao(m.aoat))
    else:
        rng = np.random.default_rng(seed)
        rab = (m.dist * BOHR)[tuple(torch.tril_indices(m.nat, m.nat, device=DEV))]
        H = density_like(m)
        state.update(P=density_like(m), H=H, rab=rab.cpu().numpy(), rad=rng.uniform(2.0, 4.0, m.nat),
                     hao=rng.uniform(-0.5, 0.5, m.n), xdiag=rng.uniform(0.5, 1.5, m.n))
    return state


# ---- the calls -----------------------------------------------------------------------------------------------

def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "batch":
        return ctx.eig_density_batch(state["systems"])[0]
    n = state["n"]
    if kind == "sm":
        P, st = ctx.sm_stupid_simple(n, state["nel"], state["H"], state["S"], state["nat"], state["xyz"], state["aoat"],
                                     case["columns"], 2, state["partition"], state["opts"], out=state["out"])
        return {"P": P, "mu": st.mu, "nel": st.nel}
    if kind == "tc" and case["device"]:
        ctx.tc_purify_device(n, state["nel"], state["H"].data_ptr(), state["S"].data_ptr(), state["P"].data_ptr(),
                             state["opts"])
        return {"P": state["P"]}
    if kind == "tc":
        return {"P": ctx.tc_purify(n, state["nel"], state["H"], state["S"], state["opts"], out=state["out"])[0]}
    if kind == "solve2":
        P, e, focc, _ = ctx.solve2(1, n, state["nel"], 0, state["H"], state["S"], state["opts"])
        return {"P": P, "e": e, "focc": focc}
    if kind == "purify":
        P, st = ctx.purification(state["settings"], n, state["H"], state["S"], state["opts"])
        return {"P": P, "mu": st.mu}
    if kind == "mlpop2":
        q, qsh, _ = ctx.mlpop2_device(state["nat"], n, state["P"].data_ptr(), state["s34"].data_ptr(),
                                      state["s14"].data_ptr(), state["aoat"], state["shells"])
        return {"q": q, "qsh": qsh}
    ctx.xc_damping_device(state["nat"], n, state["aoat"], state["rab"], state["rad"], state["hao"], state["xdiag"],
                          state["P"].data_ptr(), state["H"].data_ptr())
    return {"H": state["H"]}


# ---- what a call cannot do without -----------------------------------------------------------------------------

def orders(case):
    """Number of basis functions of the case's system."""
    if case["mol"] == "alkane":
        return 13 * case["size"] + 5 * (2 * case["size"] + 2)
    return 23 * case["size"]


def submatrices(case, n):
    """(count, order, owned columns) of a typical submatrix: the orders follow from how far the filter lets an atom
    reach, and level off at that neighbourhood's size."""
    if case["columns"] == 3:
        return 1, n, n
    if case["columns"] == 4:
        k = max(1, case["size"] // MOLECULES_PER_CLUSTER)
        return k, min(n, 1900), n // k
    reach = 250 if case["mol"] == "alkane" else 700
    count = n if case["columns"] == 1 else (3 * case["size"] + 2 if case["mol"] == "alkane" else 3 * case["size"])
    return count, min(0.75 * n, reach), n / count


def solve_flops(n, nvec):
    """Cholesky, the symmetric reduction, tridiagonalisation and nvec back-transformed vectors of one pencil."""
    return n ** 3 / 3 + n ** 3 + 4 * n ** 3 / 3 + 4.0 * n * n * nvec


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = np.linspace(20, case["atoms"], case["size"]) * 23 / 3
        return {"bytes": float((sizes * sizes / 2).sum() * 24), "flops": float(sum(solve_flops(n, 0.17 * n)
                                                                                  + 0.17 * n ** 3 for n in sizes))}
    n = orders(case)
    packed = 8.0 * n * (n + 1) / 2
    occupied = 0.174 * n
    if kind == "sm":
        count, m, own = submatrices(case, n)
        return {"bytes": 3 * packed, "flops": count * (solve_flops(m, own) + 2.0 * m * m * own)}
    if kind == "solve2":
        return {"bytes": 3 * packed, "flops": solve_flops(n, occupied) + n * n * occupied}
    if kind == "purify":
        return {"bytes": 3 * packed, "flops": solve_flops(n, n) + 2.0 * n ** 3}
    if kind == "tc":       # orthogonalisation, about 30 squares of a symmetric matrix, back-transform
        return {"bytes": 3 * packed, "flops": 34.0 * n ** 3}
    if kind == "mlpop2":
        return {"bytes": packed + 8.0 * n * n, "flops": 2.0 * n ** 3}
    return {"bytes": 3 * packed, "flops": 3.0 * packed / 8}


# ---- the same results from plain torch in 64 bits ---------------------------------------------------------------

def full(packed, n, cut=0.0):
    if cut > 0.0:
        packed = torch.where(packed.abs() < cut, 0.0, packed)
    c, r = packed_index(n)
    a = torch.zeros(n, n, device=DEV, dtype=torch.float64)
    a[c, r] = packed
    a[r, c] = packed
    return a


def pack(a):
    c, r = packed_index(a.shape[0])
    return a[c, r]


def pencil(H, S):
    """Eigenvalues and S-orthonormal eigenvectors of H u = e S u."""
    L = torch.linalg.cholesky(S)
    A = torch.linalg.solve_triangular(L, torch.linalg.solve_triangular(L, H, upper=False).T, upper=False)
    e, v = torch.linalg.eigh(0.5 * (A + A.T))
    return e, torch.linalg.solve_triangular(L.T, v, upper=True)


def projector(H, S, nel):
    """2 sum over the nel/2 lowest eigenvectors; large systems by trace-correcting squares in 64 bits."""
    n = H.shape[0]
    if n <= 2600:
        u = pencil(H, S)[1][:, : nel // 2]
        return 2.0 * (u @ u.T)
    L = torch.linalg.cholesky(S)
    A = torch.linalg.solve_triangular(L, torch.linalg.solve_triangular(L, H, upper=False).T, upper=False)
    radius = A.abs().sum(1) - A.diagonal().abs()
    lo, hi = float((A.diagonal() - radius).min()), float((A.diagonal() + radius).max())
    X = A.mul_(-1.0 / (hi - lo))
    X.diagonal().add_(hi / (hi - lo))
    left, last = math.inf, math.inf
    for step in range(80):
        X2 = X @ X
        X2 = 0.5 * (X2 + X2.T)
        t, t2 = float(X.trace()), float(X2.trace())
        X = X2 if abs(t2 - nel / 2) < abs(2 * t - t2 - nel / 2) else 2 * X - X2
        left, last = abs(t - t2), left
        if step > 20 and left < 1e-6 and left >= last:
            break
    X = torch.linalg.solve_triangular(L.T, X, upper=True)
    X = torch.linalg.solve_triangular(L.T, X.T, upper=True)
    return X + X.T


def submatrix_density(case, seed, m, H, S):
    """The submatrix method: strictly positive couplings pick each submatrix's rows, occupations 2 / 1 / 0 by a
    bisected mu, and every submatrix keeps the columns it owns."""
    n = m.n
    if case["columns"] == 1:
        label = np.arange(n)
    elif case["columns"] == 2:
        label = m.aoat - 1
    elif case["columns"] == 3:
        label = np.zeros(n, dtype=np.int64)
    else:
        label = clustering(m, case["size"], seed)[m.aoat - 1] - 1
    on = (H > 0.0) | (S > 0.0)
    on.fill_diagonal_(True)
    kept = []
    for k in range(int(label.max()) + 1):
        own = torch.from_numpy(np.nonzero(label == k)[0]).to(DEV)
        rows = torch.nonzero(on[:, own].any(1))[:, 0]
        mine = torch.searchsorted(rows, own)
        s = S[rows][:, rows]
        e, u = pencil(H[rows][:, rows], s)
        weight = ((s[mine] @ u) * u[mine]).sum(0)
        kept.append((own, rows, mine, e, u, weight))
    e, weight = torch.cat([k[3] for k in kept]), torch.cat([k[5] for k in kept])
    lo, hi, last = -10.0, 10.0, False
    for _ in range(100):
        mu = 0.5 * (lo + hi)
        nel = float((weight * (2.0 * (e < mu) + 1.0 * (e == mu))).sum())
        if last:
            break
        last = abs(lo - hi) < float(np.float32(1e-3)) or abs(nel - m.nel) < float(np.float32(1e-5))
        if not last:
            lo, hi = (lo, mu) if nel > m.nel else (mu, hi)
    P = torch.zeros(n, n, device=DEV, dtype=torch.float64)
    for own, rows, mine, ek, u, _ in kept:
        occ = 2.0 * (ek < mu) + 1.0 * (ek == mu)
        P[own[:, None], rows[None, :]] = (u[mine] * occ) @ u.T      # row c of P holds column c
    return {"P": pack(P), "mu": mu, "nel": nel}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sm" and case["columns"] == 1 and orders(case) > 2000:
        return None       # thousands of small pencils one after another take plain torch too long
    if kind == "batch":
        return [pack(projector(full(m.H, m.n), full(m.S, m.n), m.nel)) for m in lattices(case, seed)]
    if kind in ("mlpop2", "xc"):
        s = prepare(case, seed)
        n = s["n"]
        if kind == "mlpop2":
            d = ((s["s14"].double() @ full(s["P"], n)) * s["s34"].double().T).sum(1).cpu().numpy()
            q, qsh = np.zeros(s["nat"]), np.zeros((s["nat"], 10))
            np.add.at(q, s["aoat"] - 1, d)
            np.add.at(qsh, (s["aoat"] - 1, s["shells"] - 1), d)
            return {"q": q, "qsh": qsh}
        hao, xdiag, rad, rab = (torch.from_numpy(s[k]).to(DEV) for k in ("hao", "xdiag", "rad", "rab"))
        at = torch.from_numpy(s["aoat"] - 1).to(DEV)
        i, j = torch.tril_indices(s["nat"], s["nat"], device=DEV)
        r = rad[i] + rad[j]
        xab = 0.5 * (1.0 + torch.erf(-1.8 * ((rab - r) / r)))
        c, r = packed_index(n)
        pair = at[c] * (at[c] + 1) // 2 + at[r]
        factor = torch.where(c == r, 2.0 * xdiag[c] * hao[c], hao[c] + hao[r])
        return {"H": s["H"] + s["P"] * factor * xab[pair]}
    m = molecule(case, seed)
    H, S = full(m.H, m.n, case["filter"]), full(m.S, m.n, case["filter"])
    if kind == "sm":
        return submatrix_density(case, seed, m, H, S)
    if kind == "solve2":
        e, u = pencil(H, S)
        focc = torch.zeros(m.n, device=DEV, dtype=torch.float64)
        focc[: m.nel // 2] = 2.0      # the gap is hundreds of kT
        return {"P": pack(2.0 * (u[:, : m.nel // 2] @ u[:, : m.nel // 2].T)), "e": e, "focc": focc}
    P = pack(projector(H, S, m.nel))
    return {"P": P, "mu": None} if kind == "purify" else {"P": P}
