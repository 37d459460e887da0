// Divide and conquer for the tridiagonal eigenproblems of a batch,
// T = Z diag(w) Z^T, in stages over every problem of the batch at once (included by
// sm_eig.cu inside its namespace).
//
// Cuppen's split T = diag(T1, T2) + |beta| u u^T, u = e_last + sign(beta) e_first;
// Gu and Eisenstat's recomputed z for orthogonal eigenvectors.  Leaves of at most
// kDcLeaf rows are solved by a warp with the implicit QL iteration (every lane runs
// the same scalar iteration and applies each rotation to its own row of the leaf's
// Z).  A merge of the blocks [lo, mid) and [mid, hi):
//   deflate   z = [last row of Z1, sign(beta) first row of Z2] / sqrt 2, rho =
//             2|beta|; merged order of the two sorted blocks; rho |z_j| <= tol ->
//             eigenpair (d_j, q_j); two close d's -> a Givens rotation zeroes one z
//             entry (LAPACK's dlaed2 rules, tol = 8 eps max(|d|, rho))
//   permute   Q = the block columns in the merged order, rotated
//   secular   roots lambda_i = d_org + tau in (d_i, d_i+1), each step modelling the
//             left and right sums by one pole each
//   zhat      zhat_j^2 = (lambda_j - d_j) prod_{i != j} (lambda_i - d_j) /
//             (d_i - d_j) / rho, and the ascending position of every eigenvalue
//   vectors   v_i = (zhat_j / (d_j - lambda_i))_j normalised, columns of V (k x k)
//   product   Z_new = Q [V | deflated columns] in two halves (rows of block 1 against
//             the columns that touch it, rows of block 2 likewise)
// Each of these is one launch over all merges of a level (levels counted from the
// leaves, so problems of different orders share launches), split over as many CTAs
// as the level's elements or tiles give: one CTA per problem spent its time on CTA
// barriers between short phases and on one-thread-per-root loops.  The top merge's
// product is not formed where only rows of Z times given vectors are wanted.
constexpr int kDcLeaf = 32;
constexpr int kDcChunk = 32;      // roots (or columns) of one CTA of the per-element stages
constexpr int kDcRows = 64;       // rows of Q of one CTA of the permute stage

struct DcMerge {
    int pi, lo, mid, hi;
};
// Per-element arrays, each of the batch's total order; a merge's part starts at its
// problem's voff + lo.  cnt: 8 ints per merge.
struct DcArr {
    double *D, *Ds, *zs, *dk, *zk, *tau, *zh, *val;
    double2* rcs;
    int *perm, *org, *sec, *dl, *rank, *cls, *ktop, *kbot, *qtop, *qbot;
    int2* rpair;
    int* cnt;
};
constexpr size_t kDcBytes = 8 * sizeof(double) + sizeof(double2) + 10 * sizeof(int) + sizeof(int2);
enum { DC_K = 0, DC_ND = 1, DC_NROT = 2, DC_NTOP = 3, DC_NBOT = 4 };

inline DcArr dc_arrays(void* base, int64_t n, int* cnt) {   // n: a multiple of 2
    DcArr s;
    double* d = static_cast<double*>(base);
    s.D = d;
    s.Ds = d + n;
    s.zs = d + 2 * n;
    s.dk = d + 3 * n;
    s.zk = d + 4 * n;
    s.tau = d + 5 * n;
    s.zh = d + 6 * n;
    s.val = d + 7 * n;
    s.rcs = reinterpret_cast<double2*>(d + 8 * n);
    s.rpair = reinterpret_cast<int2*>(s.rcs + n);
    int* ip = reinterpret_cast<int*>(s.rpair + n);
    s.perm = ip;
    s.org = ip + n;
    s.sec = ip + 2 * n;
    s.dl = ip + 3 * n;
    s.rank = ip + 4 * n;
    s.cls = ip + 5 * n;
    s.ktop = ip + 6 * n;
    s.kbot = ip + 7 * n;
    s.qtop = ip + 8 * n;
    s.qbot = ip + 9 * n;
    s.cnt = cnt;
    return s;
}

// Levels of a problem of order m (0: one leaf) and the start of part q of 2^lev.
__host__ __device__ inline int dc_levels(int m) {
    int L = 0;
    while (((m + (1 << L) - 1) >> L) > kDcLeaf) ++L;
    return L;
}
__host__ __device__ inline int dc_start(int m, int q, int lev) { return (int)(((int64_t)q * m) >> lev); }

// Leaf: the implicit QL iteration on d[0..s), e[0..s-1) with Z = I accumulated, in the steps
// of EISPACK's imtql2 (Martin and Wilkinson, Numer. Math. 12, 377 (1968); Dubrulle, Numer.
// Math. 15, 450 (1970)): the shift from the leading 2 x 2 block, the chase of the bulge by
// plane rotations and the restart where a rotation vanishes.  Every lane runs the same scalar iteration on its own copies of d and e and rotates
// its own row z of Z (lane r holds row r), so no lane reads another's data.
__device__ bool dc_leaf(int s, double* d, double* e, double* z, int lane) {
    const double eps = 2.220446049250313e-16;
    for (int c = 0; c < kDcLeaf; ++c) z[c] = (c == lane) ? 1.0 : 0.0;
    for (int l = 0; l < s; ++l) {
        int iter = 0;
        for (;;) {
            int mm = l;
            for (; mm < s - 1; ++mm)
                if (fabs(e[mm]) <= eps * (fabs(d[mm]) + fabs(d[mm + 1]))) break;
            if (mm == l) break;
            if (++iter > kQlMaxIter) return false;
            double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
            double r = hypot(g, 1.0);
            g = d[mm] - d[l] + e[l] / (g + copysign(r, g));
            double sn = 1.0, c = 1.0, pp = 0.0;
            bool underflow = false;
            for (int i = mm - 1; i >= l; --i) {
                const double f = sn * e[i], b = c * e[i];
                // the rotation of (f, g): one rsqrt where the squares neither
                // overflow nor lose bits, the chain's longest step
                const double h = fma(f, f, g * g);
                if (h > 1e-270 && h < 1e270) {
                    const double ri = rsqrt(h);
                    e[i + 1] = h * ri;
                    sn = f * ri;
                    c = g * ri;
                } else {
                    r = hypot(f, g);
                    e[i + 1] = r;
                    if (r == 0.0) {
                        d[i + 1] -= pp;
                        e[mm] = 0.0;
                        underflow = true;
                        break;
                    }
                    sn = f / r;
                    c = g / r;
                }
                g = d[i + 1] - pp;
                r = (d[i] - g) * sn + 2.0 * c * b;
                pp = sn * r;
                d[i + 1] = g + pp;
                g = c * r - b;
                const double zi = z[i], zi1 = z[i + 1];
                z[i + 1] = sn * zi + c * zi1;
                z[i] = c * zi - sn * zi1;
            }
            if (underflow) continue;
            d[l] -= pp;
            e[l] = g;
            e[mm] = 0.0;
        }
    }
    return true;
}

// Leaves: a warp each (leaves[]: problem, part of 2^L).
constexpr int kLeafWarps = 2;
__global__ void __launch_bounds__(32 * kLeafWarps) k_dc_leaves(const EigProb* __restrict__ probs,
                                                               const int2* __restrict__ leaves, int nleaves,
                                                               const double* __restrict__ Da,
                                                               const double* __restrict__ Ea, double* __restrict__ Za,
                                                               DcArr S, int* __restrict__ status) {
    const int lane = threadIdx.x & 31, id = blockIdx.x * kLeafWarps + (threadIdx.x >> 5);
    if (id >= nleaves) return;
    const int2 lf = leaves[id];
    if (status[lf.x] != kStOk) return;
    const EigProb p = probs[lf.x];
    const int m = p.m, L = dc_levels(m);
    const int lo = dc_start(m, lf.y, L), hi = dc_start(m, lf.y + 1, L), s = hi - lo;
    const double* eo = Ea + p.voff;
    double* Z = Za + p.aoff;
    double dl[kDcLeaf], el[kDcLeaf], zl[kDcLeaf];
    for (int i = 0; i < kDcLeaf; ++i) {
        double d = 0.0;
        if (i < s) {
            // the rank-one terms of the splits at this leaf's ends
            d = Da[p.voff + lo + i];
            if (i == 0 && lo > 0) d -= fabs(eo[lo - 1]);
            if (i == s - 1 && hi < m) d -= fabs(eo[hi - 1]);
        }
        dl[i] = d;
        el[i] = (i < s - 1) ? eo[lo + i] : 0.0;
    }
    if (!dc_leaf(s, dl, el, zl, lane)) {
        if (lane == 0) status[lf.x] = kStNoConv;
        return;
    }
    // eigenvalues ascending (ties by index) and the columns in that order
    int rk = 0;
    if (lane < s) {
        const double x = dl[lane];
        for (int c = 0; c < s; ++c) rk += (dl[c] < x || (dl[c] == x && c < lane)) ? 1 : 0;
    }
    for (int c = 0; c < s; ++c) {
        const int rc = __shfl_sync(0xffffffffu, rk, c);
        if (lane < s) Z[(int64_t)(lo + lane) + (int64_t)(lo + rc) * m] = zl[c];
    }
    if (lane < s) {
        S.D[p.voff + lo + rk] = dl[lane];
        if (L == 0) {   // no merge follows: the leaf's Z stands for the top merge's Q
            S.val[p.voff + rk] = dl[lane];
            S.sec[p.voff + lane] = lane;
        }
    }
}

// Ordered compaction over a CTA of NT threads: calls put(position, index) for
// every index of [0, n) with pred(index), positions from 0; returns their number.
// ws: NT / 32 + 1 shared ints.
template <int NT, class Pred, class Put>
__device__ int cta_compact(int n, int* ws, Pred pred, Put put) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int base = 0;
    for (int c0 = 0; c0 < n; c0 += NT) {
        const int i = c0 + tid;
        const bool on = i < n && pred(i);
        const unsigned b = __ballot_sync(0xffffffffu, on);
        if (lane == 0) ws[warp] = __popc(b);
        __syncthreads();
        int before = base, tot = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) {
            if (w < warp) before += ws[w];
            tot += ws[w];
        }
        if (on) put(before + __popc(b & ((1u << lane) - 1u)), i);
        base += tot;
        __syncthreads();
    }
    return base;
}

constexpr int kDeflT = 256;
__global__ void __launch_bounds__(kDeflT) k_dc_deflate(const EigProb* __restrict__ probs,
                                                       const DcMerge* __restrict__ merges, int m0,
                                                       const double* __restrict__ Ea, const double* __restrict__ Za,
                                                       DcArr S, const int* __restrict__ status) {
    __shared__ int ws[kDeflT / 32 + 1], sc[4];
    const int mi = m0 + blockIdx.x;
    const DcMerge mg = merges[mi];
    if (status[mg.pi] != kStOk) return;
    const EigProb p = probs[mg.pi];
    const int m = p.m, lo = mg.lo, mid = mg.mid, n1 = mid - lo, n2 = mg.hi - mid, n = n1 + n2, tid = threadIdx.x;
    const int64_t o = p.voff + lo;
    const double* Z = Za + p.aoff;
    const double beta = Ea[p.voff + mid - 1], rho = 2.0 * fabs(beta), sgn = beta >= 0.0 ? 1.0 : -1.0;
    const double rs2 = 0.70710678118654752440, eps = 2.220446049250313e-16;
    double *Ds = S.Ds + o, *zs = S.zs + o;
    int *perm = S.perm + o, *cls = S.cls + o, *sec = S.sec + o, *dl = S.dl + o, *list = S.ktop + o;
    const double *D1 = S.D + o, *D2 = D1 + n1;
    // merged order, sorted d and z, column classes (1: block 1, 2: block 2)
    for (int j = tid; j < n; j += kDeflT) {
        int r, a = 0;
        double x, z;
        if (j < n1) {
            x = D1[j];
            z = Z[(int64_t)(mid - 1) + (int64_t)(lo + j) * m] * rs2;
            int b = n2;
            while (a < b) {
                const int c = (a + b) >> 1;
                if (D2[c] < x) a = c + 1;
                else b = c;
            }
            r = j + a;
        } else {
            x = D2[j - n1];
            z = sgn * Z[(int64_t)mid + (int64_t)(lo + j) * m] * rs2;
            int b = n1;
            while (a < b) {
                const int c = (a + b) >> 1;
                if (D1[c] <= x) a = c + 1;
                else b = c;
            }
            r = (j - n1) + a;
        }
        perm[r] = j;
        Ds[r] = x;
        zs[r] = z;
        cls[r] = j < n1 ? 1 : 2;
    }
    __syncthreads();
    const double tol = 8.0 * eps * fmax(fmax(fabs(Ds[0]), fabs(Ds[n - 1])), rho);
    // small z: deflated at once
    const int nz = cta_compact<kDeflT>(n, ws, [&](int r) { return !(rho * fabs(zs[r]) <= tol); },
                                       [&](int t, int r) { list[t] = r; });
    const int nd0 = cta_compact<kDeflT>(n, ws, [&](int r) { return rho * fabs(zs[r]) <= tol; },
                                        [&](int t, int r) { dl[t] = r; });
    // close pairs among the rest: rare, so the walk that rotates them runs only if
    // some pair of neighbours is close
    int close = 0;
    for (int t = 1 + tid; t < nz; t += kDeflT) {
        const double sn = zs[list[t - 1]], c = zs[list[t]], dd = Ds[list[t]] - Ds[list[t - 1]];
        const double h = hypot(c, sn);
        close |= fabs(dd * (c / h) * (sn / h)) <= tol;
    }
    int k = nz, nd = nd0, nrot = 0;
    if (__syncthreads_or(close)) {
        if (tid == 0) {
            k = 0;
            int pj = nz > 0 ? list[0] : -1;
            for (int t = 1; t < nz; ++t) {
                const int r = list[t];
                double sn = zs[pj], c = zs[r];
                const double h = hypot(c, sn);
                const double dd = Ds[r] - Ds[pj];
                c /= h;
                sn = -sn / h;
                if (fabs(dd * c * sn) <= tol) {
                    zs[r] = h;
                    zs[pj] = 0.0;
                    S.rpair[o + nrot] = make_int2(pj, r);
                    S.rcs[o + nrot] = make_double2(c, sn);
                    ++nrot;
                    const double t2 = Ds[pj] * c * c + Ds[r] * sn * sn;
                    Ds[r] = Ds[pj] * sn * sn + Ds[r] * c * c;
                    Ds[pj] = t2;
                    cls[r] |= cls[pj];
                    cls[pj] = cls[r];
                    dl[nd++] = pj;
                } else {
                    sec[k++] = pj;
                }
                pj = r;
            }
            if (pj >= 0) sec[k++] = pj;
            sc[0] = k;
            sc[1] = nd;
            sc[2] = nrot;
        }
        __syncthreads();
        k = sc[0];
        nd = sc[1];
        nrot = sc[2];
    } else {
        for (int t = tid; t < nz; t += kDeflT) sec[t] = list[t];
        __syncthreads();
    }
    // the order [secular | deflated] of the merge's columns
    for (int t = tid; t < nd; t += kDeflT) {
        sec[k + t] = dl[t];
        S.val[o + k + t] = Ds[dl[t]];
    }
    for (int t = tid; t < k; t += kDeflT) {
        S.dk[o + t] = Ds[sec[t]];
        S.zk[o + t] = zs[sec[t]];
    }
    __syncthreads();   // list (= ktop) is free from here
    const int nt = cta_compact<kDeflT>(k, ws, [&](int t) { return (cls[sec[t]] & 1) != 0; },
                                       [&](int q, int t) {
                                           S.ktop[o + q] = t;
                                           S.qtop[o + q] = sec[t];
                                       });
    const int nb = cta_compact<kDeflT>(k, ws, [&](int t) { return (cls[sec[t]] & 2) != 0; },
                                       [&](int q, int t) {
                                           S.kbot[o + q] = t;
                                           S.qbot[o + q] = sec[t];
                                       });
    if (tid == 0) {
        int* c = S.cnt + 8 * (int64_t)mi;
        c[DC_K] = k;
        c[DC_ND] = nd;
        c[DC_NROT] = nrot;
        c[DC_NTOP] = nt;
        c[DC_NBOT] = nb;
    }
}

// Q: the block columns in the merged order (zero outside their block), then the
// deflation's rotations, kDcRows rows per CTA.
__global__ void __launch_bounds__(256) k_dc_permute(const EigProb* __restrict__ probs,
                                                    const DcMerge* __restrict__ merges,
                                                    const int2* __restrict__ tasks, const double* __restrict__ Za,
                                                    double* __restrict__ Qa, DcArr S,
                                                    const int* __restrict__ status) {
    const int2 tk = tasks[blockIdx.x];
    const DcMerge mg = merges[tk.x];
    if (status[mg.pi] != kStOk) return;
    const EigProb p = probs[mg.pi];
    const int m = p.m, lo = mg.lo, n1 = mg.mid - lo, n = mg.hi - lo;
    const int64_t o = p.voff + lo;
    const double* Z = Za + p.aoff;
    double* Q = Qa + p.aoff + (int64_t)lo * m;
    const int i = tk.y * kDcRows + (threadIdx.x & (kDcRows - 1)), half = i < n1 ? 0 : 1;
    if (i < n)
#pragma unroll 4
        for (int r = threadIdx.x / kDcRows; r < n; r += 256 / kDcRows) {
            const int j = min(max(S.perm[o + r], 0), n - 1);   // in range whatever the eigenvalues are
            Q[i + (int64_t)r * n] = (j < n1) == (half == 0) ? Z[(int64_t)(lo + i) + (int64_t)(lo + j) * m] : 0.0;
        }
    const int nrot = S.cnt[8 * (int64_t)tk.x + DC_NROT];
    if (nrot == 0) return;
    __syncthreads();
    if (threadIdx.x < kDcRows && i < n)
        for (int q = 0; q < nrot; ++q) {
            const int2 pr = S.rpair[o + q];
            const double2 cs = S.rcs[o + q];
            const double a = Q[i + (int64_t)pr.x * n], b = Q[i + (int64_t)pr.y * n];
            Q[i + (int64_t)pr.x * n] = cs.x * a + cs.y * b;
            Q[i + (int64_t)pr.y * n] = -cs.y * a + cs.x * b;
        }
}

__device__ __forceinline__ double sum8(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

// Root i of 1 + rho sum_t z_t^2 / (dk_t - lambda) = 0 (dk ascending, k roots), eight
// lanes per root over the terms: returns tau with lambda = dk[*org] + tau.  Every
// lane of the warp calls it (active: the lane's root exists).
__device__ double dc_secular(int k, const double* __restrict__ dk, const double* __restrict__ zk, double rho, int i,
                             bool active, int* org_out) {
    const double eps = 2.220446049250313e-16;
    const int l8 = threadIdx.x & 7;
    if (!active) i = 0;
    const bool last = i == k - 1;
    const double di = dk[i], mid = last ? 0.0 : 0.5 * (dk[i + 1] - di);
    double f0 = 0.0, z2 = 0.0;
    for (int t = l8; t < k; t += 8) {
        const double z = zk[t];
        z2 = fma(z, z, z2);
        if (!last) f0 += rho * z * z / ((dk[t] - di) - mid);
    }
    f0 = 1.0 + sum8(f0);
    z2 = sum8(z2);
    int org = i;
    double lo = 0.0, hi = rho * z2;
    if (!last) {
        hi = mid;
        if (!(f0 >= 0.0)) {
            org = i + 1;
            lo = -mid;
            hi = 0.0;
        }
    }
    const double dorg = dk[org];
    const double a = di - dorg;
    const double b = last ? 0.0 : dk[i + 1] - dorg;
    double tau = 0.5 * (lo + hi);
    bool done = !active;
    for (int it = 0; it < 100 && __any_sync(0xffffffffu, !done); ++it) {
        double psi = 0.0, phi = 0.0, dpsi = 0.0, dphi = 0.0;
        int t = l8;
        for (; t <= i; t += 8) {
            const double r = 1.0 / ((dk[t] - dorg) - tau), z = zk[t], q = rho * z * z * r;
            psi += q;
            dpsi = fma(q, r, dpsi);
        }
        for (; t < k; t += 8) {
            const double r = 1.0 / ((dk[t] - dorg) - tau), z = zk[t], q = rho * z * z * r;
            phi += q;
            dphi = fma(q, r, dphi);
        }
        psi = sum8(psi);
        phi = sum8(phi);
        dpsi = sum8(dpsi);
        dphi = sum8(dphi);
        if (done) continue;
        const double f = 1.0 + psi + phi;
        if (f > 0.0) hi = tau;
        else if (f < 0.0) lo = tau;
        if (f == 0.0 || fabs(f) <= 16.0 * eps * (1.0 + fabs(psi) + fabs(phi))) {
            done = true;
            continue;
        }
        const double B = dpsi * (a - tau) * (a - tau);
        const double A = psi - B / (a - tau);
        double nt;
        if (!last) {
            const double E = dphi * (b - tau) * (b - tau);
            const double Cc = phi - E / (b - tau);
            const double c0 = 1.0 + A + Cc;
            const double qb = -(c0 * (a + b) + B + E);
            const double qc = c0 * a * b + B * b + E * a;
            if (c0 == 0.0) {
                nt = -qc / qb;
            } else {
                const double disc = fmax(qb * qb - 4.0 * c0 * qc, 0.0);
                const double r1 = (-qb - copysign(sqrt(disc), qb)) / (2.0 * c0);
                const double r2 = (r1 != 0.0) ? qc / (c0 * r1) : r1;
                nt = (lo < r1 && r1 < hi) ? r1 : r2;
            }
        } else {
            const double c0 = 1.0 + A + phi;
            nt = (c0 != 0.0) ? a + B / c0 : 0.5 * (lo + hi);
        }
        if (!(lo < nt && nt < hi)) nt = 0.5 * (lo + hi);
        done = fabs(nt - tau) <= 2.0 * eps * fabs(nt);
        tau = nt;
    }
    *org_out = org;
    return tau;
}

// Per-element stages, kDcChunk elements per CTA of 256 threads (eight lanes each).
__global__ void __launch_bounds__(256) k_dc_secular(const EigProb* __restrict__ probs,
                                                    const DcMerge* __restrict__ merges,
                                                    const int2* __restrict__ tasks, const double* __restrict__ Ea,
                                                    DcArr S, const int* __restrict__ status) {
    const int2 tk = tasks[blockIdx.x];
    const DcMerge mg = merges[tk.x];
    if (status[mg.pi] != kStOk) return;
    const int k = S.cnt[8 * (int64_t)tk.x + DC_K];
    if (tk.y * kDcChunk >= k) return;
    const EigProb p = probs[mg.pi];
    const int64_t o = p.voff + mg.lo;
    const double rho = 2.0 * fabs(Ea[p.voff + mg.mid - 1]);
    const int i = tk.y * kDcChunk + (threadIdx.x >> 3);
    int org;
    const double tau = dc_secular(k, S.dk + o, S.zk + o, rho, i, i < k, &org);
    if (i < k && (threadIdx.x & 7) == 0) {
        S.tau[o + i] = tau;
        S.org[o + i] = org;
        S.val[o + i] = S.dk[o + org] + tau;
    }
}

__global__ void __launch_bounds__(256) k_dc_zhat(const EigProb* __restrict__ probs,
                                                 const DcMerge* __restrict__ merges, const int2* __restrict__ tasks,
                                                 const double* __restrict__ Ea, DcArr S,
                                                 const int* __restrict__ status) {
    const int2 tk = tasks[blockIdx.x];
    const DcMerge mg = merges[tk.x];
    if (status[mg.pi] != kStOk) return;
    const int k = S.cnt[8 * (int64_t)tk.x + DC_K], n = mg.hi - mg.lo;
    const EigProb p = probs[mg.pi];
    const int64_t o = p.voff + mg.lo;
    const double rho = 2.0 * fabs(Ea[p.voff + mg.mid - 1]);
    const int j = tk.y * kDcChunk + (threadIdx.x >> 3), l8 = threadIdx.x & 7;
    const double* dk = S.dk + o;
    double w = 1.0;
    if (j < k) {
        const double dj = dk[j];
        if (l8 == 0) w = (dk[S.org[o + j]] - dj) + S.tau[o + j];
        for (int i = l8; i < k; i += 8)
            if (i != j) w *= ((dk[S.org[o + i]] - dj) + S.tau[o + i]) / (dk[i] - dj);
    }
    w *= __shfl_xor_sync(0xffffffffu, w, 4);
    w *= __shfl_xor_sync(0xffffffffu, w, 2);
    w *= __shfl_xor_sync(0xffffffffu, w, 1);
    if (j < k && l8 == 0) S.zh[o + j] = copysign(sqrt(fmax(w / rho, 0.0)), S.zk[o + j]);
    // ascending position of eigenvalue j (ties by index)
    int r = 0;
    if (j < n) {
        const double x = S.val[o + j];
        for (int b = l8; b < n; b += 8) r += (S.val[o + b] < x || (S.val[o + b] == x && b < j)) ? 1 : 0;
    }
    r += __shfl_xor_sync(0xffffffffu, r, 4);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    if (j < n && l8 == 0) S.rank[o + j] = mg.lo + r;
}

// Columns of V (a warp each) and the new block's sorted eigenvalues.
__global__ void __launch_bounds__(256) k_dc_vectors(const EigProb* __restrict__ probs,
                                                    const DcMerge* __restrict__ merges,
                                                    const int2* __restrict__ tasks, double* __restrict__ Va, DcArr S,
                                                    const int* __restrict__ status) {
    const int2 tk = tasks[blockIdx.x];
    const DcMerge mg = merges[tk.x];
    if (status[mg.pi] != kStOk) return;
    const int k = S.cnt[8 * (int64_t)tk.x + DC_K], n = mg.hi - mg.lo;
    const EigProb p = probs[mg.pi];
    const int64_t o = p.voff + mg.lo;
    const int c0 = tk.y * kDcChunk, lane = threadIdx.x & 31;
    if (threadIdx.x < kDcChunk && c0 + threadIdx.x < n)
        S.D[p.voff + S.rank[o + c0 + threadIdx.x]] = S.val[o + c0 + threadIdx.x];
    double* V = Va + p.aoff + (int64_t)mg.lo * p.m;
    const double *dk = S.dk + o, *zh = S.zh + o;
    for (int i = c0 + (threadIdx.x >> 5); i < min(k, c0 + kDcChunk); i += 8) {
        const double dorg = dk[S.org[o + i]], ti = S.tau[o + i];
        double nrm = 0.0;
        for (int j = lane; j < k; j += 32) {
            const double v = zh[j] / ((dk[j] - dorg) - ti);
            nrm = fma(v, v, nrm);
        }
        const double sc = 1.0 / sqrt(warp_sum(nrm));
        for (int j = lane; j < k; j += 32) V[j + (int64_t)i * k] = sc * (zh[j] / ((dk[j] - dorg) - ti));
    }
}

// Z block = Q [V | deflated columns], one 64 x 64 tile per CTA (tasks: merge, row tile
// of the two halves << 16 | column tile).  nocc > 0 problems (densities) need the
// top merge's columns below nocc only.
constexpr size_t kTileSmem = sizeof(double) * 2 * kStageOp;
__global__ void __launch_bounds__(kT, 2) k_dc_product(const EigProb* __restrict__ probs,
                                                      const DcMerge* __restrict__ merges,
                                                      const int2* __restrict__ tasks, double* __restrict__ Za,
                                                      const double* __restrict__ Qa, const double* __restrict__ Va,
                                                      DcArr S, const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    double* sB = sA + kStageOp;
    const int2 tk = tasks[blockIdx.x];
    const DcMerge mg = merges[tk.x];
    if (status[mg.pi] != kStOk) return;
    const EigProb p = probs[mg.pi];
    const int m = p.m, lo = mg.lo, n1 = mg.mid - lo, n = mg.hi - lo;
    const int64_t o = p.voff + lo;
    const int* cnt = S.cnt + 8 * (int64_t)tk.x;
    const int k = cnt[DC_K];
    const int nt1 = (n1 + TS - 1) / TS;
    int rt = tk.y >> 16;
    const int c0 = (tk.y & 0xffff) * TS;
    const bool top = rt < nt1;
    const int r0 = top ? rt * TS : n1 + (rt - nt1) * TS, r1 = min(r0 + TS, top ? n1 : n);
    const int ncols = (p.mode == 2 && n == m) ? p.nocc : m;   // columns wanted (by position)
    double* Z = Za + p.aoff;
    const double* Q = Qa + p.aoff + (int64_t)lo * m;
    const double* V = Va + p.aoff + (int64_t)lo * m;
    const int* rank = S.rank + o;
    if (c0 < k && rank[c0] < ncols)
        tile_gemm<false>(Z, m, lo, rank, r0, c0, r1 - r0, min(TS, k - c0), Q, n, (top ? S.qtop : S.qbot) + o, V, k,
                         (top ? S.ktop : S.kbot) + o, top ? cnt[DC_NTOP] : cnt[DC_NBOT], sA, sB);
    // deflated columns: copies of Q's columns
    const int ca = max(c0, k), cb = min(c0 + TS, n);
    for (int q = threadIdx.x; q < (cb - ca) * (r1 - r0); q += kT) {
        const int i = r0 + q % (r1 - r0), c = ca + q / (r1 - r0);
        if (rank[c] < ncols) Z[(int64_t)(lo + i) + (int64_t)rank[c] * m] = Q[i + (int64_t)S.sec[o + c] * n];
    }
}
