// From the tridiagonal problems' eigenvectors to what leaves the solver, in stages
// over every problem of a batch (included by sm_eig.cu inside its namespace).
//   submatrix method: owned rows of S U and U, fe; later the owned columns of P
//   density:          U_occ = L^-T Q Z_occ and the upper tiles of U_occ U_occ^T
//   all vectors:      U = L^-T Q Z
// Tasks are (problem, 64-vector block) where a stage is a chain along the reflectors
// or the triangular solve, (problem, tile) where it is a product.

// T of one panel of reflectors per CTA (tasks: problem, panel).
constexpr size_t kWySmem = sizeof(double) * (2 * kStageOp + TS * TS + TS * kTld);
__global__ void __launch_bounds__(kT, 2) k_vec_panels(const EigProb* __restrict__ probs,
                                                      const int2* __restrict__ tasks, const double* __restrict__ Ca,
                                                      const double* __restrict__ Ta, double* __restrict__ Ka,
                                                      const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    double* sB = sA + kStageOp;
    double* G = sB + kStageOp;
    const int2 tk = tasks[blockIdx.x];
    if (status[tk.x] != kStOk) return;
    const EigProb p = probs[tk.x];
    build_T(Ca + p.coff, p.ldc, p.m, Ta + p.voff, Ka + p.koff + (int64_t)tk.y * TS * TS, tk.y, G, G + TS * TS, sA, sB);
}

constexpr size_t kChainSmem = sizeof(double) * (2 * kStageOp + TS * TS + TS * kY2ld);

// Rows of L (S U) and of L^-T (U) for the owned columns, times Q: block u of the 2 nown
// vectors (the rows of L first).  A chain of panels per task, so 64 vectors a task rather
// than a wider tile: the tasks of a batch fill the SMs twice (512-H2O clusters 36 -> 18 ms
// with the panels and solves of wy_apply and trsm_cols).
__global__ void __launch_bounds__(kT, 2) k_vec_rows(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                    const double* __restrict__ Ca, const double* __restrict__ La,
                                                    const double* __restrict__ Ia, const double* __restrict__ Ka, const int* __restrict__ own_cols,
                                                    const int* __restrict__ ipos, double* __restrict__ Ba,
                                                    const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    double* sB = sA + kStageOp;
    double* Y = sB + kStageOp;
    const int2 tk = tasks[blockIdx.x];
    if (status[tk.x] != kStOk) return;
    const EigProb p = probs[tk.x];
    const int m = p.m, no = p.nown, u0 = tk.y * TS, u1 = min(2 * no, u0 + TS);
    const double* L = La + p.aoff;
    double* R = Ba + p.boff;
    int top = m;   // L^-1 e_c is zero above row c
    for (int u = u0; u < u1; ++u) {
        const int ct = ipos[own_cols[p.o0 + (u < no ? u : u - no)]];
        if (u >= no) top = min(top, ct);
        double* x = R + (int64_t)u * m;
        for (int r = threadIdx.x; r < m; r += kT)
            x[r] = (u < no) ? ((r <= ct) ? L[ct + (int64_t)r * m] : 0.0) : ((r == ct) ? 1.0 : 0.0);
    }
    __syncthreads();
    const int s0 = max(u0, no);
    if (s0 < u1) trsm_cols(true, L, m, Ia + p.ioff, R + (int64_t)s0 * m, m, u1 - s0, sA, sB, top);
    wy_apply(Ca + p.coff, p.ldc, m, Ka + p.koff, R + (int64_t)u0 * m, u1 - u0, true, Y, Y + TS * TS, sA, sB);
}

// Z = Q V of the top merge is not formed: Q (m x m, at Qa; the leaf's Z of a problem
// without merges) and V (k x k), the columns in the order ord = [secular | deflated].
struct ZTop {
    const double *Q, *V;
    const int* ord;
    int k;
};
__device__ __forceinline__ ZTop z_top(const EigProb& p, const double* Za, const double* Qa, const double* Va,
                                      const DcArr& S) {
    ZTop z;
    z.Q = (p.topm < 0 ? Za : Qa) + p.aoff;
    z.V = Va + p.aoff;
    z.ord = S.sec + p.voff;
    z.k = p.topm < 0 ? 0 : S.cnt[8 * (int64_t)p.topm + DC_K];
    return z;
}

// T1 = Q^T R^T (m x 2 nown): tasks (problem, row tile << 16 | vector tile).
__global__ void __launch_bounds__(kT, 2) k_vec_rq(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                  const double* __restrict__ Za, const double* __restrict__ Qa,
                                                  const double* __restrict__ Va, DcArr S, double* __restrict__ Ba,
                                                  const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    const int2 tk = tasks[blockIdx.x];
    if (status[tk.x] != kStOk) return;
    const EigProb p = probs[tk.x];
    const ZTop z = z_top(p, Za, Qa, Va, S);
    const int m = p.m, r0 = (tk.y >> 16) * TS, c0 = (tk.y & 0xffff) * TS, nv = 2 * p.nown;
    tile_gemm<true>(Ba + p.boff + (int64_t)nv * m, m, 0, nullptr, r0, c0, min(TS, m - r0), min(TS, nv - c0), z.Q, m,
                    nullptr, Ba + p.boff, m, nullptr, m, sA, sA + kStageOp);
}

// G = [V | I]^T T1[ord] into R's place (rows of S U, then of U, times Z), same tasks.
__global__ void __launch_bounds__(kT, 2) k_vec_rv(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                  const double* __restrict__ Za, const double* __restrict__ Qa,
                                                  const double* __restrict__ Va, DcArr S, double* __restrict__ Ba,
                                                  const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    const int2 tk = tasks[blockIdx.x];
    if (status[tk.x] != kStOk) return;
    const EigProb p = probs[tk.x];
    const ZTop z = z_top(p, Za, Qa, Va, S);
    const int m = p.m, r0 = (tk.y >> 16) * TS, c0 = (tk.y & 0xffff) * TS, nv = 2 * p.nown;
    double* G = Ba + p.boff;
    const double* T1 = G + (int64_t)nv * m;
    if (r0 < z.k)
        tile_gemm<true>(G, m, 0, nullptr, r0, c0, min(TS, z.k - r0), min(TS, nv - c0), z.V, z.k, nullptr, T1, m, z.ord,
                        z.k, sA, sA + kStageOp);
    const int ra = max(r0, z.k), nr = min(r0 + TS, m) - ra, nc = min(TS, nv - c0);
    for (int q = threadIdx.x; q < nr * nc; q += kT) {
        const int r = ra + q % nr;
        const int64_t u = c0 + q / nr;
        G[r + u * m] = T1[z.ord[r] + u * m];
    }
}

// e and fe of 64 eigenvalues per CTA (tasks: problem, block).
__global__ void __launch_bounds__(256) k_vec_fe(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                const double* __restrict__ Ba, DcArr S, double* __restrict__ e_out,
                                                double* __restrict__ fe_out, const int* __restrict__ status) {
    __shared__ double part[4][TS];
    const int2 tk = tasks[blockIdx.x];
    if (status[tk.x] != kStOk) return;
    const EigProb p = probs[tk.x];
    const int m = p.m, no = p.nown, c = threadIdx.x & (TS - 1), g = threadIdx.x / TS, j = tk.y * TS + c;
    const double* G = Ba + p.boff;
    const double* G2 = G + (int64_t)no * m;
    double f = 0.0;
    if (j < m)
        for (int t = g; t < no; t += 4) f = fma(G[(int64_t)t * m + j], G2[(int64_t)t * m + j], f);
    part[g][c] = f;
    __syncthreads();
    if (g == 0 && j < m) {
        e_out[p.eoff + j] = S.val[p.voff + j];
        fe_out[p.eoff + j] = (part[0][c] + part[1][c]) + (part[2][c] + part[3][c]);
    }
}

// ---- owned columns of P at mu: W0 = occ o U[c, :]^T, T2 = [V | I] W0, W = Q[:, ord] T2,
// then L^-T Q_H W, scattered into the packed result (rows map(i) <= c of column c)
__global__ void __launch_bounds__(256) k_fin_occ(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                 DcArr S, double* __restrict__ Ba, double mu) {
    const int2 tk = tasks[blockIdx.x];
    const EigProb p = probs[tk.x];
    const int m = p.m, no = p.nown, c = threadIdx.x & (TS - 1), j = tk.y * TS + c;
    if (j >= m) return;
    const double* U = Ba + p.boff + (int64_t)no * m;
    double* W0 = Ba + p.boff + 2 * (int64_t)no * m;
    const double e = S.val[p.voff + j], occ = e < mu ? 2.0 : (e == mu ? 1.0 : 0.0);
    for (int t = threadIdx.x / TS; t < no; t += 4) W0[j + (int64_t)t * m] = occ * U[j + (int64_t)t * m];
}

__global__ void __launch_bounds__(kT, 2) k_fin_vw(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                  const double* __restrict__ Za, const double* __restrict__ Qa,
                                                  const double* __restrict__ Va, DcArr S, double* __restrict__ Ba) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    const int2 tk = tasks[blockIdx.x];
    const EigProb p = probs[tk.x];
    const ZTop z = z_top(p, Za, Qa, Va, S);
    const int m = p.m, no = p.nown, r0 = (tk.y >> 16) * TS, c0 = (tk.y & 0xffff) * TS;
    const double* W0 = Ba + p.boff + 2 * (int64_t)no * m;
    double* T2 = Ba + p.boff + 3 * (int64_t)no * m;
    if (r0 < z.k)
        tile_gemm<false>(T2, m, 0, nullptr, r0, c0, min(TS, z.k - r0), min(TS, no - c0), z.V, z.k, nullptr, W0, m,
                         nullptr, z.k, sA, sA + kStageOp);
    const int ra = max(r0, z.k), nr = min(r0 + TS, m) - ra, nc = min(TS, no - c0);
    for (int q = threadIdx.x; q < nr * nc; q += kT) {
        const int64_t at = ra + q % nr + (int64_t)(c0 + q / nr) * m;
        T2[at] = W0[at];
    }
}

__global__ void __launch_bounds__(kT, 2) k_fin_qw(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                  const double* __restrict__ Za, const double* __restrict__ Qa,
                                                  const double* __restrict__ Va, DcArr S, double* __restrict__ Ba) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    const int2 tk = tasks[blockIdx.x];
    const EigProb p = probs[tk.x];
    const ZTop z = z_top(p, Za, Qa, Va, S);
    const int m = p.m, no = p.nown, r0 = (tk.y >> 16) * TS, c0 = (tk.y & 0xffff) * TS;
    tile_gemm<false>(Ba + p.boff, m, 0, nullptr, r0, c0, min(TS, m - r0), min(TS, no - c0), z.Q, m, z.ord,
                     Ba + p.boff + 3 * (int64_t)no * m, m, nullptr, m, sA, sA + kStageOp);
}

__global__ void __launch_bounds__(kT, 2) k_fin_cols(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                    const double* __restrict__ Ca, const double* __restrict__ La,
                                                    const double* __restrict__ Ia, const double* __restrict__ Ka, const int* __restrict__ maps,
                                                    const int* __restrict__ own_cols, double* __restrict__ Ba,
                                                    double* __restrict__ Ppk, double* __restrict__ Pdense) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    double* sB = sA + kStageOp;
    double* Y = sB + kStageOp;
    const int2 tk = tasks[blockIdx.x];
    const EigProb p = probs[tk.x];
    const int m = p.m, t0 = tk.y * TS, nt = min(TS, p.nown - t0);
    double* W = Ba + p.boff + (int64_t)t0 * m;
    wy_apply(Ca + p.coff, p.ldc, m, Ka + p.koff, W, nt, false, Y, Y + TS * TS, sA, sB);
    __syncthreads();
    trsm_cols(false, La + p.aoff, m, Ia + p.ioff, W, m, nt, sA, sB);
    if (Pdense) {
        for (int64_t q = threadIdx.x; q < (int64_t)nt * m; q += kT) Pdense[p.poff + (int64_t)t0 * m + q] = W[q];
        return;
    }
    const int* mp = maps + p.moff;
    for (int t = 0; t < nt; ++t) {
        const int64_t cgl = own_cols[p.o0 + t0 + t];
        double* col = Ppk + cgl * (cgl + 1) / 2;
        for (int i = threadIdx.x; i < m; i += kT) {
            const int64_t gi = mp[i];
            if (gi <= cgl) col[gi] = W[i + (int64_t)t * m];
        }
    }
}

// ---- eigenvectors U = L^-T Q Z in place of Z, 64 columns per CTA (all of them, or the
// nocc lowest for a density): order 1495, 24 CTAs, 6.6 -> 3.6 ms, the chain of K chunks
__global__ void __launch_bounds__(kT, 2) k_vec_back(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                    const double* __restrict__ Ca, const double* __restrict__ La,
                                                    const double* __restrict__ Ia, const double* __restrict__ Ka, double* __restrict__ Za,
                                                    const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    double* sB = sA + kStageOp;
    double* Y = sB + kStageOp;
    const int2 tk = tasks[blockIdx.x];
    if (status[tk.x] != kStOk) return;
    const EigProb p = probs[tk.x];
    const int m = p.m, nv = p.mode == 2 ? p.nocc : m, t0 = tk.y * TS, nt = min(TS, nv - t0);
    double* U = Za + p.aoff + (int64_t)t0 * m;
    wy_apply(Ca + p.coff, p.ldc, m, Ka + p.koff, U, nt, false, Y, Y + TS * TS, sA, sB);
    __syncthreads();
    if (p.kind == 0) trsm_cols(false, La + p.aoff, m, Ia + p.ioff, U, m, nt, sA, sB);
}

// Upper tiles of U_occ U_occ^T (tasks: problem, row tile << 16 | column tile); the
// factor 2 is applied when packing.
__global__ void __launch_bounds__(kT, 2) k_vec_density(const EigProb* __restrict__ probs,
                                                       const int2* __restrict__ tasks, const double* __restrict__ Za,
                                                       double* __restrict__ Ba, const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    const int2 tk = tasks[blockIdx.x];
    if (status[tk.x] != kStOk) return;
    const EigProb p = probs[tk.x];
    const int m = p.m, r0 = (tk.y >> 16) * TS, c0 = (tk.y & 0xffff) * TS;
    const double* U = Za + p.aoff;
    tile_mma<false, true, MMA_SET, false>(Ba + p.boff, m, 0, nullptr, r0, c0, min(TS, m - r0), min(TS, m - c0), U, m,
                                          nullptr, U, m, nullptr, p.nocc, sA, sA + kStageOp);
}

// Ascending eigenvalues of every problem (the order of the vectors).
__global__ void __launch_bounds__(256) k_vec_values(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                    DcArr S, double* __restrict__ e_out,
                                                    const int* __restrict__ status) {
    const int2 tk = tasks[blockIdx.x];
    if (status[tk.x] != kStOk) return;
    const EigProb p = probs[tk.x];
    const int j = tk.y * TS + threadIdx.x;
    if (threadIdx.x < TS && j < p.m) e_out[p.eoff + j] = S.D[p.voff + j];
}
