// Householder tridiagonalisation of one symmetric matrix on one CTA (included by
// sm_eig.cu inside its namespace).
//
// LAPACK's blocked scheme (dsytrd / dlatrd, lower): inside a panel of nb columns
// the trailing block stays as it was at the panel's start, y = A v is one pass
// over its lower triangle, and the panel's earlier reflectors correct it through
// V and W; after the panel A -= V W^T + W V^T.  What bounds it: the pass over the
// lower triangle, m^3/6 doubles out of L2 in all, and four CTA barriers per column.
//   * V, W, the reflector and every partial sum live in shared memory; nb is the
//     widest of 16, 12, 8, 4 columns that fits the panel's order.
//   * A v: the lower triangle as 32 x 32 blocks, row by row, cut into one
//     contiguous run of blocks per warp (run lengths differ by one block at most).
//     A warp loads a block whole (32 coalesced loads in flight), keeps the row sums
//     in registers along a strip and turns its 32 columns' products into column
//     sums by a transposing butterfly: 31 exchanges per block, where one reduction
//     per column would take 160.  Row sums go to a slot per (warp of the strip,
//     row), column sums to a slot per block; both are added in a fixed order.
//   * The update after the panel runs on the FP64 tensor cores (DMMA) straight from
//     the shared V and W, a 32 x 32 block per warp and no barrier.
// NT = 512 threads (one CTA per SM) or 256 (two CTAs per SM, smaller orders).
// Measured: 96 problems of order 218-595, one CTA each: 9.5 ms (29 ms with the
// unblocked reduction that read and wrote the whole trailing square per column);
// 602 problems of order <= 253, two CTAs per SM: 4.9 ms.

__host__ __device__ constexpr int trd_ld(int s) { return ((s + 11) / 16) * 16 + 4; }   // >= s, = 4 mod 16
__host__ __device__ constexpr int trd_strips(int s) { return (s + 31) / 32; }
__host__ __device__ constexpr int trd_blocks(int s) { return trd_strips(s) * (trd_strips(s) + 1) / 2; }
// Row slots: the most warps that one strip's blocks are spread over.
__host__ __device__ constexpr int trd_row_slots(int s, int nw) {
    const int T = trd_strips(s), nblk = trd_blocks(s), run = nblk / nw > 1 ? nblk / nw : 1;
    return (T - 1 + run - 1) / run + 1;
}
// Doubles of shared memory of a panel of nb columns at trailing order s.
__host__ __device__ constexpr int trd_panel_doubles(int s, int nb, int nw) {
    return (2 * nb + trd_row_slots(s, nw) + 1) * trd_ld(s) + trd_blocks(s) * 32 + trd_strips(s) * 32;
}
constexpr int kTrdFixed = 128;   // doubles of the scalars in front of the panel's arrays
__host__ __device__ constexpr int trd_panel_width(int s, int nw, int cap) {
    return trd_panel_doubles(s, 16, nw) + kTrdFixed <= cap   ? 16
           : trd_panel_doubles(s, 12, nw) + kTrdFixed <= cap ? 12
           : trd_panel_doubles(s, 8, nw) + kTrdFixed <= cap  ? 8
           : trd_panel_doubles(s, 4, nw) + kTrdFixed <= cap  ? 4
                                                             : 0;
}
constexpr int kTrdCap512 = 232448 / 8;          // one CTA per SM
constexpr int kTrdCap256 = (232448 / 2 - 1024) / 8;   // two
constexpr int kTrdMax512 = 800;                 // orders one CTA takes (panels of 8 columns or more)
constexpr int kTrdMax256 = 288;                 // orders two CTAs per SM take (panels of 8 columns or more)
static_assert(trd_panel_width(kTrdMax512, 16, kTrdCap512) >= 8, "panel fits one CTA per SM");
static_assert(trd_panel_width(kTrdMax256, 8, kTrdCap256) >= 8, "panel fits two CTAs per SM");

// 32 column sums of a warp's 32 x 32 products: x[c] is this lane's product in
// column c; returns the sum of column `lane` over the lanes (fixed order).
__device__ __forceinline__ double warp_transpose_sum(double (&x)[32], int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const double send = up ? x[i] : x[i + o], keep = up ? x[i + o] : x[i];
            x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return x[0];
}

template <int NT>
__device__ void stage_trd(const EigProb& p, double* __restrict__ Ca, double* __restrict__ Da, double* __restrict__ Ea,
                          double* __restrict__ Ta, double* smem) {
    constexpr int NW = NT / 32, RPT = 2;   // rows per thread
    constexpr int cap = NT == 512 ? kTrdCap512 : kTrdCap256;
    const int m = p.m, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* A = Ca + p.aoff;
    double* d = Da + p.voff;
    double* e = Ea + p.voff;
    double* tau = Ta + p.voff;
    double* red = smem;           // 16: partial |x|^2 of the warps
    double* rva = smem + 16;      // 16: partial v^T A v
    double* vtv = smem + 32;      // 16: V^T v
    double* wtv = smem + 48;      // 16: W^T v
    double* arr = smem + kTrdFixed;
    for (int j0 = 0; j0 < m - 1;) {
        const int s = m - j0, ld = trd_ld(s), T = trd_strips(s), nblk = trd_blocks(s);
        const int width = trd_panel_width(s, NW, cap), nb = min(width, m - 1 - j0);
        const int nwe = min(NW, nblk);
        double* V = arr;                       // V[q ld + r], r relative to j0
        double* W = V + width * ld;
        double* rowp = W + width * ld;         // [slot][r]
        double* yl = rowp + trd_row_slots(s, NW) * ld;
        double* colp = yl + ld;                // [block][32]
        double* vb = colp + nblk * 32;         // reflector, zero outside its rows
        double* Aj = A + j0 + (int64_t)j0 * m; // element (r, c) of the trailing block at Aj[r + c m]
        // this thread's rows and the slots of their row sums
        int row[RPT], strip[RPT], nsl[RPT];
        double nxt[RPT];
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
            row[k] = tid + k * NT;
            strip[k] = row[k] >> 5;
            const int b0 = strip[k] * (strip[k] + 1) / 2;
            nsl[k] = ((b0 + strip[k] + 1) * nwe - 1) / nblk - ((b0 + 1) * nwe - 1) / nblk + 1;
            nxt[k] = row[k] < s ? Aj[row[k]] : 0.0;
        }
        // columns of a last, narrower panel up to the next multiple of 4 (K of the update)
        for (int q = nb; q < ((nb + 3) & ~3); ++q)
            for (int r = tid; r < ld; r += NT) V[q * ld + r] = W[q * ld + r] = 0.0;
        double tq = 0.0;   // tau of the panel's last reflector
        auto finish_w = [&](int q) {   // w of reflector q from the partial sums
            double vav = 0.0, vw = 0.0;
#pragma unroll
            for (int w = 0; w < NW; ++w) vav += rva[w];
            for (int i = 0; i < q; ++i) vw = fma(vtv[i], wtv[i], vw);
            const double hc = 0.5 * tq * (vav - 2.0 * vw);
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const int r = row[k];
                if (r > q && r < s) {
                    double y = 0.0;
                    for (int t = 0; t < nsl[k]; ++t) y += rowp[t * ld + r];
                    for (int I = strip[k]; I < T; ++I) y += colp[(I * (I + 1) / 2 + strip[k]) * 32 + lane];
                    for (int i = 0; i < q; ++i) y -= V[i * ld + r] * wtv[i] + W[i * ld + r] * vtv[i];
                    W[q * ld + r] = tq * (y - hc * V[q * ld + r]);
                } else if (r < ld) {
                    W[q * ld + r] = 0.0;
                }
            }
        };
        for (int jj = 0; jj < nb; ++jj) {
            const int j = j0 + jj;
            // ---- w of the previous reflector
            if (jj > 0) finish_w(jj - 1);
            __syncthreads();
            // ---- column j with the panel's updates, |x|^2 of its part below the subdiagonal
            double part = 0.0;
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const int r = row[k];
                if (r >= jj && r < s) {
                    double a = nxt[k];
                    for (int q = 0; q < jj; ++q) a -= V[q * ld + r] * W[q * ld + jj] + W[q * ld + r] * V[q * ld + jj];
                    nxt[k] = a;
                    yl[r] = a;
                    if (r >= jj + 2) part = fma(a, a, part);
                }
            }
            part = warp_sum(part);
            if (lane == 0) red[warp] = part;
            __syncthreads();
            // ---- reflector (dlarfg's convention), V^T v and W^T v
            double xn2 = 0.0;
#pragma unroll
            for (int w = 0; w < NW; ++w) xn2 += red[w];
            const double alpha = yl[jj + 1];
            double beta = alpha, sc = 0.0;
            tq = 0.0;
            if (xn2 != 0.0) {
                beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
                tq = (beta - alpha) / beta;
                sc = 1.0 / (alpha - beta);
            }
            for (int q = warp; q < jj; q += NW) {
                double dv = 0.0, dw = 0.0;
                for (int r = jj + 2 + lane; r < s; r += 32) {
                    dv = fma(V[q * ld + r], yl[r], dv);
                    dw = fma(W[q * ld + r], yl[r], dw);
                }
                dv = warp_sum(dv);
                dw = warp_sum(dw);
                if (lane == 0) {
                    vtv[q] = fma(sc, dv, V[q * ld + jj + 1]);
                    wtv[q] = fma(sc, dw, W[q * ld + jj + 1]);
                }
            }
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const int r = row[k];
                if (r < T * 32) {
                    const double v = (r < s && r > jj) ? (r == jj + 1 ? 1.0 : nxt[k] * sc) : 0.0;
                    vb[r] = v;
                    if (r < ld) V[jj * ld + r] = v;
                    if (r > jj + 1 && r < s) Aj[r + (int64_t)jj * m] = v;
                }
                // the next column, as it was at the panel's start
                if (jj + 1 < nb) nxt[k] = (r > jj && r < s) ? Aj[r + (int64_t)(jj + 1) * m] : 0.0;
            }
            if (tid == 0) {
                d[j] = yl[jj];
                e[j] = beta;
                tau[j] = tq;
            }
            __syncthreads();
            // ---- A v: this warp's run of lower-triangle blocks
            double vav = 0.0;
            if (warp < nwe) {
                int b = (int)((int64_t)nblk * warp / nwe);
                const int bend = (int)((int64_t)nblk * (warp + 1) / nwe);
                int I = (int)((sqrtf(8.0f * (float)b + 1.0f) - 1.0f) * 0.5f);
                while ((I + 1) * (I + 2) / 2 <= b) ++I;
                while (I * (I + 1) / 2 > b) --I;
                int J = b - I * (I + 1) / 2;
                double rp = 0.0;
                for (; b < bend; ++b) {
                    const int r = I * 32 + lane;
                    const double vr = vb[r];
                    const double* pa = Aj + (r < s ? r : 0) + (int64_t)J * 32 * m;
                    const double2* vc = reinterpret_cast<const double2*>(vb + J * 32);
                    double x[32];
                    if (I != J) {
#pragma unroll
                        for (int c = 0; c < 32; ++c) x[c] = pa[(int64_t)c * m];
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            const double2 v2 = vc[c];
                            rp = fma(x[2 * c], v2.x, rp);
                            rp = fma(x[2 * c + 1], v2.y, rp);
                        }
#pragma unroll
                        for (int c = 0; c < 32; ++c) x[c] *= vr;
                    } else {   // the diagonal block: its diagonal counts in the row sums only
#pragma unroll
                        for (int c = 0; c < 32; ++c) x[c] = (c <= lane && r < s) ? pa[(int64_t)c * m] : 0.0;
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            const double2 v2 = vc[c];
                            rp = fma(x[2 * c], v2.x, rp);
                            rp = fma(x[2 * c + 1], v2.y, rp);
                        }
#pragma unroll
                        for (int c = 0; c < 32; ++c) x[c] = c < lane ? x[c] * vr : 0.0;
                    }
                    const double cs = warp_transpose_sum(x, lane);
                    colp[b * 32 + lane] = cs;
                    vav = fma(vb[J * 32 + lane], cs, vav);
                    if (++J > I || b + 1 == bend) {   // the strip's sums of this warp
                        const int slot = warp - ((I * (I + 1) / 2 + 1) * nwe - 1) / nblk;
                        if (r < s) {
                            rowp[slot * ld + r] = rp;
                            vav = fma(vr, rp, vav);
                        }
                        rp = 0.0;
                        if (J > I) {
                            ++I;
                            J = 0;
                        }
                    }
                }
            }
            vav = warp_sum(vav);
            if (lane == 0) rva[warp] = vav;
            __syncthreads();
        }
        finish_w(nb - 1);
        __syncthreads();
        // ---- trailing block A -= V W^T + W V^T (lower 32 x 32 blocks, one per warp)
        const int s2 = s - nb, T2 = trd_strips(s2), nblk2 = T2 * (T2 + 1) / 2, K = (nb + 3) & ~3;
        const int g = lane >> 2, t4 = lane & 3;
        double* A2 = Aj + nb + (int64_t)nb * m;
        for (int b = warp; b < nblk2; b += NW) {
            int I = (int)((sqrtf(8.0f * (float)b + 1.0f) - 1.0f) * 0.5f);
            while ((I + 1) * (I + 2) / 2 <= b) ++I;
            while (I * (I + 1) / 2 > b) --I;
            const int J = b - I * (I + 1) / 2;
            // 16 rows of the block at a time (accumulators of 2 x 4 fragments)
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int r0 = I * 32 + h * 16, c0 = J * 32;
                if (r0 >= s2) break;
                double acc[2][4][2];
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y)
#pragma unroll
                        for (int z = 0; z < 2; ++z) {
                            const int r = r0 + 8 * x + g, c = c0 + 8 * y + 2 * t4 + z;
                            acc[x][y][z] = (r < s2 && c <= r) ? A2[r + (int64_t)c * m] : 0.0;
                        }
                for (int k = t4; k < K; k += 4) {
                    const double* Vk = V + k * ld + nb;
                    const double* Wk = W + k * ld + nb;
                    double av[2], aw[2], bv[4], bw[4];
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const int r = min(r0 + 8 * x + g, s2 - 1);   // rows past the end are not stored
                        av[x] = -Vk[r];
                        aw[x] = -Wk[r];
                    }
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        const int c = min(c0 + 8 * y + g, s2 - 1);
                        bv[y] = Vk[c];
                        bw[y] = Wk[c];
                    }
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int y = 0; y < 4; ++y) {
                            dmma(acc[x][y][0], acc[x][y][1], av[x], bw[y]);
                            dmma(acc[x][y][0], acc[x][y][1], aw[x], bv[y]);
                        }
                }
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y)
#pragma unroll
                        for (int z = 0; z < 2; ++z) {
                            const int r = r0 + 8 * x + g, c = c0 + 8 * y + 2 * t4 + z;
                            if (r < s2 && c <= r) A2[r + (int64_t)c * m] = acc[x][y][z];
                        }
            }
        }
        __syncthreads();
        j0 += nb;
    }
    if (tid == 0) {
        d[m - 1] = A[(m - 1) + (int64_t)(m - 1) * m];
        tau[m - 1] = 0.0;
    }
}
