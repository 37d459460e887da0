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
//     contiguous run of half blocks (32 x 16) per warp (run lengths differ by one
//     at most); the next half block's loads are in flight while one is multiplied.
//     A lane holds two rows and eight columns of a half block (16-byte loads, 256
//     bytes of two columns per instruction: 65 to 75 bytes per clock and SM, where
//     32 bytes of four columns per 8 lanes reach 31), so the row sums add up in its
//     registers and the column sums take 8 exchanges (one reduction per column
//     would take 80).  Row sums go to a slot per (warp of the strip, row), column
//     sums to a slot per block; both are added in a fixed order.
//   * The update after the panel runs on the FP64 tensor cores (DMMA) straight from
//     the shared V and W, a 32 x 32 block per warp and no barrier.
// NT = 512 threads (one CTA per SM) or 256 (two CTAs per SM, smaller orders).
// Measured: 96 problems of order 218-595, one CTA each: 7.0 ms (9.2 with 32
// bytes of four columns per 8 lanes, 29 with the unblocked reduction that read and wrote
// the whole trailing square per column); 602 problems of order <= 253, two CTAs per SM: 3.7 ms.

__host__ __device__ constexpr int trd_ld(int s) { return ((s + 11) / 16) * 16 + 4; }   // >= s, = 4 mod 16
__host__ __device__ constexpr int trd_strips(int s) { return (s + 31) / 32; }
__host__ __device__ constexpr int trd_blocks(int s) { return trd_strips(s) * (trd_strips(s) + 1) / 2; }
// Row slots: the most warps that one strip's half blocks are spread over.
__host__ __device__ constexpr int trd_row_slots(int s, int nw) {
    const int U = 2 * trd_strips(s), n = 2 * trd_blocks(s), run = n / nw > 1 ? n / nw : 1;
    return (U - 1 + run - 1) / run + 1;
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
// Shared memory per SM that the launch asks for, in doubles per CTA: what is not
// shared memory is L1, and the loads in flight need L1 lines.  With the panel filling
// the whole 227 KB the pass over the lower triangle ran at 29 bytes per clock and SM;
// panels of 8 columns in the smallest configuration that holds them leave 92 KB of L1
// at order 576.  Candidates: 132, 164, 196 and 227 KB per SM.
constexpr int kTrdCaps[4] = {132 * 1024, 164 * 1024, 196 * 1024, 232448 + 1024};
constexpr int trd_cap(int m, int nt) {   // doubles of one CTA of nt threads (512 / nt CTAs per SM), 0: too large
    for (int i = 0; i < 4; ++i) {
        const int cap = (kTrdCaps[i] * (nt / 32) / 16 - 1024) / 8;
        if (trd_panel_width(m, nt / 32, cap) >= 8) return cap;
    }
    return 0;
}
constexpr int kTrdMax512 = 800;   // orders one CTA takes (panels of 8 columns or more)
constexpr int kTrdMax256 = 288;   // orders two CTAs per SM take (panels of 8 columns or more)
static_assert(trd_cap(kTrdMax512, 512) > 0, "panel fits one CTA per SM");
static_assert(trd_cap(kTrdMax256, 256) > 0, "panel fits two CTAs per SM");

// 16-byte load that stays where it is written: ahead of the arithmetic before its use.
__device__ __forceinline__ double2 ld_ahead(const double* p) {
    double2 v;
    asm volatile("ld.global.v2.f64 {%0,%1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}

template <int NT>
__device__ void stage_trd(const EigProb& p, double* __restrict__ Ca, double* __restrict__ Da, double* __restrict__ Ea,
                          double* __restrict__ Ta, double* smem, int cap) {
    constexpr int NW = NT / 32, RPT = 2;   // rows per thread
    const int m = p.m, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double* A = Ca + p.coff;
    const int64_t lda = p.ldc;
    double* d = Da + p.voff;
    double* e = Ea + p.voff;
    double* tau = Ta + p.voff;
    double* red = smem;           // 16: partial |x|^2 of the warps
    double* rva = smem + 16;      // 16: partial v^T A v
    double* vtv = smem + 32;      // 16: V^T v
    double* wtv = smem + 48;      // 16: W^T v
    double* arr = smem + kTrdFixed;
    if (m & 1)   // the odd row's partner in the 16-byte loads
        for (int c = tid; c < m; c += NT) A[m + c * lda] = 0.0;
    __syncthreads();
    for (int j0 = 0; j0 < m - 1;) {
        const int s = m - j0, ld = trd_ld(s), T = trd_strips(s), nblk = trd_blocks(s), nun = 2 * nblk;
        const int width = trd_panel_width(s, NW, cap), nb = min(width, m - 1 - j0);
        const int nwe = min(NW, nun);
        double* V = arr;                       // V[q ld + r], r relative to j0
        double* W = V + width * ld;
        double* rowp = W + width * ld;         // [slot][r]
        double* yl = rowp + trd_row_slots(s, NW) * ld;
        double* colp = yl + ld;                // [block][32]
        double* vb = colp + nblk * 32;         // reflector, zero outside its rows
        double* Aj = A + j0 + (int64_t)j0 * lda; // element (r, c) of the trailing block at Aj[r + c lda]
        // this thread's rows and the slots of their row sums
        int row[RPT], strip[RPT], nsl[RPT];
        double nxt[RPT];
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
            row[k] = tid + k * NT;
            strip[k] = row[k] >> 5;
            const int u0 = strip[k] * (strip[k] + 1);
            nsl[k] = ((u0 + 2 * strip[k] + 2) * nwe - 1) / nun - ((u0 + 1) * nwe - 1) / nun + 1;
            nxt[k] = row[k] < s ? Aj[row[k]] : 0.0;
        }
        // this warp's run of half blocks: unit u = (strip I, columns 16 q ...), I (I + 1) + q
        const int ubeg = warp < nwe ? nun * warp / nwe : 0, uend = warp < nwe ? nun * (warp + 1) / nwe : 0;
        int Ibeg = (int)((sqrtf(4.0f * (float)ubeg + 1.0f) - 1.0f) * 0.5f);
        while ((Ibeg + 1) * (Ibeg + 2) <= ubeg) ++Ibeg;
        while (Ibeg * (Ibeg + 1) > ubeg) --Ibeg;
        // columns of a last, narrower panel up to the next multiple of 4 (K of the update)
        for (int q = nb; q < ((nb + 3) & ~3); ++q)
            for (int r = tid; r < ld; r += NT) V[q * ld + r] = W[q * ld + r] = 0.0;
        double tq = 0.0;   // tau of the panel's last reflector
        auto finish_w = [&](int q) {   // w of reflector q from the partial sums
            const double vav = warp_sum((lane < NW ? rva[lane & (NW - 1)] : 0.0) -
                                        (lane < q ? 2.0 * vtv[lane & 15] * wtv[lane & 15] : 0.0));
            const double hc = 0.5 * tq * vav;
#pragma unroll
            for (int k = 0; k < RPT; ++k) {
                const int r = row[k];
                if (r > q && r < s) {
                    double y = 0.0;
                    for (int t = 0; t < nsl[k]; ++t) y += rowp[t * ld + r];
#pragma unroll 4
                    for (int I = strip[k]; I < T; ++I) y += colp[(I * (I + 1) / 2 + strip[k]) * 32 + lane];
#pragma unroll 4
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
#pragma unroll 4
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
#pragma unroll 4
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
                    if (r > jj + 1 && r < s) Aj[r + jj * lda] = v;
                }
                // the next column, as it was at the panel's start
                if (jj + 1 < nb) nxt[k] = (r > jj && r < s) ? Aj[r + (jj + 1) * lda] : 0.0;
            }
            if (tid == 0) {
                d[j] = yl[jj];
                e[j] = beta;
                tau[j] = tq;
            }
            __syncthreads();
            // ---- A v: this warp's run of the lower triangle.  Lane (l, h) holds rows 2l,
            // 2l + 1 and the columns 2i + h of a half block.  Rows past the end are read
            // as row 0 or as the zeroed padding and meet zeros of v; columns past the
            // end (in a diagonal block only) are read as the last one and masked.
            double vav = 0.0;
            if (ubeg < uend) {
                const int l = lane & 15, h = lane >> 4;
                auto load = [&](double2(&x)[8], int I, int c0) {
                    const int r = I * 32 + 2 * l;
                    const double* pa = Aj + (r < s ? r : 0);
                    if (c0 + 16 <= s) {
                        pa += (c0 + h) * lda;
#pragma unroll
                        for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const double2*>(pa + 2 * i * lda);
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            x[i] = *reinterpret_cast<const double2*>(pa + min(c0 + h + 2 * i, s - 1) * lda);
                    }
                };
                int I = Ibeg, q = ubeg - I * (I + 1), u = ubeg;
                double rp0 = 0.0, rp1 = 0.0;
                double2 vr = *reinterpret_cast<const double2*>(vb + I * 32 + 2 * l);
                // one half block out of x, the next one's loads going into xn
                auto unit = [&](const double2(&x)[8], double2(&xn)[8]) {
                    const bool strip_end = q + 1 == 2 * (I + 1), more = u + 1 < uend;
                    const int In = strip_end ? I + 1 : I, qn = strip_end ? 0 : q + 1;
                    if (more) load(xn, In, qn * 16);
                    const int c0 = q * 16 + h, r0 = I * 32 + 2 * l;
                    double cs[8];
                    if (q < 2 * I) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const double vc = vb[c0 + 2 * i];
                            rp0 = fma(x[i].x, vc, rp0);
                            rp1 = fma(x[i].y, vc, rp1);
                            cs[i] = fma(x[i].x, vr.x, x[i].y * vr.y);
                        }
                    } else {   // a diagonal block: lower triangle, its diagonal in the row sums only
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int c = c0 + 2 * i;
                            const double vc = vb[c], a = c <= r0 ? x[i].x : 0.0, b = c <= r0 + 1 ? x[i].y : 0.0;
                            rp0 = fma(a, vc, rp0);
                            rp1 = fma(b, vc, rp1);
                            cs[i] = (c < r0 ? a * vr.x : 0.0) + (c <= r0 ? b * vr.y : 0.0);
                        }
                    }
                    // column sums over l: lane (l, h) ends with column 2 (l / 2) + h
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) {
                        const bool up = l & (2 * o);
#pragma unroll
                        for (int i = 0; i < o; ++i) {
                            const double send = up ? cs[i] : cs[i + o], keep = up ? cs[i + o] : cs[i];
                            cs[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * o);
                        }
                    }
                    cs[0] += __shfl_xor_sync(0xffffffffu, cs[0], 1);
                    if (!(l & 1)) {
                        const int c = q * 16 + l + h;
                        colp[(I * (I + 1) / 2) * 32 + c] = cs[0];
                        vav = fma(vb[c], cs[0], vav);
                    }
                    if (strip_end || !more) {   // the strip's sums of this warp
                        const int slot = warp - ((I * (I + 1) + 1) * nwe - 1) / nun;
                        const double rs = (h ? rp1 : rp0) + __shfl_xor_sync(0xffffffffu, h ? rp0 : rp1, 16);
                        if (r0 + h < s) {
                            rowp[slot * ld + r0 + h] = rs;
                            vav = fma(h ? vr.y : vr.x, rs, vav);
                        }
                        rp0 = rp1 = 0.0;
                        if (more) vr = *reinterpret_cast<const double2*>(vb + In * 32 + 2 * l);
                    }
                    I = In;
                    q = qn;
                    return ++u < uend;
                };
                double2 xa[8], xb[8];
                load(xa, I, q * 16);
                while (unit(xa, xb) && unit(xb, xa)) {}
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
        double* A2 = Aj + nb + nb * lda;
        // (the last panel leaves one element; every other one is a multiple of 4 wide,
        // so that rows pair up on 16-byte boundaries)
        for (int b = warp; b < nblk2; b += NW) {
            int I = (int)((sqrtf(8.0f * (float)b + 1.0f) - 1.0f) * 0.5f);
            while ((I + 1) * (I + 2) / 2 <= b) ++I;
            while (I * (I + 1) / 2 > b) --I;
            const int J = b - I * (I + 1) / 2;
            const bool inner = I != J && (I + 1) * 32 <= s2;
            // 16 columns of the block at a time: fragment (x, y) holds columns 8x + g and
            // rows 8y + 2 t4 + {0, 1}
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int r0 = I * 32, c0 = J * 32 + h * 16;
                double acc[2][4][2];
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        const int r = r0 + 8 * y + 2 * t4, c = c0 + 8 * x + g;
                        const double* pa = A2 + r + c * lda;
                        if (inner) {
                            const double2 v = *reinterpret_cast<const double2*>(pa);
                            acc[x][y][0] = v.x;
                            acc[x][y][1] = v.y;
                        } else {
                            acc[x][y][0] = (r < s2 && c <= r) ? pa[0] : 0.0;
                            acc[x][y][1] = (r + 1 < s2 && c <= r + 1) ? pa[1] : 0.0;
                        }
                    }
                for (int k = t4; k < K; k += 4) {
                    const double* Vk = V + k * ld + nb;
                    const double* Wk = W + k * ld + nb;
                    double av[2], aw[2], bv[4], bw[4];
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const int c = min(c0 + 8 * x + g, s2 - 1);   // columns and rows past the end are not stored
                        av[x] = -Vk[c];
                        aw[x] = -Wk[c];
                    }
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        const int r = min(r0 + 8 * y + g, s2 - 1);
                        bv[y] = Vk[r];
                        bw[y] = Wk[r];
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
                    for (int y = 0; y < 4; ++y) {
                        const int r = r0 + 8 * y + 2 * t4, c = c0 + 8 * x + g;
                        double* pa = A2 + r + c * lda;
                        if (inner) {
                            *reinterpret_cast<double2*>(pa) = make_double2(acc[x][y][0], acc[x][y][1]);
                        } else {
                            if (r < s2 && c <= r) pa[0] = acc[x][y][0];
                            if (r + 1 < s2 && c <= r + 1) pa[1] = acc[x][y][1];
                        }
                    }
            }
        }
        __syncthreads();
        j0 += nb;
    }
    if (tid == 0) {
        d[m - 1] = A[(m - 1) + (m - 1) * lda];
        tau[m - 1] = 0.0;
    }
}
