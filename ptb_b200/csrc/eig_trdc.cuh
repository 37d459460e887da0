// Householder tridiagonalisation of one symmetric matrix on a thread-block cluster
// (included by sm_eig.cu inside its namespace): the scheme of eig_trd.cuh spread over G
// CTAs.  What bounds it: the pass over the lower triangle, m^3/6 doubles out of L2 (out
// of HBM where the triangles of a batch exceed L2), and the chain of short steps per
// column.
//   * Rows are owned in 32-row chunks (chunk index modulo G, relative to the panel's
//     first row).  V, W and the partial sums of the owned rows live in the owner's
//     shared memory; nb is the widest of 16, 12, 8, 4 columns that fits.
//   * A v: the lower triangle in strips of 128 rows, cut into units of 128 x 8 elements;
//     every warp of the group takes a contiguous run of units (equal up to one), the next
//     32 rows' loads in flight while 32 rows of a unit are multiplied.  A lane holds two
//     rows of every 32 and every other column of a unit (16-byte loads, 256 bytes of two
//     columns per instruction), so row sums add up in its registers along the strip and
//     column sums over the strip's rows; 5 exchanges per unit remain.  Alone, the pass
//     runs at 76 bytes per clock and SM out of L2; with strips of 64 rows and units of
//     64 x 16 (less read above the diagonal, more exchanged) at 63, with the column sums
//     exchanged for every 32 rows at 52, with 32 bytes of four columns per 8 lanes at 31
//     (the L1 lines per instruction).  Row sums go to a slot per (warp of the strip,
//     row), column sums to a slot per strip, both in the owner's shared memory; they are
//     added in a fixed order.
//   * The updated column, the partial dot products and the panel's next row are
//     stored straight into every CTA's shared memory: two cluster barriers per column.
//   * The update after the panel runs on the FP64 tensor cores (DMMA), a 32 x 32
//     block per warp and no barrier.
constexpr int kTcFixed = 1024;      // doubles of the scalars in front of the panel's arrays
constexpr int kTcRed = 34;          // doubles of one CTA's partial sums: |x|^2, V^T x (16), W^T x (16)
constexpr int kTcNoRow = 1 << 30;
constexpr int kTcSr = 4;             // 32-row steps of a strip
constexpr int kTcRows = 32 * kTcSr;  // rows of a strip and of a unit
constexpr int kTcCols = 32 / kTcSr;  // columns of a unit
// Unit q of strip I is number tc_start(I) + q of the lower triangle.
__host__ __device__ constexpr int tc_strips(int s) { return (s + kTcRows - 1) / kTcRows; }
__host__ __device__ constexpr int tc_start(int I) { return kTcSr * kTcSr * (I * (I + 1) / 2); }
__host__ __device__ constexpr int tc_strip_units(int s) { return (s + kTcCols - 1) / kTcCols; }   // of the last strip
__host__ __device__ constexpr int tc_units(int s) { return tc_start(tc_strips(s) - 1) + tc_strip_units(s); }
// Warps that take part (runs of two units or more: more warps mean more row slots to add)
// and the row slots of a strip: the most warps that its units are spread over.
__host__ __device__ constexpr int tc_warps(int s, int nw) {
    const int w = tc_units(s) / 2;
    return w >= nw ? nw : w > 1 ? w : 1;
}
__host__ __device__ constexpr int tc_row_slots(int s, int nw) {
    const int run = tc_units(s) / tc_warps(s, nw);
    return (tc_strip_units(s) - 1 + run - 1) / run + 1;
}
__host__ __device__ constexpr int tc_own(int s, int G) { return ((s + 31) / 32 + G - 1) / G; }   // chunks per CTA
// Doubles of shared memory per CTA of a panel of nb columns at trailing order s, G CTAs.
constexpr int kTcWarps = kT / 32;
__host__ __device__ constexpr int tc_panel_doubles(int s, int nb, int G) {
    const int nown = tc_own(s, G), ldo = nown * 32 + 4, Ts = tc_strips(s);
    return (2 * nb + 1 + tc_row_slots(s, G * kTcWarps)) * ldo + Ts * kTcRows + nown * Ts * 32;
}
__host__ __device__ constexpr int tc_panel_width(int s, int G, int cap) {
    return tc_panel_doubles(s, 16, G) + kTcFixed <= cap   ? 16
           : tc_panel_doubles(s, 12, G) + kTcFixed <= cap ? 12
           : tc_panel_doubles(s, 8, G) + kTcFixed <= cap  ? 8
           : tc_panel_doubles(s, 4, G) + kTcFixed <= cap  ? 4
                                                          : 0;
}
// Shared memory per SM that a launch asks for (what is not shared memory is L1, and the
// loads in flight need L1 lines), in doubles per CTA: the smallest with panels of
// kTcMinWidth columns or more, 0: too large for G CTAs.
constexpr int kTcMinWidth = 8;
constexpr int tc_cap(int m, int G) {
    if (tc_own(m, G) > kTcWarps) return 0;   // a warp owns one chunk at most
    for (int i = 0; i < 4; ++i) {
        const int cap = (kTrdCaps[i] - 1024) / 8;
        if (tc_panel_width(m, G, cap) >= kTcMinWidth) return cap;
    }
    return 0;
}
constexpr int kTcPadCols = 16;      // zeroed columns after a problem's C, and 128 rows
constexpr int kTcPadRows = 128;
// Pg: the panel's V and W rows for the update, m x 32 doubles of global scratch (row r: V
// 16, W 16).
__device__ void stage_trd_cluster(const EigProb& p, double* __restrict__ Ca, double* __restrict__ Da,
                                  double* __restrict__ Ea, double* __restrict__ Ta, double* __restrict__ Pg,
                                  double* smem, int cap) {
    constexpr int NT = kT, NW = kTcWarps, SR = kTcSr, H = kTcRows, UC = SR * SR, NC = kTcCols / 2;
    cg::cluster_group cl = cg::this_cluster();
    const int G = (int)cl.num_blocks(), rk = (int)cl.block_rank(), gsh = 31 - __clz(G);   // G: a power of two
    const int m = p.m, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gw = rk * NW + warp;
    auto at = [&](double* q, int g) { return cl.map_shared_rank(q, g); };
    double* A = Ca + p.coff;
    const int64_t lda = p.ldc;
    double* d = Da + p.voff;
    double* e = Ea + p.voff;
    double* tau = Ta + p.voff;
    double* red = smem;                  // [CTA][kTcRed]
    double* rva = smem + 16 * kTcRed;   // [warp of the group]: partial v^T A v (at most 256)
    double* rows = rva + 256;            // two rows of the panel: [parity][V 16, W 16]
    double* vtv = rows + 64;             // 16
    double* wtv = vtv + 16;              // 16
    double* scal = wtv + 16;             // a_jj, a_jj+1
    double* arr = smem + kTcFixed;
    // what the pass over the lower triangle may read past the matrix: zeros
    const int pad = (int)lda - m;
    for (int64_t i = rk * NT + tid; i < (int64_t)m * pad; i += G * NT) A[m + i % pad + i / pad * lda] = 0.0;
    for (int64_t i = rk * NT + tid; i < kTcPadCols * lda + kTcPadRows; i += G * NT) A[m * lda + i] = 0.0;
    cl.sync();
    for (int j0 = 0; j0 < m - 1;) {
        const int s = m - j0, Ts = tc_strips(s), nun = tc_units(s);
        const int nown = tc_own(s, G), ldo = nown * 32 + 4;
        const int width = tc_panel_width(s, G, cap), nb = min(width, m - 1 - j0);
        const int nwe = tc_warps(s, NW * G);
        double* V = arr;                       // [q][owned row]
        double* W = V + width * ldo;
        double* yl = W + width * ldo;          // owned rows of the updated column
        double* rowp = yl + ldo;               // [slot][owned row]
        double* vb = rowp + tc_row_slots(s, NW * G) * ldo;   // the column, then the reflector (Ts H)
        double* colp = vb + Ts * H;            // [owned chunk][strip][32]
        double* Aj = A + j0 + j0 * lda;        // element (r, c) of the trailing block at Aj[r + c lda]
        // this thread's row (rows past s: the owned arrays hold zeros) and its place there
        const int r = warp < nown ? (rk + G * warp) * 32 + lane : kTcNoRow, o = warp * 32 + lane;
        double nxt = r < s ? Aj[r] : 0.0;
        // slots of strip I: from the warp of its first unit to the warp of its last
        auto first_warp = [&](int I) { return ((tc_start(I) + 1) * nwe - 1) / nun; };
        auto slots = [&](int I) {
            const int end = I + 1 == Ts ? nun : tc_start(I + 1);
            return (end * nwe - 1) / nun - first_warp(I) + 1;
        };
        const int nsl = r < s ? slots(r / H) : 0;
        const int nsl0 = slots(0);
        // this warp's run of units
        const int ubeg = gw < nwe ? nun * gw / nwe : 0, uend = gw < nwe ? nun * (gw + 1) / nwe : 0;
        int Ibeg = 0;
        while (tc_start(Ibeg + 1) <= ubeg) ++Ibeg;
        double tq = 0.0;   // tau of the panel's last reflector
        // w of reflector q on the owned rows; on a cluster also V and W at row q + 1 (the
        // next column's) for every CTA: that row is in chunk 0, owned by CTA 0
        auto finish_w = [&](int q) {
            double vav = 0.0;
            for (int w = lane; w < NW * G; w += 32) vav += rva[w];
            if (lane < q) vav -= 2.0 * vtv[lane] * wtv[lane];
            const double hc = 0.5 * tq * warp_sum(vav);
            if (warp == NW - 1) {
                const double *rp0 = at(rowp, 0), *cp0 = at(colp, 0), *rw = rows + ((q + 1) & 1) * 32;
                double y = 0.0;
                for (int t = lane; t < nsl0; t += 32) y += rp0[t * ldo + q + 1];
                for (int I = lane; I < Ts; I += 32) y += cp0[I * 32 + q + 1];
                if (lane < q) y -= rw[lane] * wtv[lane] + rw[16 + lane] * vtv[lane];
                y = warp_sum(y);
                if (lane == 0) {
                    rows[((q + 1) & 1) * 32 + q] = 1.0;
                    rows[((q + 1) & 1) * 32 + 16 + q] = tq * (y - hc);
                }
            }
            if (r >= kTcNoRow) return;
            double w = 0.0;
            if (r > q && r < s) {
                double y = 0.0;
#pragma unroll 4
                for (int t = 0; t < nsl; ++t) y += rowp[t * ldo + o];
                const double* cp = colp + warp * Ts * 32 + lane;
#pragma unroll 4
                for (int I = r / H; I < Ts; ++I) y += cp[I * 32];
#pragma unroll 4
                for (int i = 0; i < q; ++i) y -= V[i * ldo + o] * wtv[i] + W[i * ldo + o] * vtv[i];
                w = tq * (y - hc * V[q * ldo + o]);
            }
            W[q * ldo + o] = w;
        };
        for (int jj = 0; jj < nb; ++jj) {
            const int j = j0 + jj;
            const double *rv = rows + (jj & 1) * 32, *rw = rv + 16;   // V and W at row jj
            if (jj > 0) finish_w(jj - 1);
            __syncthreads();
            // ---- column j with the panel's updates, to every CTA; |x|^2, V^T x, W^T x
            double part = 0.0;
            if (r >= jj && r < s) {
                double a = nxt;
#pragma unroll 4
                for (int q = 0; q < jj; ++q) a -= V[q * ldo + o] * rw[q] + W[q * ldo + o] * rv[q];
                nxt = a;
                yl[o] = r >= jj + 2 ? a : 0.0;
                if (r >= jj + 2) part = fma(a, a, part);
                for (int g = 0; g < G; ++g) at(vb, g)[r] = a;
                if (r <= jj + 1)
                    for (int g = 0; g < G; ++g) at(scal, g)[r - jj] = a;
            } else if (r < kTcNoRow) {
                yl[o] = 0.0;
            }
            part = warp_sum(part);
            if (lane == 0) rva[warp] = part;   // (rva is free between its reads above and the next A v)
            __syncthreads();
            for (int t = warp; t < 2 * jj + 1; t += NW) {
                double acc = 0.0;
                if (t == 2 * jj) {
                    acc = lane < NW ? rva[lane] : 0.0;
                } else {
                    const double* col = t < jj ? V + t * ldo : W + (t - jj) * ldo;
#pragma unroll 4
                    for (int i = lane; i < nown * 32; i += 32) acc = fma(col[i], yl[i], acc);
                }
                acc = warp_sum(acc);
                const int slot = t == 2 * jj ? 0 : t < jj ? 1 + t : 17 + t - jj;
                if (lane < G) at(red, lane)[rk * kTcRed + slot] = acc;
            }
            if (rk == 0 && warp == NW - 1 && lane < jj)   // the panel's row jj + 1
                for (int g = 0; g < G; ++g) {
                    double* rn = at(rows, g) + ((jj + 1) & 1) * 32;
                    rn[lane] = V[lane * ldo + jj + 1];
                    rn[16 + lane] = W[lane * ldo + jj + 1];
                }
            cl.sync();
            // ---- reflector (dlarfg's convention), V^T v and W^T v
            double xn2 = 0.0;
            for (int g = 0; g < G; ++g) xn2 += red[g * kTcRed];
            const double alpha = scal[1];
            double beta = alpha, sc = 0.0;
            tq = 0.0;
            if (xn2 != 0.0) {
                beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
                tq = (beta - alpha) / beta;
                sc = 1.0 / (alpha - beta);
            }
            if (tid < 2 * jj) {
                const int q = tid < jj ? tid : tid - jj, i = tid < jj ? q : 16 + q;
                double acc = 0.0;
                for (int g = 0; g < G; ++g) acc += red[g * kTcRed + 1 + i];
                (tid < jj ? vtv : wtv)[q] = fma(sc, acc, rows[((jj + 1) & 1) * 32 + i]);
            }
            for (int i = tid; i < Ts * H; i += NT)
                vb[i] = (i > jj && i < s) ? (i == jj + 1 ? 1.0 : vb[i] * sc) : 0.0;
            if (r < kTcNoRow) {
                const double v = (r < s && r > jj) ? (r == jj + 1 ? 1.0 : nxt * sc) : 0.0;
                V[jj * ldo + o] = v;
                if (r > jj + 1 && r < s) Aj[r + jj * lda] = v;
            }
            // the next column, as it was at the panel's start
            if (jj + 1 < nb) nxt = (r > jj && r < s) ? Aj[r + (jj + 1) * lda] : 0.0;
            if (rk == 0 && tid == 0) {
                d[j] = scal[0];
                e[j] = beta;
                tau[j] = tq;
            }
            __syncthreads();
            // ---- A v over this warp's units.  Lane (l, h) holds rows 2l, 2l + 1 of each 32
            // and the columns 2i + h.  What is read past the end are finite numbers: past
            // the last row they meet zeros of v, past the last column they are masked
            // with the rest above the diagonal.  One 32-row step is loaded ahead.
            double vav = 0.0;
            if (ubeg < uend) {
                const int l = lane & 15, h = lane >> 4;
                int I = Ibeg, q = ubeg - tc_start(Ibeg);
                double2 buf[2][NC];
                auto load = [&](int k, const double* pa) {
#pragma unroll
                    for (int i = 0; i < NC; ++i) buf[k & 1][i] = ld_ahead(pa + 32 * k + 2 * i * lda);
                };
                double rp[SR][2];
#pragma unroll
                for (int k = 0; k < SR; ++k) rp[k][0] = rp[k][1] = 0.0;
                const double* pa = Aj + I * H + 2 * l + (q * (2 * NC) + h) * lda;
                load(0, pa);
                for (int u = ubeg;;) {
                    const bool strip_end = q + 1 == UC * (I + 1), more = ++u < uend;
                    const int c0 = q * (2 * NC) + h, r0 = I * H + 2 * l;
                    const double* vc = vb + c0;
                    double cs[NC];
#pragma unroll
                    for (int i = 0; i < NC; ++i) cs[i] = 0.0;
#pragma unroll
                    for (int k = 0; k < SR; ++k) {
                        if (k + 1 < SR) {
                            load(k + 1, pa);
                        } else if (more) {
                            pa = strip_end ? Aj + (I + 1) * H + 2 * l + h * lda : pa + 2 * NC * lda;
                            load(0, pa);
                        }
                        const int r = r0 + 32 * k;
                        const double2 vr = *reinterpret_cast<const double2*>(vb + r);
                        if (q < UC * I) {
#pragma unroll
                            for (int i = 0; i < NC; ++i) {
                                const double2 x = buf[k & 1][i];
                                rp[k][0] = fma(x.x, vc[2 * i], rp[k][0]);
                                rp[k][1] = fma(x.y, vc[2 * i], rp[k][1]);
                                cs[i] = fma(x.x, vr.x, fma(x.y, vr.y, cs[i]));
                            }
                        } else {   // on the diagonal: lower triangle, the diagonal in the row sums only
#pragma unroll
                            for (int i = 0; i < NC; ++i) {
                                const double2 x = buf[k & 1][i];
                                const int c = c0 + 2 * i;
                                const double a = c <= r ? x.x : 0.0, b = c <= r + 1 ? x.y : 0.0;
                                rp[k][0] = fma(a, vc[2 * i], rp[k][0]);
                                rp[k][1] = fma(b, vc[2 * i], rp[k][1]);
                                cs[i] += (c < r ? a * vr.x : 0.0) + (c <= r ? b * vr.y : 0.0);
                            }
                        }
                    }
                    // column sums over l: lane (l, h) ends with column 2 (l / SR) + h
#pragma unroll
                    for (int o = NC / 2; o > 0; o >>= 1) {
                        const bool up = l & (SR * o);
#pragma unroll
                        for (int i = 0; i < o; ++i) {
                            const double send = up ? cs[i] : cs[i + o], keep = up ? cs[i + o] : cs[i];
                            cs[i] = keep + __shfl_xor_sync(0xffffffffu, send, SR * o);
                        }
                    }
#pragma unroll
                    for (int o = SR / 2; o > 0; o >>= 1) cs[0] += __shfl_xor_sync(0xffffffffu, cs[0], o);
                    if (!(l & (SR - 1))) {
                        const int c = q * (2 * NC) + 2 * (l / SR) + h, ch = c >> 5;
                        at(colp, ch & (G - 1))[((ch >> gsh) * Ts + I) * 32 + (c & 31)] = cs[0];
                        vav = fma(vb[c], cs[0], vav);
                    }
                    if (strip_end || !more) {   // the strip's sums of this warp
                        const int slot = gw - first_warp(I);
#pragma unroll
                        for (int k = 0; k < SR; ++k) {
                            const int ch = I * SR + k, r = ch * 32 + 2 * l + h;
                            const double t = (h ? rp[k][1] : rp[k][0]) +
                                             __shfl_xor_sync(0xffffffffu, h ? rp[k][0] : rp[k][1], 16);
                            if (r < s) {
                                at(rowp, ch & (G - 1))[slot * ldo + (ch >> gsh) * 32 + 2 * l + h] = t;
                                vav = fma(vb[r], t, vav);
                            }
                            rp[k][0] = rp[k][1] = 0.0;
                        }
                    }
                    if (!more) break;
                    I = strip_end ? I + 1 : I;
                    q = strip_end ? 0 : q + 1;
                }
            }
            vav = warp_sum(vav);
            if (lane < G) at(rva, lane)[gw] = vav;
            cl.sync();
        }
        finish_w(nb - 1);
        __syncthreads();
        if (r < s) {   // the panel's rows to global memory, row r: V 16, W 16
            double2* pr = reinterpret_cast<double2*>(Pg + (int64_t)r * 32);
            for (int q = 0; q < 8; ++q) {
                const int a = 2 * q, b = 2 * q + 1;
                pr[q] = make_double2(a < nb ? V[a * ldo + o] : 0.0, b < nb ? V[b * ldo + o] : 0.0);
                pr[8 + q] = make_double2(a < nb ? W[a * ldo + o] : 0.0, b < nb ? W[b * ldo + o] : 0.0);
            }
        }
        cl.sync();
        // ---- trailing block A -= V W^T + W V^T (lower 32 x 32 blocks, one per warp, 16
        // columns at a time): fragment (x, y) holds columns 8x + g and rows 8y + 2 t4 +
        // {0, 1}.  The last panel leaves one element; every other one is a multiple of 4
        // wide, so that rows pair up on 16-byte boundaries.
        const int s2 = s - nb, T2 = (s2 + 31) / 32, nblk2 = T2 * (T2 + 1) / 2;
        const int g = lane >> 2, t4 = lane & 3;
        double* A2 = Aj + nb + nb * lda;
        for (int b = gw; b < nblk2; b += NW * G) {
            int I = (int)((sqrtf(8.0f * (float)b + 1.0f) - 1.0f) * 0.5f);
            while ((I + 1) * (I + 2) / 2 <= b) ++I;
            while (I * (I + 1) / 2 > b) --I;
            const int J = b - I * (I + 1) / 2;
            const bool inner = I != J && (I + 1) * 32 <= s2;
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
                // a lane's k of step kk is 4 t4 + kk: 32 consecutive bytes of a row
                auto mul = [&](const double(&av)[2], const double(&aw)[2], const double(&bv)[4], const double(&bw)[4]) {
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int y = 0; y < 4; ++y) {
                            dmma(acc[x][y][0], acc[x][y][1], -av[x], bw[y]);
                            dmma(acc[x][y][0], acc[x][y][1], -aw[x], bv[y]);
                        }
                };
                // columns and rows past the end are not stored
#pragma unroll 1
                for (int k2 = 0; k2 < 2; ++k2) {
                    double2 av[2], aw[2], bv[4], bw[4];
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const double* pr = Pg + (int64_t)(nb + min(c0 + 8 * x + g, s2 - 1)) * 32 + 4 * t4 + 2 * k2;
                        av[x] = *reinterpret_cast<const double2*>(pr);
                        aw[x] = *reinterpret_cast<const double2*>(pr + 16);
                    }
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        const double* pr = Pg + (int64_t)(nb + min(r0 + 8 * y + g, s2 - 1)) * 32 + 4 * t4 + 2 * k2;
                        bv[y] = *reinterpret_cast<const double2*>(pr);
                        bw[y] = *reinterpret_cast<const double2*>(pr + 16);
                    }
                    mul({av[0].x, av[1].x}, {aw[0].x, aw[1].x}, {bv[0].x, bv[1].x, bv[2].x, bv[3].x},
                        {bw[0].x, bw[1].x, bw[2].x, bw[3].x});
                    mul({av[0].y, av[1].y}, {aw[0].y, aw[1].y}, {bv[0].y, bv[1].y, bv[2].y, bv[3].y},
                        {bw[0].y, bw[1].y, bw[2].y, bw[3].y});
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
        cl.sync();
        j0 += nb;
    }
    if (rk == 0 && tid == 0) {
        d[m - 1] = A[(m - 1) + (m - 1) * lda];
        tau[m - 1] = 0.0;
    }
}
