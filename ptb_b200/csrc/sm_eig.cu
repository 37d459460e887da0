// Batched FP64 generalized eigensolver: the submatrix method's pencils, the
// many-molecule densities and single dense problems.
//
// The reference solves H_k U = S_k U diag(e) with LAPACK dsygvd per submatrix
// (la_sygvd, source/sm.f90:296-299), forms S_k U for the electron-count
// weights fe (source/sm.f90:305-310) and, at the final chemical potential,
// P_k = U occ U^T of which only the owned columns are kept
// (source/sm.f90:343-362).  Only these quantities leave the solver, and all of
// them are reached without forming U:
//
//   S_k = L L^T                      Cholesky, blocked
//   C   = L^-1 H_k L^-T              two blocked triangular solves, the second for the
//                                    lower triangle only
//   C   = Q T Q^T                    Householder tridiagonalisation, lower,
//                                    Q = H_0 H_1 ... H_{m-3}
//   T   = Z diag(e) Z^T              divide and conquer (eig_dc.cuh)
//   U   = L^-T Q Z                   never formed (eig_vec.cuh):
//     rows c of U    = (L^-T)[c,:] Q Z,  rows c of S U = L[c,:] Q Z  for the
//     owned columns c, so fe_j = sum_c (SU)[c,j] U[c,j];
//     P_k[:,c] = U (occ o U[c,:]^T) = L^-T (Q (Z w)).
//
// Every stage is a launch (or a few) over all problems of the batch, with its own
// split: one CTA or one thread-block cluster per problem where the stage is a chain over
// the whole problem (tridiagonalisation), one CTA per 64-row block, panel, tile or chunk
// of roots where it is not, largest problems first.  A batch of uneven problems then
// costs its total work over the SMs in all stages but that one, where one CTA or
// cluster per problem for everything cost the largest problem's whole chain.
//
// Each step's quantities are summed in a fixed order, so results do not depend
// on scheduling.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <numeric>
#include <vector>

#include "sm_eig.cuh"

namespace ptb {

namespace cg = cooperative_groups;

namespace {

constexpr int kT = 512;           // threads of the per-problem CTAs (16 warps)
constexpr int NB = 32;            // panel width of the blocked stages
constexpr int TS = 64;            // output tile of the blocked updates
constexpr int kQlMaxIter = 30;    // QL sweeps per eigenvalue of a leaf before giving up (as LAPACK's dsteqr)

// Status words per problem.
constexpr int kStOk = 0;
constexpr int kStNoConv = -1;     // a leaf's QL sweeps exhausted
// > 0: leading minor of that order of S_k is not positive definite

struct EigProb {
    int k, m, nown;
    int kind;             // 0: H U = S U e; 1: standard problem (S not read, L = I)
    int mode;             // 0: eigenvalues, fe, owned rows; 1: all vectors; 2: density U_occ U_occ^T (m x m at boff)
    int nocc;             // mode 2: occupied eigenvectors (the lowest)
    int64_t moff, eoff, o0;
    int64_t gbase, gld;   // the problem's H / S: element (i, j) at gbase + map(i) + map(j) gld
    int64_t poff;         // dense output of the owned columns of P (m x nown, column-major)
    int64_t aoff;     // L, Z and merge-workspace arenas (m x m, column-major, ld = m)
    int64_t coff;     // C arena (m columns, ld = ldc: a multiple of 16, so that columns start on 128-byte lines)
    int ldc;
    int64_t voff;     // d, e, tau, eigenvalue arenas (m)
    int64_t boff;     // owned-row arena (4 nown x m)
    int64_t xoff;     // scratch of the cluster and grid tridiagonalisations
    int64_t koff;     // T of the compact WY panels (t_panels(m) x TS^2)
    int64_t ioff;     // inverses of the diagonal blocks of L (TS^2 per 64 rows)
    int topm;         // index of the divide and conquer's last merge (-1: one leaf)
};

// ---------------------------------------------------------------------------
// Tile products on the FP64 tensor cores: one TS x TS output tile per CTA, the
// K range staged through shared memory in NB-deep chunks (the next chunk's
// loads in flight in registers while the current one is multiplied), each of
// the 16 warps owning a 16 x 16 block of the tile as 2 x 2 fragments of
// mma.m8n8k4.f64 (A fragment: lane holds A[g][t4]; B fragment: B[t4][g];
// accumulator: C[g][2 t4 + h], g = lane / 4, t4 = lane % 4).
//   A(i, k) = AT ? A[kg + (r0+i) lda] : A[(r0+i) + kg lda],   kg = kx ? kx[k] : k
//   B(k, j) = BT ? B[(c0+j) + kg ldb] : B[kg + (c0+j) ldb],   kg = kxb ? kxb[k] : k
//   MMA_SET: C[crow + r0 + i, col] = sum_k A(i,k) B(k,j); MMA_SUB: C[...] -= sum;
//   MMA_NEG: C[...] = -sum;
//   col = ccol ? ccol[c0+j] : c0+j; LOWER: only r0+i >= c0+j is written.
// Staged layouts keep both the stores (contiguous global runs) and the
// fragment reads free of bank conflicts: the operand whose global run is along
// the tile edge is stored k-major with row stride 68, the other edge-major with
// stride 36 (both = 4 mod 16 doubles).
constexpr int kStageOp = 2304;   // doubles of one staged operand chunk (max of 32 x 68 and 64 x 36)
enum { MMA_SET = 0, MMA_SUB = 1, MMA_NEG = 2 };

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}
template <bool AT>
__device__ __forceinline__ int sa_idx(int i, int k) {
    return AT ? i * 36 + k : k * 68 + i;
}
template <bool BT>
__device__ __forceinline__ int sb_idx(int k, int j) {
    return BT ? k * 68 + j : j * 36 + k;
}

// AREF / BREF: the operand is a panel of Householder reflectors stored as
// below, read with its implicit structure (1 where the row equals the
// reflector's index, the stored value below it, 0 above): A(i, k) is reflector
// r0+i at row k when AT, row r0+i of reflector k otherwise; B(k, j) is row k of
// reflector c0+j.
template <bool AT, bool BT, int MODE, bool LOWER, bool AREF = false, bool BREF = false>
__device__ void tile_mma(double* __restrict__ C, int64_t ldc, int crow, const int* ccol, int r0, int c0, int mr,
                         int nc, const double* __restrict__ A, int64_t lda, const int* kx,
                         const double* __restrict__ B, int64_t ldb, const int* kxb, int K, double* sA, double* sB) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int wr = (warp & 3) * 16, wc = (warp >> 2) * 16;
    double acc[2][2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    constexpr int kPer = TS * NB / kT;   // staged elements of A (and of B) per thread
    double ra[kPer], rb[kPer];
    auto fetch = [&](int k0) {
        const int kk = min(NB, K - k0);
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int t = tid + q * kT;
            const int i = AT ? t / NB : t % TS, k = AT ? t % NB : t / TS;
            double v = 0.0;
            if (i < mr && k < kk) {
                const int64_t kg = kx ? kx[k0 + k] : (k0 + k);
                if (AREF) {
                    const int64_t ig = r0 + i;   // AT: reflector ig at row kg; else row ig of reflector kg
                    const int64_t row = AT ? kg : ig, refl = AT ? ig : kg;
                    v = (row == refl) ? 1.0 : (row > refl ? A[row + refl * lda] : 0.0);
                } else {
                    v = AT ? A[kg + (int64_t)(r0 + i) * lda] : A[(int64_t)(r0 + i) + kg * lda];
                }
            }
            ra[q] = v;
            const int j = BT ? t % TS : t / NB, kb = BT ? t / TS : t % NB;
            double w = 0.0;
            if (j < nc && kb < kk) {
                const int64_t kg = kxb ? kxb[k0 + kb] : (k0 + kb);
                if (BREF) {
                    const int64_t refl = c0 + j;
                    w = (kg == refl) ? 1.0 : (kg > refl ? B[kg + refl * ldb] : 0.0);
                } else {
                    w = BT ? B[(int64_t)(c0 + j) + kg * ldb] : B[kg + (int64_t)(c0 + j) * ldb];
                }
            }
            rb[q] = w;
        }
    };
    auto stash = [&]() {
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int t = tid + q * kT;
            const int i = AT ? t / NB : t % TS, k = AT ? t % NB : t / TS;
            sA[sa_idx<AT>(i, k)] = ra[q];
            const int j = BT ? t % TS : t / NB, kb = BT ? t / TS : t % NB;
            sB[sb_idx<BT>(kb, j)] = rb[q];
        }
    };
    fetch(0);
    stash();
    __syncthreads();
    for (int k0 = 0; k0 < K; k0 += NB) {
        const bool more = k0 + NB < K;
        if (more) fetch(k0 + NB);
        const int ksteps = (min(NB, K - k0) + 3) >> 2;
        for (int ks = 0; ks < ksteps; ++ks) {
            const int k = ks * 4 + t4;
            const double a0 = sA[sa_idx<AT>(wr + g, k)], a1 = sA[sa_idx<AT>(wr + 8 + g, k)];
            const double b0 = sB[sb_idx<BT>(k, wc + g)], b1 = sB[sb_idx<BT>(k, wc + 8 + g)];
            dmma(acc[0][0][0], acc[0][0][1], a0, b0);
            dmma(acc[0][1][0], acc[0][1][1], a0, b1);
            dmma(acc[1][0][0], acc[1][0][1], a1, b0);
            dmma(acc[1][1][0], acc[1][1][1], a1, b1);
        }
        __syncthreads();
        if (more) {
            stash();
            __syncthreads();
        }
    }
    // accumulator acc[a][b][h] is C(wr + 8a + g, wc + 8b + 2 t4 + h); for a
    // read-modify-write every load is issued before any store
    double cv[2][2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = wr + 8 * a + g, j = wc + 8 * b + 2 * t4 + h;
                const bool ok = i < mr && j < nc && !(LOWER && r0 + i < c0 + j);
                cv[a][b][h] = 0.0;
                if (MODE == MMA_SUB && ok) {
                    const int64_t col = ccol ? ccol[c0 + j] : (c0 + j);
                    cv[a][b][h] = C[(int64_t)(crow + r0 + i) + col * ldc];
                }
            }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = wr + 8 * a + g, j = wc + 8 * b + 2 * t4 + h;
                const bool ok = i < mr && j < nc && !(LOWER && r0 + i < c0 + j);
                if (ok) {
                    const int64_t col = ccol ? ccol[c0 + j] : (c0 + j);
                    C[(int64_t)(crow + r0 + i) + col * ldc] =
                        MODE == MMA_SUB   ? cv[a][b][h] - acc[a][b][h]
                        : MODE == MMA_NEG ? -acc[a][b][h]
                                          : acc[a][b][h];
                }
            }
    __syncthreads();
}

// C[r0+i, c0+j] -= sum_{k < kk} A(i,k) B(k,j) on one TS x TS tile (mr x nc
// valid):  A(i,k) = A[(r0+i) + k lda],  B(k,j) = BT ? B[(c0+j) + k ldb] : B[k + (c0+j) ldb].
// LOWER: only elements on or below the diagonal of C are written.
template <bool BT, bool LOWER>
__device__ void tile_update(double* __restrict__ C, int ldc, int r0, int c0, int mr, int nc,
                            const double* __restrict__ A, int lda, const double* __restrict__ B, int ldb, int kk,
                            double* sA, double* sB) {
    tile_mma<false, BT, MMA_SUB, LOWER>(C, ldc, 0, nullptr, r0, c0, mr, nc, A, lda, nullptr, B, ldb, nullptr, kk,
                                        sA, sB);
}

// Fixed-order sum over the CTA (every thread gets the result).
__device__ double cta_sum(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += red[q];
    __syncthreads();
    return s;
}

__device__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------
// C[crow + r0 + i, col(c0 + j)] = sum_k A(i, kx(k)) B(kxb(k), j) on one TS x TS
// output tile (tile_mma, MMA_SET).
template <bool AT, bool BT = false>
__device__ void tile_gemm(double* __restrict__ C, int64_t ldc, int crow, const int* ccol, int r0, int c0, int mr,
                          int nc, const double* __restrict__ A, int64_t lda, const int* kx,
                          const double* __restrict__ B, int64_t ldb, const int* kxb, int K, double* sA, double* sB) {
    tile_mma<AT, BT, MMA_SET, false>(C, ldc, crow, ccol, r0, c0, mr, nc, A, lda, kx, B, ldb, kxb, K, sA, sB);
}

static_assert(TS * NB % kT == 0, "tile staging divides over the CTA");

// ---------------------------------------------------------------------------
// Compact WY panels of Q = H_0 ... H_{m-3}: TS reflectors each, so that V^T X fills
// the rows of a tile product and X - V Y2 has a K range of two chunks.
__host__ __device__ constexpr int64_t t_panels(int m) { return m > 2 ? (m - 2 + TS - 1) / TS : 0; }
constexpr int kTld = TS + 1;

// T of the compact WY form I - V T V^T of panel `pan`: the panel's Gram V^T V as one
// tile product reading the reflectors in place, the two halves' T column by column
// (T_bb = tau_b, T[0:b, b] = -tau_b T[0:b, 0:b] G[0:b, b]) by one warp each, and
// between them T12 = -T11 G12 T22.  Tp: TS x TS, column-major, zero outside the
// panel's nb x nb upper triangle.  G: TS x TS, T: TS x kTld shared.
__device__ void build_T(const double* __restrict__ C, int64_t ldc, int m, const double* __restrict__ tau,
                        double* __restrict__ Tp, int pan, double* G, double* T, double* sA, double* sB) {
    static_assert(TS == 64 && NB == 32, "a panel is two halves of one warp's width");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int j0 = pan * TS, nb = min(TS, m - 2 - j0), r0 = j0 + 1, len = m - r0;
    const double* Vb = C + r0 + (int64_t)j0 * ldc;
    tile_mma<true, false, MMA_SET, false, true, true>(G, TS, 0, nullptr, 0, 0, nb, nb, Vb, ldc, nullptr, Vb, ldc,
                                                      nullptr, len, sA, sB);
    for (int q = tid; q < TS * TS; q += kT) {
        const int a = q % TS, b = q / TS;
        T[a + b * kTld] = (a <= b && b < nb) ? G[a + b * TS] : 0.0;
    }
    __syncthreads();
    if (warp < 2) {
        double* Th = T + warp * NB * (kTld + 1);
        const int nh = min(NB, nb - warp * NB);
        for (int b = 0; b < nh; ++b) {
            const double tb = tau[j0 + warp * NB + b];
            double acc = 0.0;
            if (lane < b)
                for (int c2 = lane; c2 < b; ++c2) acc = fma(Th[lane + c2 * kTld], Th[c2 + b * kTld], acc);
            __syncwarp();
            if (lane < b) Th[lane + b * kTld] = -tb * acc;
            if (lane == b) Th[b + b * kTld] = tb;
            __syncwarp();
        }
    }
    __syncthreads();
    // W = G12 T22 (in G), then T12 = -T11 W
    for (int q = tid; q < NB * NB; q += kT) {
        const int a = q % NB, b = q / NB;
        double w = 0.0;
        for (int k = 0; k <= b; ++k) w = fma(T[a + (NB + k) * kTld], T[NB + k + (NB + b) * kTld], w);
        G[a + b * NB] = w;
    }
    __syncthreads();
    for (int q = tid; q < NB * NB; q += kT) {
        const int a = q % NB, b = q / NB;
        double w = 0.0;
        for (int k = a; k < NB; ++k) w = fma(T[a + k * kTld], G[k + b * NB], w);
        T[a + (NB + b) * kTld] = -w;
    }
    __syncthreads();
    for (int q = tid; q < TS * TS; q += kT) Tp[q] = T[q % TS + (q / TS) * kTld];
}

// X (len x nv, nv <= TS) -= V Y2 with the panel's reflectors V (nb of them, read in
// place) and Y2 (TS x nv, in shared memory with column stride kY2ld = 4 mod 16, the
// layout of a B fragment): Y2 stays where it is, each 64-row tile of V goes through
// sA once, and the next tile's V and this tile's X are on their way to registers
// while a tile is multiplied.
constexpr int kY2ld = TS + 4;
__device__ void wy_update(const double* __restrict__ Vb, int64_t ldv, int nb, double* X, int64_t ldx, int len, int nv,
                          const double* Y2, double* sA) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int wr = (warp & 3) * 16, wc = (warp >> 2) * 16;
    constexpr int kPer = TS * TS / kT;
    const int vi = tid % TS, vk = tid / TS;   // row and first reflector of this thread's loads
    double va[kPer];
    auto fetch = [&](int i0) {
        const int row = i0 + vi;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int k = vk + q * (kT / TS);
            va[q] = (k < nb && row < len) ? (row == k ? 1.0 : row > k ? Vb[row + (int64_t)k * ldv] : 0.0) : 0.0;
        }
    };
    fetch(0);
    const int ksteps = (nb + 3) >> 2;
    for (int i0 = 0; i0 < len; i0 += TS) {
        const int mr = min(TS, len - i0);
        double cv[2][2][2], acc[2][2][2];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = wr + 8 * a + g, j = wc + 8 * b + 2 * t4 + h;
                    cv[a][b][h] = (i < mr && j < nv) ? X[i0 + i + (int64_t)j * ldx] : 0.0;
                    acc[a][b][h] = 0.0;
                }
#pragma unroll
        for (int q = 0; q < kPer; ++q) sA[(vk + q * (kT / TS)) * kY2ld + vi] = va[q];
        __syncthreads();
        if (i0 + TS < len) fetch(i0 + TS);
        for (int ks = 0; ks < ksteps; ++ks) {
            const int k = ks * 4 + t4;
            const double a0 = sA[k * kY2ld + wr + g], a1 = sA[k * kY2ld + wr + 8 + g];
            const double b0 = Y2[(wc + g) * kY2ld + k], b1 = Y2[(wc + 8 + g) * kY2ld + k];
            dmma(acc[0][0][0], acc[0][0][1], a0, b0);
            dmma(acc[0][1][0], acc[0][1][1], a0, b1);
            dmma(acc[1][0][0], acc[1][0][1], a1, b0);
            dmma(acc[1][1][0], acc[1][1][1], a1, b1);
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int i = wr + 8 * a + g, j = wc + 8 * b + 2 * t4 + h;
                    if (i < mr && j < nv) X[i0 + i + (int64_t)j * ldx] = cv[a][b][h] - acc[a][b][h];
                }
        __syncthreads();
    }
}

// Q = H_0 ... H_{m-3} applied to nv <= TS vectors (X, ld m) on the FP64 tensor cores,
// a panel at a time as I - V T V^T with the panels' T from build_T: Y = V^T X,
// Y2 = T^T Y (trans: panels in order) or T Y (panels in reverse), X -= V Y2.  Y: TS x
// TS, Y2: TS x kY2ld shared.  Bound by the FP64 tensor pipe with two CTAs per SM
// (a chunk of V^T X 3.9k clocks each, 3.45k of them multiplying) and by the chain of
// chunks with one.
__device__ void wy_apply(const double* __restrict__ C, int64_t ldc, int m, const double* __restrict__ Tall, double* X,
                         int nv, bool trans, double* Y, double* Y2, double* sA, double* sB) {
    const int npan = (int)t_panels(m);
    if (nv <= 0) return;
    for (int pp = 0; pp < npan; ++pp) {
        const int pan = trans ? pp : npan - 1 - pp;
        const int j0 = pan * TS, nb = min(TS, m - 2 - j0), r0 = j0 + 1, len = m - r0;
        const double* Vb = C + r0 + (int64_t)j0 * ldc;
        const double* Tp = Tall + (int64_t)pan * TS * TS;
        tile_mma<true, false, MMA_SET, false, true, false>(Y, TS, 0, nullptr, 0, 0, nb, nv, Vb, ldc, nullptr, X + r0, m,
                                                           nullptr, len, sA, sB);
        if (trans)
            tile_mma<true, false, MMA_SET, false>(Y2, kY2ld, 0, nullptr, 0, 0, TS, nv, Tp, TS, nullptr, Y, TS, nullptr,
                                                  nb, sA, sB);
        else
            tile_mma<false, false, MMA_SET, false>(Y2, kY2ld, 0, nullptr, 0, 0, TS, nv, Tp, TS, nullptr, Y, TS, nullptr,
                                                   nb, sA, sB);
        wy_update(Vb, ldc, nb, X + r0, m, len, nv, Y2, sA);
    }
}

// X <- L^-1 X (lower = true) or X <- L^-T X (lower = false) for the nc <= TS columns of
// X (ld ldx), L lower (ld m): over 64-row blocks (from the top, or from the bottom
// for L^-T), the earlier blocks' contribution as one tile product, then the
// diagonal block's inverse (Inv: TS x TS per block) as another.  One CTA.  X is zero
// above row `top` (lower): the blocks before it are skipped.
//   With a substitution in place of the inverse, a block took 60k clocks besides its
// products of 3.7k per chunk (two CTAs per SM); the inverse takes 8k.
__device__ void trsm_cols(bool lower, const double* __restrict__ L, int m, const double* __restrict__ Inv, double* X,
                          int64_t ldx, int nc, double* sA, double* sB, int top = 0) {
    const int nrb = (m + TS - 1) / TS, q0 = top / TS, k0 = q0 * TS;
    for (int q = q0; q < nrb; ++q) {
        const int rb = lower ? q : nrb - 1 - q + q0;
        const int i0 = rb * TS, mr = min(TS, m - i0), i1 = i0 + mr;
        const double* Ib = Inv + (int64_t)rb * TS * TS;
        if (lower) {
            if (i0 > k0)
                tile_mma<false, false, MMA_SUB, false>(X, ldx, 0, nullptr, i0, 0, mr, nc, L + (int64_t)k0 * m, m, nullptr,
                                                       X + k0, ldx, nullptr, i0 - k0, sA, sB);
            tile_mma<false, false, MMA_SET, false>(X, ldx, i0, nullptr, 0, 0, mr, nc, Ib, TS, nullptr, X + i0, ldx,
                                                   nullptr, mr, sA, sB);
        } else {
            if (i1 < m)   // (L^T)[i, k] = L[k, i] for k >= i1
                tile_mma<true, false, MMA_SUB, false>(X, ldx, 0, nullptr, i0, 0, mr, nc, L + i1, m, nullptr, X + i1,
                                                      ldx, nullptr, m - i1, sA, sB);
            tile_mma<true, false, MMA_SET, false>(X, ldx, i0, nullptr, 0, 0, mr, nc, Ib, TS, nullptr, X + i0, ldx,
                                                  nullptr, mr, sA, sB);
        }
    }
}

#include "eig_dc.cuh"
#include "eig_vec.cuh"

// ---------------------------------------------------------------------------
// status[pi]: 0, the order of a non-positive pivot of S_k, or kStNoConv; a problem
// that failed is skipped by the later stages.
#include "eig_trd.cuh"
#include "eig_trdc.cuh"

// ---- gather, Cholesky and reduction: stages over the 64-row (or 64-column) blocks
// of every problem (tasks: problem, block)

// H_k, S_k (source/sm.f90:240-246) into the X and L arenas, 64 columns per CTA; of S the
// lower triangle, zeros above it.  A standard problem needs no reduction: its matrix
// goes where that leaves it.
__global__ void __launch_bounds__(kT, 2) k_eig_gather(const EigProb* __restrict__ probs,
                                                      const int2* __restrict__ tasks, const int* __restrict__ maps,
                                                      const double* __restrict__ H, const double* __restrict__ S,
                                                      double* __restrict__ Ca, double* __restrict__ Xa,
                                                      double* __restrict__ La) {
    const int2 t = tasks[blockIdx.x];
    const EigProb p = probs[t.x];
    const int m = p.m;
    const int* mp = maps + p.moff;
    double* X = p.kind == 0 ? Xa + p.aoff : Ca + p.coff;
    const int64_t ldx = p.kind == 0 ? m : p.ldc;
    double* L = La + p.aoff;
    // 64 rows x 8 columns at a time: loads of scattered elements, whose latency the eight
    // columns share (one column at a time 41 us for the 92 rows of 4 H2O)
    const int tx = threadIdx.x % TS, ty = threadIdx.x / TS;
    for (int j = t.y * TS + ty; j < min(m, (t.y + 1) * TS); j += kT / TS) {
        const int64_t gj = p.gbase + (int64_t)mp[j] * p.gld;
#pragma unroll 4
        for (int i = tx; i < m; i += TS) {
            const int64_t q = (int64_t)mp[i] + gj;
            X[i + (int64_t)j * ldx] = H[q];
            if (p.kind == 0) L[i + (int64_t)j * m] = i >= j ? S[q] : 0.0;
        }
    }
}

// Factor and inverse of one TS x TS diagonal block (its first mr rows at L, ld m; the
// rest counts as the identity), by elimination on [A | I]: thread (i, g) holds row i,
// columns g, g + 8, ... of both in registers, and a step eliminates two columns, which
// it broadcasts with the two rows of the right half through shared memory (two
// buffers, one barrier a step).
// With A = (unit lower) D (unit lower)^T: L = lower sqrt(D), L^-1 = D^-1/2 lower^-1.
// Bound by the chain of TS / 2 steps of a barrier, two divisions and the updates
// (46k clocks; with one column a step 48k).  Returns
// the first non-positive pivot's position (1-based; 0: none), the same on every thread.
__device__ int diag_factor(double* __restrict__ L, int m, int mr, double* __restrict__ Inv) {
    constexpr int NG = kT / TS, NQ = TS / NG;
    __shared__ double colb[2][2][TS], rowb[2][2][TS], piv[TS];
    const int i = threadIdx.x % TS, g = threadIdx.x / TS;
    double a[NQ], e[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int c = g + NG * q;
        a[q] = (i < mr && c <= i) ? L[i + (int64_t)c * m] : (i == c ? 1.0 : 0.0);
        e[q] = i == c ? 1.0 : 0.0;
    }
    int bad = 0;
#pragma unroll
    for (int kq = 0; kq < NQ; ++kq) {
#pragma unroll 1
        for (int kg = 0; kg < NG; kg += 2) {
            const int k = kq * NG + kg;
            double(*cb)[TS] = colb[(kg >> 1) & 1];
            double(*rb)[TS] = rowb[(kg >> 1) & 1];
            if (g == kg || g == kg + 1) cb[g - kg][i] = a[kq];
            if (i == k || i == k + 1) {
#pragma unroll
                for (int q = 0; q <= kq; ++q) rb[i - k][g + NG * q] = e[q];
            }
            __syncthreads();
            // the second column after the first one's step: pivot p1, entry y
            const double p0 = cb[0][k], p10 = cb[0][k + 1], r0 = 1.0 / p0, l = p10 * r0;
            const double p1 = fma(-l, p10, cb[1][k + 1]), r1 = 1.0 / p1;
            if (bad == 0) bad = !(p0 > 0.0) ? k + 1 : !(p1 > 0.0) ? k + 2 : 0;
            if (threadIdx.x == 0) {
                piv[k] = p0;
                piv[k + 1] = p1;
            }
            const double f0 = i > k ? cb[0][i] * r0 : 0.0;
            const double y = fma(-f0, p10, cb[1][i]);
            const double f1 = i > k + 1 ? y * r1 : 0.0, h0 = fma(-f1, l, f0);
#pragma unroll
            for (int q = 0; q <= kq; ++q) {
                const int c = g + NG * q;
                e[q] = fma(-f1, rb[1][c], fma(-h0, rb[0][c], e[q]));
            }
            if (g == kg + 1) a[kq] = y;
            else if (g > kg + 1) a[kq] = fma(-f1, cb[1][g + NG * kq], fma(-h0, cb[0][g + NG * kq], a[kq]));
#pragma unroll
            for (int q = kq + 1; q < NQ; ++q) {
                const int c = g + NG * q;
                a[q] = fma(-f1, cb[1][c], fma(-h0, cb[0][c], a[q]));
            }
        }
    }
    __syncthreads();
    if (bad) return bad;
    const double si = sqrt(piv[i]);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int c = g + NG * q;
        if (i < mr && c < mr) L[i + (int64_t)c * m] = i > c ? a[q] / sqrt(piv[c]) : i == c ? si : 0.0;
        Inv[i + c * TS] = (i < mr && c <= i) ? e[q] / si : 0.0;
    }
    return 0;
}

// Block column j of the Cholesky factor, left-looking: every 64 x 64 tile of the column
// gets the earlier columns' contribution as one product, the CTA of the diagonal tile
// goes on to factor and invert it; then the tiles below are multiplied by the
// inverse's transpose (k_chol_scale).  Two launches per block column over the whole
// batch.  One CTA (order <= 800) or cluster per problem, with 32-wide panels and
// rank-32 updates, took 2.3 ms against 0.6 for 32 H2O and 28 ms against 10.2
// for 512-H2O clusters (orders to 2773).
__global__ void __launch_bounds__(kT, 2) k_chol_column(const EigProb* __restrict__ probs,
                                                       const int2* __restrict__ tasks, int j, double* __restrict__ La,
                                                       double* __restrict__ Ia, int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    const int2 t = tasks[blockIdx.x];
    if (t.y < j || status[t.x] != kStOk) return;
    const EigProb p = probs[t.x];
    const int m = p.m, i0 = t.y * TS, j0 = j * TS, mr = min(TS, m - i0), nc = min(TS, m - j0);
    double* L = La + p.aoff;
    if (j > 0)
        tile_mma<false, true, MMA_SUB, false>(L, m, 0, nullptr, i0, j0, mr, nc, L, m, nullptr, L, m, nullptr, j0, sA,
                                              sA + kStageOp);
    if (t.y == j) {
        const int f = diag_factor(L + i0 + (int64_t)i0 * m, m, mr, Ia + p.ioff + (int64_t)j * TS * TS);
        if (f != 0 && threadIdx.x == 0) status[t.x] = i0 + f;
    }
}

__global__ void __launch_bounds__(kT, 2) k_chol_scale(const EigProb* __restrict__ probs,
                                                      const int2* __restrict__ tasks, int j, double* __restrict__ La,
                                                      const double* __restrict__ Ia, const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    const int2 t = tasks[blockIdx.x];
    if (t.y <= j || status[t.x] != kStOk) return;
    const EigProb p = probs[t.x];
    const int m = p.m, i0 = t.y * TS;
    double* Lj = La + p.aoff + (int64_t)j * TS * m;
    tile_mma<false, true, MMA_SET, false>(Lj, m, 0, nullptr, i0, 0, min(TS, m - i0), TS, Lj, m, nullptr,
                                          Ia + p.ioff + (int64_t)j * TS * TS, TS, nullptr, TS, sA, sA + kStageOp);
}

// X <- L^-1 X on one 64-column block of X per CTA.
__global__ void __launch_bounds__(kT, 2) k_eig_trsm(const EigProb* __restrict__ probs, const int2* __restrict__ tasks,
                                                    const double* __restrict__ La, const double* __restrict__ Ia,
                                                    double* __restrict__ Xa, const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double* sA = reinterpret_cast<double*>(smraw);
    const int2 t = tasks[blockIdx.x];
    if (status[t.x] != kStOk) return;
    const EigProb p = probs[t.x];
    const int m = p.m, c0 = t.y * TS;
    trsm_cols(true, La + p.aoff, m, Ia + p.ioff, Xa + p.aoff + (int64_t)c0 * m, m, min(TS, m - c0), sA, sA + kStageOp);
}

// Row block i of the lower triangle of A = X L^-T into the C arena (zeros above it), one
// per CTA, the last and longest rows of a problem first: block column j as X_ij less
// one product with the row's earlier blocks, times the transpose of the diagonal block's
// inverse.  A third of the products of a solve over whole columns, and no transposed
// copy (14.8 -> 5.7 ms for 512-H2O clusters).
__global__ void __launch_bounds__(kT, 2) k_eig_rsolve(const EigProb* __restrict__ probs,
                                                      const int2* __restrict__ tasks, const double* __restrict__ La,
                                                      const double* __restrict__ Ia, double* __restrict__ Xa,
                                                      double* __restrict__ Ca, const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double *sA = reinterpret_cast<double*>(smraw), *sB = sA + kStageOp;
    const int2 t = tasks[blockIdx.x];
    if (status[t.x] != kStOk) return;
    const EigProb p = probs[t.x];
    const int m = p.m, i = (m + TS - 1) / TS - 1 - t.y, i0 = i * TS, mr = min(TS, m - i0);
    const double* L = La + p.aoff;
    double *X = Xa + p.aoff, *C = Ca + p.coff;
    for (int j = 0; j <= i; ++j) {
        const int j0 = j * TS, nc = min(TS, m - j0);
        if (j > 0)
            tile_mma<false, true, MMA_SUB, false>(X, m, 0, nullptr, i0, j0, mr, nc, C, p.ldc, nullptr, L, m, nullptr, j0,
                                                  sA, sB);
        tile_mma<false, true, MMA_SET, false>(C + (int64_t)j0 * p.ldc, p.ldc, 0, nullptr, i0, 0, mr, nc,
                                              X + (int64_t)j0 * m, m, nullptr, Ia + p.ioff + (int64_t)j * TS * TS, TS,
                                              nullptr, nc, sA, sB);
    }
    for (int c = i0 + mr + threadIdx.x / TS; c < m; c += kT / TS)
        if (threadIdx.x % TS < mr) C[i0 + threadIdx.x % TS + (int64_t)c * p.ldc] = 0.0;
}

// Tridiagonalisation, one problem per CTA.
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) k_eig_trd(const EigProb* __restrict__ probs,
                                                          const int* __restrict__ order, double* __restrict__ Ca,
                                                          double* __restrict__ Da, double* __restrict__ Ea,
                                                          double* __restrict__ Ta, int cap,
                                                          const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int pi = order[blockIdx.x];
    if (status[pi] != kStOk) return;
    stage_trd<NT>(probs[pi], Ca, Da, Ea, Ta, reinterpret_cast<double*>(smraw), cap);
}

// ===========================================================================
// Tridiagonalisation of orders that no cluster's shared memory holds, and of single
// dense problems above kGridMin: G CTAs per problem, a thread-block cluster or a
// cooperative grid, one barrier between dependent steps and the intermediates in
// global memory (L2-resident for the vectors and panels).
//   tridiag.     blocked Householder with lazy updates (LAPACK's latrd
//                scheme): per column the panel's earlier reflectors update that
//                column, the reflector is formed, and y = A v runs over the
//                lower 64 x 64 tiles of the not yet updated trailing block (each
//                tile read once for both its row and its column contribution),
//                corrected by V (W^T v) + W (V^T v); w = tau (y - tau/2 (y.v) v);
//                after 32 columns the trailing block gets A -= V W^T + W V^T.
//                Rows are owned in 32-row chunks, partial sums go through
//                per-CTA slots summed in CTA order, so results do not depend on
//                scheduling.  Two barriers per column.
// ===========================================================================
constexpr int kLargeMax = kEigLargeMax;   // largest order it takes (its vectors live in shared memory)
constexpr int kRedW = 2 * NB + 4;         // per-CTA partial sums of the tridiagonalisation
constexpr int kRedVAv = 2 * NB + 1;       // slot of the partial v^T A v
// Software barrier over the CTAs of a cooperative launch (all resident):
// bar[0] counts arrivals, bar[1] is the generation.  The wait is bounded: after
// kGridSpin polls the CTA records the failure in *err and goes on, and every
// later barrier returns at once, so a kernel whose barrier gave up still ends
// (its results are then discarded by the host, which reports the timeout).
constexpr long long kGridSpin = 1ll << 24;

__device__ void grid_barrier(unsigned* bar, int nblocks, int* err) {
    __syncthreads();
    if (threadIdx.x == 0 && *(volatile int*)err == 0) {
        volatile unsigned* vb = bar;
        const unsigned gen = vb[1];
        __threadfence();
        if (atomicAdd(&bar[0], 1u) == (unsigned)nblocks - 1) {
            atomicExch(&bar[0], 0u);
            __threadfence();
            atomicAdd(&bar[1], 1u);
        } else {
            long long it = 0;
            while (vb[1] == gen) {
                if (++it > kGridSpin) {
                    atomicExch(err, 1);
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
    }
    __syncthreads();
}

// The CTAs that solve one problem together: a thread-block cluster (bar null,
// hardware barrier) or the whole grid of a cooperative launch (software barrier).
struct Grp {
    int rank, size;
    unsigned* bar;
    int* err;
    __device__ __forceinline__ void sync() const {
        if (!bar) cg::this_cluster().sync();
        else grid_barrier(bar, size, err);
    }
};

// Per-problem scratch of a cluster solve (offsets in doubles from p.xoff).
struct LgLayout {
    int64_t rowp, colp, red, V, W, total;
};
constexpr int kSegW = 64;    // columns of one A v work unit of the tridiagonalisation
constexpr int kAvGrp = 8;    // columns whose loads are issued together in the A v units
__host__ __device__ inline LgLayout lg_layout(int m, int G) {
    LgLayout L;
    int64_t o = 0;
    L.rowp = o;   // row sums of the A v units: [segment][m]
    o += (int64_t)((m + kSegW - 1) / kSegW + 1) * m;
    L.colp = o;   // column sums of the A v units: [64-row block][m]
    o += (int64_t)((m + TS - 1) / TS) * m;
    L.red = o;
    o += (int64_t)G * kRedW;
    L.V = o;
    o += (int64_t)m * NB;
    L.W = o;
    o += (int64_t)m * NB;
    L.total = (o + 1) & ~int64_t(1);
    return L;
}

struct LgSmem {
    double *sA, *sB;           // tile staging
    double *v, *y;             // tridiagonalisation: reflector and updated column (M each)
    double *pw, *pv, *wtv, *vtv, *wj, *vj;   // NB each
    double* red;               // kT / 32 + 2
    double* dsc;               // scalars (8)
};
__host__ __device__ constexpr size_t lg_smem_bytes(int M) {
    return sizeof(double) * (2 * kStageOp + 2 * (size_t)M + 6 * NB + kT / 32 + 2 + 8);
}
static_assert(lg_smem_bytes(kLargeMax) <= 232448, "cluster solver shared memory within the per-CTA limit");
__device__ LgSmem lg_smem(unsigned char* base, int M) {
    LgSmem s;
    double* d = reinterpret_cast<double*>(base);
    s.sA = d;
    s.sB = d + kStageOp;
    s.v = d + 2 * kStageOp;
    s.y = s.v + M;
    s.pw = s.y + M;
    s.pv = s.pw + NB;
    s.wtv = s.pv + NB;
    s.vtv = s.wtv + NB;
    s.wj = s.vtv + NB;
    s.vj = s.wj + NB;
    s.red = s.vj + NB;
    s.dsc = s.red + kT / 32 + 2;
    return s;
}

// Lower-triangle tile index -> (row block, column block), rb >= cb.
__device__ __forceinline__ void tri_decode(int64_t idx, int& rb, int& cb) {
    int r = (int)((sqrt(8.0 * (double)idx + 1.0) - 1.0) * 0.5);
    while ((int64_t)(r + 1) * (r + 2) / 2 <= idx) ++r;
    while ((int64_t)r * (r + 1) / 2 > idx) --r;
    rb = r;
    cb = (int)(idx - (int64_t)r * (r + 1) / 2);
}

// Units of the A v pass for the trailing block from row/column s: tile rows
// I in [s/64, nT), each cut into kSegW-column segments from column 64 (s/64).
__device__ __forceinline__ int av_nseg(int I, int cstart) {
    return ((I + 1) * TS - cstart + kSegW - 1) / kSegW;
}

// w of column jp of the panel (the column before j) on this CTA's rows, with the
// reflector stored into A's column j-1; w_j itself goes to sh.wj[jp], computed
// by the last warp beside the row loop.  The caller synchronises the CTA.
__device__ void lg_finish_w(const Grp& g, int m, int j, int jp, double* __restrict__ A, int64_t lda, double* __restrict__ V,
                            double* __restrict__ W, const double* __restrict__ rowp,
                            const double* __restrict__ colp, const double* __restrict__ red, const LgSmem& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double tp = sh.dsc[0];
    double vAv = 0.0;
    for (int q = 0; q < g.size; ++q) vAv += red[q * kRedW + kRedVAv];
    double vw = 0.0;
    for (int q = 0; q < jp; ++q) vw = fma(sh.vtv[q], sh.wtv[q], vw);
    const double ytv = vAv - 2.0 * vw;
    const double hc = 0.5 * tp * ytv;
    const int cstart = (j / TS) * TS, nT = (m + TS - 1) / TS;
    auto w_at = [&](int r) {
        // y_r = its row sums over the segments of its tile row, then its column
        // sums over the tile rows at and below its own, in that fixed order
        const int Ir = r / TS;
        double y = 0.0;
        const int ns = av_nseg(Ir, cstart);
        for (int q = 0; q < ns; ++q) y += rowp[(int64_t)q * m + r];
        for (int I = Ir; I < nT; ++I) y += colp[(int64_t)I * m + r];
        for (int q = 0; q < jp; ++q) y -= V[r + (int64_t)q * m] * sh.wtv[q] + W[r + (int64_t)q * m] * sh.vtv[q];
        return tp * (y - hc * sh.v[r]);
    };
    if (tid == kT - 32 && j < m) sh.wj[jp] = w_at(j);
    for (int ch = g.rank + g.size * warp; ch * 32 < m; ch += g.size * (kT / 32)) {
        const int r = ch * 32 + lane;
        if (r >= j && r < m) {
            W[r + (int64_t)jp * m] = w_at(r);
            if (r >= j + 1) A[r + (int64_t)(j - 1) * lda] = sh.v[r];
        }
    }
}

__device__ void lg_sytrd(const Grp& g, const EigProb& p, double* __restrict__ Ca, double* __restrict__ Da,
                         double* __restrict__ Ea, double* __restrict__ Ta, double* __restrict__ X, const LgSmem& sh) {
    const int m = p.m, G = g.size, rk = g.rank;
    double* A = Ca + p.coff;
    const int64_t lda = p.ldc;
    double* d = Da + p.voff;
    double* e = Ea + p.voff;
    double* tau = Ta + p.voff;
    const LgLayout lay = lg_layout(m, G);
    double* rowp = X + lay.rowp;
    double* colp = X + lay.colp;
    double* red = X + lay.red;
    double* V = X + lay.V;
    double* W = X + lay.W;
    double* v = sh.v;
    double* yl = sh.y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nT = (m + TS - 1) / TS;
    for (int j0 = 0; j0 < m - 1; j0 += NB) {
        const int nb = min(NB, m - 1 - j0);
        for (int jj = 0; jj < nb; ++jj) {
            const int j = j0 + jj;
            // ---- phase A: finish w of the previous column, update column j on own rows
            // (row j of the panel's V and earlier W columns were written before the
            // last cluster barrier; w_j of the previous column comes from lg_finish_w)
            if (tid < jj) {
                if (tid < jj - 1) sh.wj[tid] = W[j + (int64_t)tid * m];
                sh.vj[tid] = V[j + (int64_t)tid * m];
            }
            if (jj > 0) lg_finish_w(g, m, j, jj - 1, A, lda, V, W, rowp, colp, red, sh);
            __syncthreads();
            for (int ch = rk + G * warp; ch * 32 < m; ch += G * (kT / 32)) {
                const int r = ch * 32 + lane;
                if (r >= j && r < m) {
                    double a = A[r + (int64_t)j * lda];
                    for (int q = 0; q < jj; ++q)
                        a -= V[r + (int64_t)q * m] * sh.wj[q] + W[r + (int64_t)q * m] * sh.vj[q];
                    A[r + (int64_t)j * lda] = a;
                    yl[r] = a;
                }
            }
            __syncthreads();
            {
                double part = 0.0;
                for (int ch = rk + G * warp; ch * 32 < m; ch += G * (kT / 32)) {
                    const int r = ch * 32 + lane;
                    if (r >= j + 2 && r < m) part = fma(yl[r], yl[r], part);
                }
                part = cta_sum(part, sh.red);
                if (tid == 0) red[rk * kRedW + 0] = part;
            }
            for (int q = warp; q < 2 * jj; q += kT / 32) {
                const double* col = (q < jj) ? W + (int64_t)q * m : V + (int64_t)(q - jj) * m;
                double part = 0.0;
                for (int ch = rk; ch * 32 < m; ch += G) {
                    const int r = ch * 32 + lane;
                    if (r >= j + 2 && r < m) part = fma(col[r], yl[r], part);
                }
                part = warp_sum(part);
                if (lane == 0) red[rk * kRedW + ((q < jj) ? 1 + q : 1 + NB + (q - jj))] = part;
            }
            g.sync();
            // ---- phase B: reflector, then y = A v over the trailing lower tiles
            // (column j below the subdiagonal is read into v while the scale is
            // formed, and scaled in shared memory after the barrier)
            double wj1 = 0.0, vj1 = 0.0;
            if (tid < jj) {
                double a = 0.0, b = 0.0;
                for (int q = 0; q < G; ++q) {
                    a += red[q * kRedW + 1 + tid];
                    b += red[q * kRedW + 1 + NB + tid];
                }
                sh.pw[tid] = a;
                sh.pv[tid] = b;
                wj1 = W[(j + 1) + (int64_t)tid * m];
                vj1 = V[(j + 1) + (int64_t)tid * m];
            }
            for (int r = j + 2 + tid; r < m; r += kT) v[r] = A[r + (int64_t)j * lda];
            if (tid == 32) {
                double xn2 = 0.0;
                for (int q = 0; q < G; ++q) xn2 += red[q * kRedW + 0];
                const double alpha = A[(j + 1) + (int64_t)j * lda];
                const double dj = A[j + (int64_t)j * lda];
                double t, beta;
                if (xn2 == 0.0) {
                    t = 0.0;
                    beta = alpha;
                } else {
                    beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
                    t = (beta - alpha) / beta;
                }
                sh.dsc[0] = t;
                sh.dsc[1] = (t == 0.0) ? 0.0 : 1.0 / (alpha - beta);
                if (rk == 0) {
                    d[j] = dj;
                    e[j] = beta;
                    tau[j] = t;
                }
            }
            __syncthreads();
            const double sc = sh.dsc[1];
            for (int r = tid; r < m; r += kT) {
                double vr;
                if (r <= j) vr = 0.0;
                else if (r == j + 1) vr = 1.0;
                else vr = (sc == 0.0) ? 0.0 : v[r] * sc;
                v[r] = vr;
            }
            if (tid < jj) {
                sh.wtv[tid] = wj1 + sc * sh.pw[tid];
                sh.vtv[tid] = vj1 + sc * sh.pv[tid];
            }
            const int s = j + 1;
            for (int r = s + tid; r < m; r += kT) yl[r] = 0.0;
            __syncthreads();
            for (int ch = rk + G * warp; ch * 32 < m; ch += G * (kT / 32)) {
                const int r = ch * 32 + lane;
                if (r >= s && r < m) V[r + (int64_t)jj * m] = v[r];
            }
            // A v over the trailing lower triangle, one pass: every warp streams
            // its own units (64 rows x kSegW columns of one tile row) without a
            // barrier, lane holding rows I*64 + lane and + 32: the row sums stay
            // in registers for the unit, each column's sum is a warp reduction;
            // both go to their own slots (rowp[segment][r], colp[tile row][c]),
            // summed in a fixed order when w is formed.  v^T A v comes from the
            // same sums.  Warps are numbered across the CTAs (warp-major), so
            // consecutive units land on different SMs: with fewer units than
            // warps (small orders) every SM's L2 bandwidth still takes part.
            {
                const int I0 = s / TS, cstart = I0 * TS;
                const int gw = warp * G + rk, nw = G * (kT / 32);
                double vav = 0.0;
                int I = I0, ubase = 0;
                for (int u = gw;; u += nw) {
                    while (I < nT && u >= ubase + av_nseg(I, cstart)) {
                        ubase += av_nseg(I, cstart);
                        ++I;
                    }
                    if (I >= nT) break;
                    const int seg = u - ubase;
                    const int c_lo = cstart + seg * kSegW;
                    const int c_hi = min(min(c_lo + kSegW, (I + 1) * TS), m);
                    const int r0 = I * TS + lane, r1 = r0 + 32;
                    const double v0 = (r0 < m) ? v[r0] : 0.0, v1 = (r1 < m) ? v[r1] : 0.0;
                    const double* A0 = A + r0;
                    const double* A1 = A + r1;
                    double rp0 = 0.0, rp1 = 0.0;
                    for (int cb = c_lo; cb < c_hi; cb += 32) {
                        double mycol = 0.0;
#pragma unroll 1
                        for (int g8 = 0; g8 < 32; g8 += kAvGrp) {
                            double a0[kAvGrp], a1[kAvGrp];
#pragma unroll
                            for (int u8 = 0; u8 < kAvGrp; ++u8) {
                                const int c = cb + g8 + u8;
                                const bool cok = c < c_hi && c >= s;
                                a0[u8] = (cok && r0 < m && c <= r0) ? A0[(int64_t)c * lda] : 0.0;
                                a1[u8] = (cok && r1 < m && c <= r1) ? A1[(int64_t)c * lda] : 0.0;
                            }
#pragma unroll
                            for (int u8 = 0; u8 < kAvGrp; ++u8) {
                                const int c = cb + g8 + u8;
                                const double vc = (c < c_hi) ? v[c] : 0.0;
                                rp0 = fma(a0[u8], vc, rp0);
                                rp1 = fma(a1[u8], vc, rp1);
                                double cp = ((c < r0) ? a0[u8] * v0 : 0.0) + ((c < r1) ? a1[u8] * v1 : 0.0);
                                cp = warp_sum(cp);
                                if (lane == g8 + u8) mycol = cp;
                            }
                        }
                        const int c = cb + lane;
                        if (c < c_hi) {
                            colp[(int64_t)I * m + c] = mycol;
                            vav = fma(v[c], mycol, vav);
                        }
                    }
                    if (r0 < m) rowp[(int64_t)seg * m + r0] = rp0;
                    if (r1 < m) rowp[(int64_t)seg * m + r1] = rp1;
                    vav = fma(v0, rp0, fma(v1, rp1, vav));
                }
                const double part = cta_sum(vav, sh.red);
                if (tid == 0) red[rk * kRedW + kRedVAv] = part;
            }
            g.sync();
        }
        // ---- panel end: w of the last column, then the trailing block
        const int j1 = j0 + nb;
        lg_finish_w(g, m, j1, nb - 1, A, lda, V, W, rowp, colp, red, sh);
        g.sync();
        if (j1 < m) {
            const int nt = (m - j1 + TS - 1) / TS;
            const int64_t ntile = (int64_t)nt * (nt + 1) / 2;
            for (int64_t idx = rk; idx < ntile; idx += G) {
                int rb, cb;
                tri_decode(idx, rb, cb);
                const int r0 = j1 + rb * TS, c0 = j1 + cb * TS;
                const int mr = min(TS, m - r0), nc = min(TS, m - c0);
                tile_update<true, true>(A, (int)lda, r0, c0, mr, nc, V, m, W, m, nb, sh.sA, sh.sB);
                tile_update<true, true>(A, (int)lda, r0, c0, mr, nc, W, m, V, m, nb, sh.sA, sh.sB);
            }
        }
        g.sync();
    }
    if (rk == 0 && tid == 0) {
        d[m - 1] = A[(m - 1) + (int64_t)(m - 1) * lda];
        tau[m - 1] = 0.0;
    }
}

// A cluster per problem (order[]: largest first), or with bar non-null one problem on the
// whole cooperative grid.
__device__ __forceinline__ Grp lg_group(unsigned* bar, int* err) {
    if (bar) return Grp{(int)blockIdx.x, (int)gridDim.x, bar, err};
    cg::cluster_group cl = cg::this_cluster();
    return Grp{(int)cl.block_rank(), (int)cl.num_blocks(), nullptr, nullptr};
}
__global__ void __launch_bounds__(kT, 1) k_lg_trd(const EigProb* __restrict__ probs, const int* __restrict__ order,
                                                  int M, double* __restrict__ Ca, double* __restrict__ Da,
                                                  double* __restrict__ Ea, double* __restrict__ Ta,
                                                  double* __restrict__ Xa, const int* __restrict__ status,
                                                  unsigned* __restrict__ bar, int* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const LgSmem sh = lg_smem(smraw, M);
    const Grp g = lg_group(bar, err);
    const int pi = order[bar ? 0 : blockIdx.x / g.size];
    if (status[pi] != kStOk) return;
    const EigProb p = probs[pi];
    lg_sytrd(g, p, Ca, Da, Ea, Ta, Xa + p.xoff, sh);
}

__global__ void __launch_bounds__(kT, 1) k_trd_cluster(const EigProb* __restrict__ probs,
                                                       const int* __restrict__ order, double* __restrict__ Ca,
                                                       double* __restrict__ Da, double* __restrict__ Ea,
                                                       double* __restrict__ Ta, double* __restrict__ Xa, int cap,
                                                       const int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int pi = order[blockIdx.x / cg::this_cluster().num_blocks()];
    if (status[pi] != kStOk) return;
    const EigProb p = probs[pi];
    stage_trd_cluster(p, Ca, Da, Ea, Ta, Xa + p.xoff, reinterpret_cast<double*>(smraw), cap);
}

// ---- inverse of a lower triangle, in place, and the products with it (of the strict
// upper triangle the 64 x 64 diagonal blocks' parts are zeroed, the rest is not touched)

// Inverse of one TS x TS diagonal block (mr rows of it are L's), by elimination on the
// identity as in diag_factor.
__global__ void __launch_bounds__(kT, 1) k_tri_diag(int64_t n, int64_t ld, double* __restrict__ A) {
    constexpr int NG = kT / TS, NQ = TS / NG;
    __shared__ double sL[TS * (TS + 1)], rowb[2][TS];
    const int i = threadIdx.x % TS, g = threadIdx.x / TS;
    const int64_t i0 = (int64_t)blockIdx.x * TS;
    const int mr = (int)min((int64_t)TS, n - i0);
    double* L = A + i0 + i0 * ld;
    double e[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int c = g + NG * q;
        sL[i + c * (TS + 1)] = (i < mr && c <= i) ? L[i + c * ld] : (i == c ? 1.0 : 0.0);
        e[q] = i == c ? 1.0 : 0.0;
    }
    __syncthreads();
    const double dinv = 1.0 / sL[i + i * (TS + 1)];
    for (int k = 0; k < TS; ++k) {
        double* rb = rowb[k & 1];
        if (i == k) {
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                e[q] *= dinv;
                rb[g + NG * q] = e[q];
            }
        }
        __syncthreads();
        const double f = i > k ? sL[i + k * (TS + 1)] : 0.0;
#pragma unroll
        for (int q = 0; q < NQ; ++q) e[q] = fma(-f, rb[g + NG * q], e[q]);
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int c = g + NG * q;
        if (i < mr && c < mr) L[i + c * ld] = c <= i ? e[q] : 0.0;
    }
}

// One level: the off-diagonal blocks [r1, r1 + h) x [r1 - h, r1) (r1 = h, 3h, 5h, ...)
// between inverted diagonal blocks.  FIRST: W = -L21 L11^-1 (nr x h per block in Wa, nr = h
// but for a short last block); then L21 <- L22^-1 W.  One 64 x 64 tile per CTA, the zero K blocks of the triangles
// skipped, the longest K ranges first.
template <bool FIRST>
__global__ void __launch_bounds__(kT, 2) k_tri_level(int64_t n, int64_t ld, int h, double* __restrict__ A,
                                                     double* __restrict__ Wa) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double *sA = reinterpret_cast<double*>(smraw), *sB = sA + kStageOp;
    const int rt = FIRST ? blockIdx.y : gridDim.y - 1 - blockIdx.y, ct = blockIdx.x;
    const int64_t c1 = (int64_t)2 * h * blockIdx.z, r1 = c1 + h;   // the block's columns and rows
    const int nr = (int)min((int64_t)h, n - r1);
    if (rt * TS >= nr) return;
    const int r0 = rt * TS, c0 = ct * TS, mr = min(TS, nr - r0);
    double* W = Wa + (int64_t)blockIdx.z * h * h;
    double* L21 = A + r1 + c1 * ld;
    if (FIRST)
        tile_mma<false, false, MMA_NEG, false>(W, nr, 0, nullptr, r0, c0, mr, TS, L21 + c0 * ld, ld, nullptr,
                                               A + c1 + c0 + c1 * ld, ld, nullptr, h - c0, sA, sB);
    else
        tile_mma<false, false, MMA_SET, false>(L21, ld, 0, nullptr, r0, c0, mr, TS, A + r1 + r1 * ld, ld, nullptr, W, nr,
                                               nullptr, r0 + mr, sA, sB);
}

// Products with Li = L^-1 (lower, from tri_inverse; n x n, ld n), one 64 x 64 tile of the
// result per CTA, only the K range where Li is not zero, the longest ranges first:
//   TRI_LH   C = Li B                     TRI_XL   C = B Li
//   TRI_TLT  C = Li B^T, upper tiles      TRI_LTT  C = B^T Li, upper tiles
enum { TRI_LH, TRI_TLT, TRI_XL, TRI_LTT };
template <int OP>
__global__ void __launch_bounds__(kT, 2) k_tri_product(int64_t n, const double* __restrict__ Li,
                                                       const double* __restrict__ B, double* __restrict__ C) {
    extern __shared__ __align__(16) unsigned char smraw[];
    double *sA = reinterpret_cast<double*>(smraw), *sB = sA + kStageOp;
    const int nb = gridDim.x, ld = (int)n;
    const int x = blockIdx.x, y = blockIdx.y;
    if (OP == TRI_LH) {   // rows r: K up to r
        const int rt = nb - 1 - y, r0 = rt * TS, c0 = x * TS, mr = min(TS, ld - r0);
        tile_mma<false, false, MMA_SET, false>(C, n, 0, nullptr, r0, c0, mr, min(TS, ld - c0), Li, n, nullptr, B, n,
                                               nullptr, r0 + mr, sA, sB);
    } else if (OP == TRI_TLT) {   // rows r <= columns c: K up to r
        const int r0 = (nb - 1 - y) * TS, c0 = x * TS, mr = min(TS, ld - r0);
        if (c0 < r0) return;
        tile_mma<false, true, MMA_SET, false>(C, n, 0, nullptr, r0, c0, mr, min(TS, ld - c0), Li, n, nullptr, B, n,
                                              nullptr, r0 + mr, sA, sB);
    } else if (OP == TRI_XL) {   // columns c: K from c
        const int r0 = x * TS, c0 = y * TS;
        tile_mma<false, false, MMA_SET, false>(C, n, 0, nullptr, r0, c0, min(TS, ld - r0), min(TS, ld - c0),
                                               B + (int64_t)c0 * n, n, nullptr, Li + c0, n, nullptr, ld - c0, sA, sB);
    } else {   // rows r <= columns c: K from c
        const int c0 = y * TS, r0 = x * TS;
        if (r0 > c0) return;
        tile_mma<true, false, MMA_SET, false>(C, n, 0, nullptr, r0, c0, min(TS, ld - r0), min(TS, ld - c0), B + c0, n,
                                              nullptr, Li + c0, n, nullptr, ld - c0, sA, sB);
    }
}

}  // namespace

// Streams and events of a context's eigensolver calls: launches of one stage with
// different groups run side by side (side), a whole batch beside the call's stream (base).
struct EigStreams {
    static constexpr int kPerBatch = 6;            // a batch's side streams at most
    static constexpr int kSide = 2 * kPerBatch;    // of a batch on the call's stream, and of one on base
    cudaStream_t side[kSide] = {}, base = nullptr;
    cudaEvent_t fork[2] = {}, join[kSide] = {}, start = nullptr, done[kEigSlots] = {};
    EigStreams() {
        for (cudaStream_t& s : side) PTB_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        PTB_CUDA(cudaStreamCreateWithFlags(&base, cudaStreamNonBlocking));
        for (cudaEvent_t& e : join) PTB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        for (cudaEvent_t* e : {&fork[0], &fork[1], &start})
            PTB_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
        for (cudaEvent_t& e : done) PTB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    ~EigStreams() {
        for (cudaEvent_t e : join)
            if (e) cudaEventDestroy(e);
        for (cudaEvent_t e : {fork[0], fork[1], start})
            if (e) cudaEventDestroy(e);
        for (cudaEvent_t e : done)
            if (e) cudaEventDestroy(e);
        for (cudaStream_t s : side)
            if (s) cudaStreamDestroy(s);
        if (base) cudaStreamDestroy(base);
    }
};

// A failing problem and its status word (0: none).
struct EigFault {
    int k = 0, status = 0;
    void merge(const EigFault& o) {   // a non-positive pivot goes before a leaf, then the lower problem
        if (o.status == 0) return;
        const bool earlier = (o.status > 0) != (status > 0) ? o.status > 0 : o.k < k;
        if (status == 0 || earlier) *this = o;
    }
};

struct EigBatch {
    struct Seg {   // a run of a task list
        size_t off = 0;
        unsigned n = 0;
    };
    struct Level {   // one level of the divide and conquer
        int m0 = 0, nm = 0;
        Seg permute, elems, product;
    };
    struct Trd {   // problems tridiagonalised by groups of the same kind: order[off, off + n)
        int G = 0;        // CTAs per problem; 0: k_lg_trd
        int nt = 512;     // threads per CTA (G == 1)
        int off = 0, n = 0, cap = 0;
    };
    int nprob = 0;
    int G = 1;                    // CTAs per problem of k_lg_trd
    int nlarge = 0;
    bool grid = false;            // one problem on a cooperative grid
    std::vector<Trd> trd;
    std::vector<EigProb> hp;
    std::vector<int> order;       // by tridiagonalisation group, largest first in each
    std::vector<int2> lists;
    std::vector<DcMerge> merges;
    std::vector<Level> levels;
    bool timed = false;   // stage times wanted (print level 2, PTBGPU_EIG_STAGES)
    std::vector<std::pair<const char*, cudaEvent_t>> marks;   // what ended, and when
    template <class F>
    void stage_times(F&& f) const {   // of a batch that has ended
        for (size_t i = 1; i < marks.size(); ++i) {
            float ms = 0.f;
            PTB_CUDA(cudaEventElapsedTime(&ms, marks[i - 1].second, marks[i].second));
            f(marks[i].first, (double)ms);
        }
    }
    std::vector<unsigned> deep;   // tasks of `blocks` that block column j of the Cholesky factor launches
    Seg blocks, leaves, panels, rows, rq, back, density, fblocks, frq, fcols;
    WorkBuf probs, order_d, lists_d, merges_d, cnt, dc, Ca, La, Za, Qa, Va, Da, Ea, Ta, Ba, Xa, Ka, Ia, status;
    DcArr S{};
    double* Z = nullptr;          // the Z arena (Za, or the caller's array)
    int prl = 0;
    std::shared_ptr<EigStreams> st;
    bool async = false;           // launched on st->base
    int slot = 0;                 // whose done event it records there
    ~EigBatch() {
        // the arrays go back to the context's pool: nothing on the side streams may
        // still use them (work on the context's stream is ordered before their next use)
        if (st) {
            for (cudaStream_t x : st->side) cudaStreamSynchronize(x);
            cudaStreamSynchronize(st->base);
        }
    }
    const int2* list(const Seg& g) const { return lists_d.as<int2>() + g.off; }
};

namespace {

template <class K>
void smem_attr(K kern, size_t bytes) {
    PTB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

void eig_setup_attrs() {
    static const bool done = [] {
        smem_attr(k_chol_column, kTileSmem);
        smem_attr(k_tri_level<true>, kTileSmem);
        smem_attr(k_tri_level<false>, kTileSmem);
        smem_attr(k_tri_product<TRI_LH>, kTileSmem);
        smem_attr(k_tri_product<TRI_TLT>, kTileSmem);
        smem_attr(k_tri_product<TRI_XL>, kTileSmem);
        smem_attr(k_tri_product<TRI_LTT>, kTileSmem);
        smem_attr(k_chol_scale, kTileSmem);
        smem_attr(k_eig_rsolve, kTileSmem);
        smem_attr(k_eig_trsm, kTileSmem);
        smem_attr(k_eig_trd<512>, 8 * trd_cap(kTrdMax512, 512));
        smem_attr(k_eig_trd<256>, 8 * trd_cap(kTrdMax256, 256));
        smem_attr(k_lg_trd, lg_smem_bytes(kLargeMax));
        smem_attr(k_trd_cluster, kTrdCaps[3] - 1024);
        PTB_CUDA(cudaFuncSetAttribute(k_trd_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        smem_attr(k_dc_product, kTileSmem);
        smem_attr(k_vec_panels, kWySmem);
        smem_attr(k_vec_rq, kTileSmem);
        smem_attr(k_vec_rv, kTileSmem);
        smem_attr(k_fin_vw, kTileSmem);
        smem_attr(k_fin_qw, kTileSmem);
        smem_attr(k_vec_density, kTileSmem);
        smem_attr(k_vec_rows, kChainSmem);
        smem_attr(k_vec_back, kChainSmem);
        smem_attr(k_fin_cols, kChainSmem);
        PTB_CUDA(cudaFuncSetAttribute(k_lg_trd, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        return true;
    }();
    (void)done;
}

// Clusters of G CTAs of the cluster solver that fit on the device at once.
int eig_active_clusters(int G) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = G;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(G * 64);
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = lg_smem_bytes(kLargeMax);
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int ncl = 0;
    if (cudaOccupancyMaxActiveClusters(&ncl, (void*)k_lg_trd, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return ncl;
}

int eig_active_cached(ptbgpu_ctx* c, int G) {
    static int active[64][5] = {};   // known + 1
    int& a = active[c->device & 63][G == 16 ? 4 : G == 8 ? 3 : G == 4 ? 2 : G == 2 ? 1 : 0];
    if (a == 0) a = eig_active_clusters(G) + 1;
    return a - 1;
}

// CTAs of the cluster tridiagonalisation for orders beyond the shared-memory one: 16
// for one problem, else 8.  PTBGPU_EIG_CLUSTER = 1, 2, 4, 8 or 16 sets them, and those
// of every order above kEigBatchMax.
int eig_cluster_forced() {
    const char* e = getenv("PTBGPU_EIG_CLUSTER");
    const int v = e ? atoi(e) : 0;
    return v == 1 || v == 2 || v == 4 || v == 8 || v == 16 ? v : 0;
}
int eig_cluster_size(ptbgpu_ctx* c, int nlarge) {
    if (const int v = eig_cluster_forced()) return v;
    for (int G : {16, 8, 4, 2})
        if ((G < 16 || nlarge == 1) && eig_active_cached(c, G) > 0) return G;
    return 1;
}

// Clocks of one tridiagonalisation on G CTAs: a chain of short steps per column and the
// passes over the triangle.  Fitted to order 576 on one CTA and 900 to 2100 on 8 and 16;
// used for all orders, where only the ratio between the sizes matters (one problem
// alone goes from one CTA to 16 at order 360).
double trd_clocks(int m, int G) {
    const double n = m, n3 = n * n * n;
    return G == 1 ? 7.0e3 * n + 0.058 * n3 : 14.0e3 * n + 0.05 * n3 / G;
}

// CTAs for every problem's tridiagonalisation (orders in m): the smallest clusters with
// which each problem ends within T, for the smallest T in which the SMs can also hold them
// all.  One problem gets the widest cluster, a batch that fills the SMs one CTA each (or the
// smallest cluster whose shared memory holds the panel), a batch of uneven problems
// wider ones for its largest: with 96 problems of 218 to 595 the stage's length is no
// longer the largest one's on one SM.  0: beyond every cluster's shared memory.
std::vector<int> trd_groups(ptbgpu_ctx* c, const std::vector<int>& m, int small_max, int forced) {
    const int nsm = c->num_sms > 0 ? c->num_sms : 148;
    const int sizes[5] = {1, 2, 4, 8, 16};
    auto allowed = [&](int mm, int G) {
        if (G == 1) return mm <= small_max;
        // (many large triangles side by side are bound by HBM, not by their SMs: mixed
        // clusters of 2 to 16 took 155 ms on 48 problems up to 2773, 8 for all of them 144)
        if (mm > small_max && G < 8) return false;
        if (forced > 0 && mm > small_max && G != forced) return false;
        return tc_cap(mm, G) > 0 && eig_active_cached(c, G) > 0;
    };
    std::vector<int> pick(m.size(), 0);
    auto fill = [&](double T) {
        double area = 0.0;
        bool fits = true;
        for (size_t i = 0; i < m.size(); ++i) {
            int best = 0;
            for (int G : sizes) {
                if (!allowed(m[i], G)) continue;
                if (best == 0 || trd_clocks(m[i], G) < trd_clocks(m[i], best)) best = G;
                if (trd_clocks(m[i], best) <= T) break;
            }
            pick[i] = best;
            if (best == 0) continue;
            const double t = trd_clocks(m[i], best);
            area += best * t;
            fits = fits && t <= T;
        }
        return fits && area <= 0.85 * nsm * T;
    };
    double lo = 0.0, hi = 1.0e6;
    while (!fill(hi) && hi < 1.0e13) hi *= 2.0;
    for (int it = 0; it < 30; ++it) {
        const double mid = 0.5 * (lo + hi);
        (fill(mid) ? hi : lo) = mid;
    }
    fill(hi);
    return pick;
}

template <class K, class... Args>
void launch_clustered(K kern, int nclusters, int G, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = G;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(nclusters * G);
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    PTB_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
}

EigStreams& eig_streams(ptbgpu_ctx* c, EigBatch& eb) {
    if (!c->eig_streams) c->eig_streams = std::make_shared<EigStreams>();
    eb.st = std::static_pointer_cast<EigStreams>(c->eig_streams);
    return *eb.st;
}

// Arenas, task lists and uploads of a batch (on stream s).  hp holds the problems
// (k, m, nown, kind, mode, nocc, moff, eoff, o0, gbase, gld); Uout: Z's place for a
// single problem whose vectors the caller wants.
void eig_plan(ptbgpu_ctx* c, EigBatch& eb, cudaStream_t s, int small_max, double* Uout) {
    eig_setup_attrs();
    const int np = eb.nprob = (int)eb.hp.size();
    std::vector<int> all(np);   // largest first
    std::iota(all.begin(), all.end(), 0);
    std::stable_sort(all.begin(), all.end(), [&](int a, int b) { return eb.hp[a].m > eb.hp[b].m; });
    while (eb.nlarge < np && eb.hp[all[eb.nlarge]].m > small_max) ++eb.nlarge;
    if (eb.nlarge > 0 && !eb.grid) eb.G = eig_cluster_size(c, eb.nlarge);
    const int nsm = c->num_sms > 0 ? c->num_sms : 148;
    int64_t asz = 0, csz = 0, vsz = 0, bsz = 0, psz = 0, xsz = 0, ksz = 0, isz = 0;
    for (int q = 0; q < np; ++q) {
        EigProb& p = eb.hp[q];
        p.poff = psz;
        psz += (int64_t)p.m * p.nown;
        p.aoff = asz;
        p.coff = csz;
        p.ldc = (int)round_up(p.m, 16);
        csz += (int64_t)p.ldc * (p.m + kTcPadCols) + kTcPadRows;
        p.voff = vsz;
        p.boff = bsz;
        p.koff = ksz;
        p.ioff = isz;
        p.topm = -1;
        ksz += t_panels(p.m) * TS * TS;
        isz += (int64_t)((p.m + TS - 1) / TS) * TS * TS;
        asz += (int64_t)p.m * p.m;
        vsz += p.m;
        bsz += p.mode == 2 ? (int64_t)p.m * p.m : 4 * (int64_t)p.nown * p.m;
    }
    // task lists, largest problems first in each
    {
        std::vector<int> ms, pick;
        for (int q : all) ms.push_back(eb.hp[q].m);
        if (eb.grid) pick.assign(ms.size(), 0);
        else pick = trd_groups(c, ms, kTrdMax512, eig_cluster_forced());
        // two CTAs per SM only pay where the small orders fill the SMs
        int n256 = 0;
        for (size_t i = 0; i < all.size(); ++i) n256 += pick[i] == 1 && ms[i] <= kTrdMax256;
        auto group = [&](int G, int nt, auto&& mine) {
            EigBatch::Trd t;
            t.G = G;
            t.nt = nt;
            t.off = (int)eb.order.size();
            for (size_t i = 0; i < all.size(); ++i) {
                if (pick[i] != G || !mine(ms[i])) continue;
                EigProb& p = eb.hp[all[i]];
                p.xoff = xsz;
                xsz += G == 0 ? lg_layout(p.m, eb.G).total : G == 1 ? 0 : (int64_t)32 * p.m;
                if (t.n++ == 0) t.cap = G == 0 ? (p.m + 1) & ~1 : 0;
                t.cap = std::max(t.cap, G == 0 ? 0 : G == 1 ? trd_cap(p.m, nt) : tc_cap(p.m, G));
                eb.order.push_back(all[i]);
            }
            if (t.n > 0) eb.trd.push_back(t);
        };
        for (int G : {0, 16, 8, 4, 2}) group(G, 512, [](int) { return true; });
        group(1, 512, [&](int m) { return m > kTrdMax256 || n256 <= nsm; });
        group(1, 256, [&](int m) { return m <= kTrdMax256 && n256 > nsm; });
    }
    auto list = [&](EigBatch::Seg& g, auto&& fill) {
        g.off = eb.lists.size();
        fill();
        g.n = (unsigned)(eb.lists.size() - g.off);
    };
    auto put = [&](int a, int b) { eb.lists.push_back(make_int2(a, b)); };
    auto tiles = [](int n) { return (n + TS - 1) / TS; };
    list(eb.blocks, [&] {   // 64-column blocks (64-element chunks) of the generalized problems
        for (int q : all)
            for (int b = 0; b < tiles(eb.hp[q].m); ++b) put(q, b);
        // deep[j]: the leading tasks that hold every problem of more than j blocks
        eb.deep.clear();
        for (size_t i = eb.blocks.off; i < eb.lists.size(); ++i) {
            const size_t nb = (size_t)tiles(eb.hp[eb.lists[i].x].m);
            if (eb.deep.size() < nb) eb.deep.resize(nb);
            for (size_t j = 0; j < nb; ++j) eb.deep[j] = (unsigned)(i - eb.blocks.off + 1);
        }
    });
    list(eb.leaves, [&] {
        for (int q : all)
            for (int b = 0; b < (1 << dc_levels(eb.hp[q].m)); ++b) put(q, b);
    });
    list(eb.panels, [&] {
        for (int q : all)
            for (int b = 0; b < (int)t_panels(eb.hp[q].m); ++b) put(q, b);
    });
    auto grid2 = [&](int q, int nr, int nc) {
        for (int a = 0; a < nr; ++a)
            for (int b = 0; b < nc; ++b) put(q, a << 16 | b);
    };
    auto vectors = [&](auto&& count) {   // 64-vector blocks of every problem
        for (int q : all)
            for (int b = 0; b < tiles(count(eb.hp[q])); ++b) put(q, b);
    };
    list(eb.rows, [&] { vectors([](const EigProb& p) { return p.mode == 0 ? 2 * p.nown : 0; }); });
    list(eb.back, [&] {
        vectors([](const EigProb& p) { return p.mode == 0 ? 0 : p.mode == 1 ? p.m : p.nocc; });
    });
    list(eb.rq, [&] {
        for (int q : all)
            if (eb.hp[q].mode == 0) grid2(q, tiles(eb.hp[q].m), tiles(2 * eb.hp[q].nown));
    });
    list(eb.frq, [&] {
        for (int q : all)
            if (eb.hp[q].mode == 0) grid2(q, tiles(eb.hp[q].m), tiles(eb.hp[q].nown));
    });
    list(eb.fcols, [&] { vectors([](const EigProb& p) { return p.mode == 0 ? p.nown : 0; }); });
    list(eb.density, [&] {
        for (int q : all)
            if (eb.hp[q].mode == 2)   // no occupied vectors: tiles of zeros
                for (int cb = 0; cb < tiles(eb.hp[q].m); ++cb)
                    for (int rb = 0; rb <= cb; ++rb) put(q, rb << 16 | cb);
    });
    list(eb.fblocks, [&] {
        for (int q : all)
            if (eb.hp[q].mode == 0)
                for (int b = 0; b < tiles(eb.hp[q].m); ++b) put(q, b);
    });
    int nlev = 0;
    for (int q : all) nlev = std::max(nlev, dc_levels(eb.hp[q].m));
    eb.levels.resize(nlev);
    for (int t = 0; t < nlev; ++t) {
        EigBatch::Level& lv = eb.levels[t];
        lv.m0 = (int)eb.merges.size();
        for (int q : all) {
            EigProb& p = eb.hp[q];
            const int lev = dc_levels(p.m) - 1 - t;
            if (lev < 0) continue;
            for (int b = 0; b < (1 << lev); ++b) {
                if (lev == 0) p.topm = (int)eb.merges.size();
                eb.merges.push_back({q, dc_start(p.m, b, lev), dc_start(p.m, 2 * b + 1, lev + 1), dc_start(p.m, b + 1, lev)});
            }
        }
        lv.nm = (int)eb.merges.size() - lv.m0;
        auto each = [&](auto&& f) {
            for (int i = lv.m0; i < lv.m0 + lv.nm; ++i) f(i, eb.merges[i]);
        };
        list(lv.permute, [&] {
            each([&](int i, const DcMerge& g) {
                for (int b = 0; b * kDcRows < g.hi - g.lo; ++b) put(i, b);
            });
        });
        list(lv.elems, [&] {
            each([&](int i, const DcMerge& g) {
                for (int b = 0; b * kDcChunk < g.hi - g.lo; ++b) put(i, b);
            });
        });
        list(lv.product, [&] {
            each([&](int i, const DcMerge& g) {
                const EigProb& p = eb.hp[g.pi];
                if (p.mode == 0 && i == p.topm) return;   // its Q and V are used as they are
                grid2(i, tiles(g.mid - g.lo) + tiles(g.hi - g.mid), tiles(g.hi - g.lo));
            });
        });
    }

    eb.probs.reserve(c, sizeof(EigProb) * np);
    eb.order_d.reserve(c, sizeof(int) * eb.order.size());
    eb.lists_d.reserve(c, sizeof(int2) * std::max<size_t>(eb.lists.size(), 1));
    eb.merges_d.reserve(c, sizeof(DcMerge) * std::max<size_t>(eb.merges.size(), 1));
    eb.cnt.reserve(c, 8 * sizeof(int) * std::max<size_t>(eb.merges.size(), 1));
    const int64_t vpad = (vsz + 1) & ~int64_t(1);
    eb.dc.reserve(c, kDcBytes * vpad);
    eb.S = dc_arrays(eb.dc.ptr, vpad, eb.cnt.as<int>());
    eb.Ca.reserve(c, sizeof(double) * csz);
    for (WorkBuf* b : {&eb.La, &eb.Qa, &eb.Va}) b->reserve(c, sizeof(double) * asz);
    if (!Uout) eb.Za.reserve(c, sizeof(double) * asz);
    eb.Z = Uout ? Uout : eb.Za.as<double>();
    for (WorkBuf* b : {&eb.Da, &eb.Ea, &eb.Ta}) b->reserve(c, sizeof(double) * vsz);
    eb.Ba.reserve(c, sizeof(double) * std::max<int64_t>(bsz, 1));
    eb.Xa.reserve(c, sizeof(double) * std::max<int64_t>(xsz, 2));
    eb.Ka.reserve(c, sizeof(double) * std::max<int64_t>(ksz, 2));
    eb.Ia.reserve(c, sizeof(double) * std::max<int64_t>(isz, 2));
    eb.status.reserve(c, sizeof(int) * (np + 3));   // and a grid barrier's count, generation and error
    PTB_CUDA(cudaMemcpyAsync(eb.probs.ptr, eb.hp.data(), sizeof(EigProb) * np, cudaMemcpyHostToDevice, s));
    PTB_CUDA(cudaMemcpyAsync(eb.order_d.ptr, eb.order.data(), sizeof(int) * eb.order.size(), cudaMemcpyHostToDevice, s));
    PTB_CUDA(cudaMemcpyAsync(eb.lists_d.ptr, eb.lists.data(), sizeof(int2) * eb.lists.size(), cudaMemcpyHostToDevice, s));
    if (!eb.merges.empty())
        PTB_CUDA(cudaMemcpyAsync(eb.merges_d.ptr, eb.merges.data(), sizeof(DcMerge) * eb.merges.size(),
                                 cudaMemcpyHostToDevice, s));
    PTB_CUDA(cudaMemsetAsync(eb.status.ptr, 0, sizeof(int) * (np + 3), s));
}

// Every stage up to the eigenvalues, fe and owned rows (mode 0), all vectors (mode 1)
// or the densities (mode 2) on stream s.
void eig_run(ptbgpu_ctx* c, EigBatch& eb, cudaStream_t s, const double* H, const double* S, const int* d_maps,
             const int* d_own_cols, const int* d_ipos, double* d_e, double* d_fe) {
    const EigProb* dp = eb.probs.as<EigProb>();
    const int* ord = eb.order_d.as<int>();
    const DcMerge* mg = eb.merges_d.as<DcMerge>();
    double *Ca = eb.Ca.as<double>(), *La = eb.La.as<double>(), *Za = eb.Z, *Qa = eb.Qa.as<double>(),
           *Va = eb.Va.as<double>(), *Da = eb.Da.as<double>(), *Ea = eb.Ea.as<double>(), *Ta = eb.Ta.as<double>(),
           *Ba = eb.Ba.as<double>(), *Xa = eb.Xa.as<double>(), *Ka = eb.Ka.as<double>(), *Ia = eb.Ia.as<double>();
    int* st = eb.status.as<int>();
    const DcArr& D = eb.S;
    unsigned* bar = eb.grid ? reinterpret_cast<unsigned*>(st + eb.nprob) : nullptr;
    int* err = eb.grid ? st + eb.nprob + 2 : nullptr;
    // launches of one stage side by side: the first on s, the others on the side streams,
    // joined before the next stage
    const int side0 = eb.async ? EigStreams::kPerBatch : 0;
    int nside = side0;
    auto branch = [&](bool first) -> cudaStream_t {
        if (first) return s;
        EigStreams& es = eig_streams(c, eb);
        PTB_CHECK(nside < side0 + EigStreams::kPerBatch, PTBGPU_ECUDA, "eigensolver: more side launches than streams");
        PTB_CUDA(cudaStreamWaitEvent(es.side[nside], es.fork[eb.async], 0));
        return es.side[nside++];
    };
    auto fork = [&](bool many) {
        if (many) PTB_CUDA(cudaEventRecord(eig_streams(c, eb).fork[eb.async], s));
    };
    auto join = [&] {
        for (int i = side0; i < nside; ++i) {
            PTB_CUDA(cudaEventRecord(eb.st->join[i], eb.st->side[i]));
            PTB_CUDA(cudaStreamWaitEvent(s, eb.st->join[i], 0));
        }
        nside = side0;
    };
    auto launched = [&](int k = 1) {
        count_launch(k);
        PTB_CUDA(cudaGetLastError());
    };
    auto mark = [&](const char* what) {
        if (!eb.timed) return;
        eb.marks.push_back({what, c->take_event()});
        PTB_CUDA(cudaEventRecord(eb.marks.back().second, s));
    };
    mark("");
    // ---- Cholesky and C = L^-1 H L^-T (lower triangle)
    const int2* bl = eb.list(eb.blocks);
    k_eig_gather<<<eb.blocks.n, kT, 0, s>>>(dp, bl, d_maps, H, S, Ca, Qa, La);
    launched();
    if (eb.hp[0].kind == 0) {
        for (size_t j = 0; j < eb.deep.size(); ++j) {
            k_chol_column<<<eb.deep[j], kT, kTileSmem, s>>>(dp, bl, (int)j, La, Ia, st);
            launched();
            if (j + 1 == eb.deep.size()) break;
            k_chol_scale<<<eb.deep[j + 1], kT, kTileSmem, s>>>(dp, bl, (int)j, La, Ia, st);
            launched();
        }
        mark("Cholesky");
        k_eig_trsm<<<eb.blocks.n, kT, kTileSmem, s>>>(dp, bl, La, Ia, Qa, st);
        k_eig_rsolve<<<eb.blocks.n, kT, kTileSmem, s>>>(dp, bl, La, Ia, Qa, Ca, st);
        launched(2);
    }
    mark("reduction");
    // ---- tridiagonalisation, the widest groups first
    fork(eb.trd.size() > 1);
    for (size_t i = 0; i < eb.trd.size(); ++i) {
        const EigBatch::Trd& t = eb.trd[i];
        const cudaStream_t ls = branch(i + 1 == eb.trd.size());
        const int* od = ord + t.off;
        const size_t sm = sizeof(double) * t.cap;
        if (eb.grid) {
            int M = t.cap;
            void* args[] = {&dp, &od, &M, &Ca, &Da, &Ea, &Ta, &Xa, &st, &bar, &err};
            PTB_CUDA(cudaLaunchCooperativeKernel((void*)k_lg_trd, dim3(eb.G), dim3(kT), args, lg_smem_bytes(M), ls));
        } else if (t.G == 0) {
            launch_clustered(k_lg_trd, t.n, eb.G, lg_smem_bytes(t.cap), ls, dp, od, t.cap, Ca, Da, Ea, Ta, Xa,
                             (const int*)st, bar, err);
        } else if (t.G > 1) {
            launch_clustered(k_trd_cluster, t.n, t.G, sm, ls, dp, od, Ca, Da, Ea, Ta, Xa, t.cap, (const int*)st);
        } else if (t.nt == 512) {
            k_eig_trd<512><<<t.n, 512, sm, ls>>>(dp, od, Ca, Da, Ea, Ta, t.cap, st);
        } else {
            k_eig_trd<256><<<t.n, 256, sm, ls>>>(dp, od, Ca, Da, Ea, Ta, t.cap, st);
        }
        launched();
    }
    join();
    mark("tridiagonalisation");
    // ---- reflector panels, and the owned rows up to Z
    if (eb.panels.n) {
        k_vec_panels<<<eb.panels.n, kT, kWySmem, s>>>(dp, eb.list(eb.panels), Ca, Ta, Ka, st);
        launched();
    }
    if (eb.rows.n) {
        k_vec_rows<<<eb.rows.n, kT, kChainSmem, s>>>(dp, eb.list(eb.rows), Ca, La, Ia, Ka, d_own_cols, d_ipos, Ba, st);
        launched();
    }
    mark("panels");
    // ---- divide and conquer
    k_dc_leaves<<<(eb.leaves.n + kLeafWarps - 1) / kLeafWarps, 32 * kLeafWarps, 0, s>>>(
        dp, eb.list(eb.leaves), (int)eb.leaves.n, Da, Ea, Za, D, st);
    launched();
    for (const EigBatch::Level& lv : eb.levels) {
        const int2* el = eb.list(lv.elems);
        k_dc_deflate<<<lv.nm, kDeflT, 0, s>>>(dp, mg, lv.m0, Ea, Za, D, st);
        k_dc_permute<<<lv.permute.n, 256, 0, s>>>(dp, mg, eb.list(lv.permute), Za, Qa, D, st);
        k_dc_secular<<<lv.elems.n, 256, 0, s>>>(dp, mg, el, Ea, D, st);
        k_dc_zhat<<<lv.elems.n, 256, 0, s>>>(dp, mg, el, Ea, D, st);
        k_dc_vectors<<<lv.elems.n, 256, 0, s>>>(dp, mg, el, Va, D, st);
        launched(5);
        if (lv.product.n) {
            k_dc_product<<<lv.product.n, kT, kTileSmem, s>>>(dp, mg, eb.list(lv.product), Za, Qa, Va, D, st);
            launched();
        }
    }
    mark("divide and conquer");
    // ---- what leaves the solver
    if (eb.rq.n) {
        const int2* rq = eb.list(eb.rq);
        k_vec_rq<<<eb.rq.n, kT, kTileSmem, s>>>(dp, rq, Za, Qa, Va, D, Ba, st);
        k_vec_rv<<<eb.rq.n, kT, kTileSmem, s>>>(dp, rq, Za, Qa, Va, D, Ba, st);
        k_vec_fe<<<eb.fblocks.n, 256, 0, s>>>(dp, eb.list(eb.fblocks), Ba, D, d_e, d_fe, st);
        launched(3);
    }
    if (eb.hp[0].mode != 0) {
        k_vec_values<<<eb.blocks.n, TS, 0, s>>>(dp, eb.list(eb.blocks), D, d_e, st);
        launched();
    }
    if (eb.back.n) {
        k_vec_back<<<eb.back.n, kT, kChainSmem, s>>>(dp, eb.list(eb.back), Ca, La, Ia, Ka, Za, st);
        launched();
    }
    if (eb.density.n) {
        k_vec_density<<<eb.density.n, kT, kTileSmem, s>>>(dp, eb.list(eb.density), Za, Ba, st);
        launched();
    }
    mark("vectors");
}

}  // namespace

std::shared_ptr<EigBatch> eig_batch_launch(ptbgpu_ctx* c, int64_t n, const double* H, const double* S,
                                           const std::vector<EigProbHost>& probs, const int* d_maps,
                                           const int* d_own_cols, const int* d_ipos, double* d_e, double* d_fe,
                                           int prl, double* flops, int slot) {
    if (probs.empty()) return nullptr;
    auto eb = std::make_shared<EigBatch>();
    eb->prl = prl;
    eb->timed = prl >= 2;
    for (const EigProbHost& q : probs) {
        PTB_CHECK(q.m >= 1 && q.m <= kLargeMax, PTBGPU_EINVAL, "submatrix %d of order %d outside the eigensolver (1..%d)",
                  q.k + 1, q.m, kLargeMax);
        EigProb p{};
        p.k = q.k;
        p.m = q.m;
        p.nown = q.nown;
        p.moff = q.moff;
        p.eoff = q.eoff;
        p.o0 = q.o0;
        p.gbase = q.gbase;
        p.gld = q.gld < 0 ? n : q.gld;
        p.mode = q.mode;
        p.nocc = q.nocc;
        eb->hp.push_back(p);
        if (flops) *flops += 7.0 * std::pow((double)q.m, 3);
    }
    cudaStream_t s = c->stream;
    // the uploads of the plan on the context's stream: on base they would wait for the
    // batches before this one, and the host with them
    eig_plan(c, *eb, s, kEigBatchMax, nullptr);
    log_line(prl, 2, " * eigensolver: %d problems, %d above order %d, %zu merge levels", eb->nprob, eb->nlarge,
             kEigBatchMax, eb->levels.size());
    for (const EigBatch::Trd& t : eb->trd)
        log_line(prl, 2, " *   tridiagonalisation of %d on %d CTAs of %d threads each", t.n, t.G ? t.G : eb->G, t.nt);
    if (slot >= 0) {
        // beside what follows on the context's stream
        PTB_CHECK(slot < kEigSlots, PTBGPU_EINVAL, "eigensolver: no such batch slot");
        EigStreams& es = eig_streams(c, *eb);
        PTB_CUDA(cudaEventRecord(es.start, s));
        PTB_CUDA(cudaStreamWaitEvent(es.base, es.start, 0));
        s = es.base;
        eb->async = true;
        eb->slot = slot;
    }
    eig_run(c, *eb, s, H, S, d_maps, d_own_cols, d_ipos, d_e, d_fe);
    if (eb->async) PTB_CUDA(cudaEventRecord(eb->st->done[slot], s));
    return eb;
}

void eig_batch_join(ptbgpu_ctx* c, EigBatch& eb) {
    if (eb.async) PTB_CUDA(cudaStreamWaitEvent(c->stream, eb.st->done[eb.slot], 0));
}

// A batch's first failing problem: the lowest one with a non-positive-definite overlap, else
// the lowest whose leaves did not converge.  Waits for the batch (joined into the
// context's stream).
EigFault eig_batch_fault(ptbgpu_ctx* c, EigBatch& eb) {
    cudaStream_t s = c->stream;
    const int np = eb.nprob;
    std::vector<int> hst(np + 3);
    PTB_CUDA(cudaMemcpyAsync(hst.data(), eb.status.ptr, sizeof(int) * (np + 3), cudaMemcpyDeviceToHost, s));
    PTB_CUDA(cudaStreamSynchronize(s));
    PTB_CHECK(hst[np + 2] == 0, PTBGPU_ETIMEOUT, "eigensolver: a grid barrier gave up waiting");
    if (eb.timed)
        eb.stage_times([&](const char* what, double ms) {
            log_line(eb.prl, 2, " *   eigensolver stage %-20s %10.3f ms", what, ms);
        });
    EigFault f;
    for (int q = 0; q < np; ++q)
        if (hst[q] != kStOk) f.merge({eb.hp[q].k, hst[q]});
    return f;
}

void eig_fault_raise(const EigFault& f, const char* what) {
    PTB_CHECK(f.status <= 0, PTBGPU_ENOTSPD, "overlap of %s %d not positive definite (leading minor %d)", what, f.k + 1,
              f.status);
    PTB_CHECK(f.status == kStOk, PTBGPU_EITER, "tridiagonal eigensolver did not converge on %s %d", what, f.k + 1);
}

void eig_batch_check(ptbgpu_ctx* c, EigBatch& eb) { eig_fault_raise(eig_batch_fault(c, eb), "submatrix"); }

void eig_batch_final(ptbgpu_ctx* c, EigBatch& eb, double mu, const int* d_maps, const int* d_own_cols, double* dP,
                     double* dPdense) {
    if (eb.nprob == 0 || eb.fcols.n == 0) return;
    cudaStream_t s = c->stream;
    const EigProb* dp = eb.probs.as<EigProb>();
    const double *Za = eb.Z, *Qa = eb.Qa.as<double>(), *Va = eb.Va.as<double>();
    double* Ba = eb.Ba.as<double>();
    const int2* fr = eb.list(eb.frq);
    k_fin_occ<<<eb.fblocks.n, 256, 0, s>>>(dp, eb.list(eb.fblocks), eb.S, Ba, mu);
    k_fin_vw<<<eb.frq.n, kT, kTileSmem, s>>>(dp, fr, Za, Qa, Va, eb.S, Ba);
    k_fin_qw<<<eb.frq.n, kT, kTileSmem, s>>>(dp, fr, Za, Qa, Va, eb.S, Ba);
    k_fin_cols<<<eb.fcols.n, kT, kChainSmem, s>>>(dp, eb.list(eb.fcols), eb.Ca.as<double>(), eb.La.as<double>(),
                                                  eb.Ia.as<double>(), eb.Ka.as<double>(), d_maps, d_own_cols, Ba, dP, dPdense);
    count_launch(4);
    PTB_CUDA(cudaGetLastError());
}

// Matrix with both triangles set from the upper one: out[i + j n] = a[min(i,j) + max(i,j) n].
__global__ void k_sym_from_upper(int64_t n, const double* __restrict__ a, double* __restrict__ out) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n * n; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = q % n, j = q / n;
        out[q] = (i <= j) ? a[i + j * n] : a[j + i * n];
    }
}

constexpr int kGridRows = 64;   // rows per CTA of a cooperative-grid solve
constexpr int kGridMax = 64;    // CTAs of a cooperative-grid solve at most
constexpr int kGridMin = 4096;  // orders solved by one cluster instead

// By doubling: the 64 x 64 diagonal blocks, then per level every pair of neighbouring
// inverted blocks, [L11 0; L21 L22]^-1 = [L11^-1 0; -L22^-1 L21 L11^-1  L22^-1], two launches
// over all tiles of all pairs.  At order 1495 0.25 ms, bound by the chain of levels, against
// 1.9 for library calls over recursive halves, which followed one another; the four blocks
// of 2944 of order 11776 3.2 ms against 19.
//   W takes h doubles for each of a level's rows below the diagonal blocks, which are at most
// n - h and at most n / 2: n^2 / 4 in all.
void tri_inverse(ptbgpu_ctx* c, int64_t n, int64_t ld, double* A, double* W) {
    if (n <= 0) return;
    eig_setup_attrs();
    cudaStream_t s = c->stream;
    const int64_t nb = (n + TS - 1) / TS;
    k_tri_diag<<<(unsigned)nb, kT, 0, s>>>(n, ld, A);
    count_launch();
    for (int64_t h = TS; h < n; h *= 2) {
        const dim3 grid((unsigned)(h / TS), (unsigned)((std::min(h, n - h) + TS - 1) / TS),
                        (unsigned)((n - h + 2 * h - 1) / (2 * h)));
        k_tri_level<true><<<grid, kT, kTileSmem, s>>>(n, ld, (int)h, A, W);
        k_tri_level<false><<<grid, kT, kTileSmem, s>>>(n, ld, (int)h, A, W);
        count_launch(2);
    }
    PTB_CUDA(cudaGetLastError());
}

// A = Li H Li^T over H (both triangles) and P = X -> Li^T X Li over X (upper triangle), T
// n x n scratch: tile products with the inverse, of which the second stays in one
// triangle.  At order 2208 0.63 ms each (and 0.42 for the inverse), against 2.5 and 2.4 for
// two library triangular solves each.
void tri_congruence(ptbgpu_ctx* c, int64_t n, const double* Li, double* H, double* T) {
    eig_setup_attrs();
    const unsigned nb = (unsigned)((n + TS - 1) / TS);
    k_tri_product<TRI_LH><<<dim3(nb, nb), kT, kTileSmem, c->stream>>>(n, Li, H, T);
    k_tri_product<TRI_TLT><<<dim3(nb, nb), kT, kTileSmem, c->stream>>>(n, Li, T, H);
    count_launch(2);
    PTB_CUDA(cudaGetLastError());
    symmetrize_upper(c->stream, n, n, H);
}
void tri_back(ptbgpu_ctx* c, int64_t n, const double* Li, double* X, double* T) {
    eig_setup_attrs();
    const unsigned nb = (unsigned)((n + TS - 1) / TS);
    k_tri_product<TRI_XL><<<dim3(nb, nb), kT, kTileSmem, c->stream>>>(n, Li, X, T);
    k_tri_product<TRI_LTT><<<dim3(nb, nb), kT, kTileSmem, c->stream>>>(n, Li, T, X);
    count_launch(2);
    PTB_CUDA(cudaGetLastError());
}

void eig_full(ptbgpu_ctx* c, int64_t n, const double* H, const double* S, double* w, double* U) {
    PTB_CHECK(n >= 1 && n <= kLargeMax, PTBGPU_EINVAL, "eigenproblem of order %lld outside the eigensolver (1..%d)",
              (long long)n, kLargeMax);
    eig_setup_attrs();
    cudaStream_t s = c->stream;
    const int m = (int)n;
    EigBatch eb;
    EigProb p{};
    p.m = m;
    p.kind = S ? 0 : 1;
    p.mode = 1;
    p.gld = n;
    eb.hp.push_back(p);
    // up to order kGridMin one thread-block cluster (hardware barrier), above it
    // a cooperative grid of one CTA per kGridRows rows, at most kGridMax CTAs
    // (the software barrier's latency grows with the CTA count)
    eb.grid = m > kGridMin;
    if (eb.grid) {
        int per_sm = 0;
        PTB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lg_trd, kT, lg_smem_bytes(kLargeMax)));
        PTB_CHECK(per_sm >= 1, PTBGPU_ECUDA, "eigensolver kernel does not fit an SM");
        const int nsm = c->num_sms > 0 ? c->num_sms : 148;
        eb.G = std::min({nsm * per_sm, kGridMax, std::max(1, m / kGridRows)});
    }
    WorkBuf map;   // the identity row map
    map.reserve(c, sizeof(int) * n);
    std::vector<int> ident(n);
    for (int i = 0; i < m; ++i) ident[i] = i;
    PTB_CUDA(cudaMemcpyAsync(map.ptr, ident.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s));
    // PTBGPU_EIG_STAGES=1: stage times on stderr
    static const bool stages = getenv("PTBGPU_EIG_STAGES") != nullptr;
    eb.timed = stages;
    eig_plan(c, eb, s, 0, U);
    eig_run(c, eb, s, H, S, map.as<int>(), nullptr, nullptr, w, nullptr);
    int hs[4];
    PTB_CUDA(cudaMemcpyAsync(hs, eb.status.ptr, sizeof(int) * 4, cudaMemcpyDeviceToHost, s));
    PTB_CUDA(cudaStreamSynchronize(s));
    if (eb.timed) {
        fprintf(stderr, "eig_full n=%d:", m);
        eb.stage_times([](const char* what, double ms) { fprintf(stderr, " %s %.3f", what, ms); });
        fprintf(stderr, " ms\n");
    }
    PTB_CHECK(hs[3] == 0, PTBGPU_ETIMEOUT, "eigensolver: a grid barrier gave up waiting");
    PTB_CHECK(hs[0] <= 0, PTBGPU_ENOTSPD, "overlap matrix not positive definite (leading minor %d)", hs[0]);
    PTB_CHECK(hs[0] == kStOk, PTBGPU_EITER, "tridiagonal eigensolver did not converge");
}

void eig_full_upper(ptbgpu_ctx* c, int64_t n, double* A, double* B, double* w) {
    cudaStream_t s = c->stream;
    WorkBuf h, b, u;
    h.reserve(c, sizeof(double) * n * n);
    u.reserve(c, sizeof(double) * n * n);
    const int grid = (int)std::min<int64_t>((n * n + 255) / 256, 148 * 16);
    k_sym_from_upper<<<grid, 256, 0, s>>>(n, A, h.as<double>());
    count_launch();
    if (B) {
        b.reserve(c, sizeof(double) * n * n);
        k_sym_from_upper<<<grid, 256, 0, s>>>(n, B, b.as<double>());
        count_launch();
    }
    PTB_CUDA(cudaGetLastError());
    eig_full(c, n, h.as<double>(), B ? b.as<double>() : nullptr, w, u.as<double>());
    PTB_CUDA(cudaMemcpyAsync(A, u.ptr, sizeof(double) * n * n, cudaMemcpyDeviceToDevice, s));
    PTB_CUDA(cudaStreamSynchronize(s));
}

// Packed upper triangle of scale * P (P m x m column-major, read above the diagonal).
__global__ void k_pack_scaled(int64_t m, const double* __restrict__ P, double scale, double* __restrict__ pk) {
    const int64_t np = m * (m + 1) / 2;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < np; q += (int64_t)gridDim.x * blockDim.x) {
        int64_t j = (int64_t)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
        while ((j + 1) * (j + 2) / 2 <= q) ++j;
        while (j * (j + 1) / 2 > q) --j;
        const int64_t i = q - j * (j + 1) / 2;
        pk[q] = scale * P[i + j * m];
    }
}

void eig_density_batch(ptbgpu_ctx* c, int64_t ninst, const int64_t* ndim, const int64_t* nel,
                       const double* const* Hpk, const double* const* Spk, double* const* Ppk, double filter,
                       int prl, ptbgpu_stats* st) {
    if (ninst <= 0) return;
    cudaStream_t s = c->stream;
    // The systems above kEigBatchMax go first, in up to kEigSlots parts of the input
    // order, each a batch on a stream of its own: a part is copied in while the one
    // before it is solved, and copied out while the next is.  The small systems are
    // copied in after them and solved and copied out beside them.  A part of few systems
    // leaves SMs idle, so that two parts lose against one below 20 large systems and pay
    // above (ndim 1000 to 3060, pageable host arrays, copies inside; two parts against one:
    // 8 systems 217 / 168 ms, 16 272 / 262, 20 305 / 304, 24 325 / 343, 28 375 / 412, 32
    // 401 / 468), and more than two need parts of 24 each (64 systems in two parts 550 ms, in
    // four 590, in one 659; 100 862 -> 782, 256 1.79 -> 1.65 s).
    constexpr size_t kPartMin = 24;
    std::vector<int64_t> large, small;
    std::vector<int64_t> pkoff((size_t)ninst + 1, 0);
    int64_t hsz = 0, nsum = 0;
    std::vector<EigProbHost> pr((size_t)ninst);
    for (int64_t k = 0; k < ninst; ++k) {
        const int64_t m = ndim[k];
        PTB_CHECK(m >= 1 && m <= kLargeMax, PTBGPU_EINVAL, "system %lld: ndim %lld outside the eigensolver (1..%d)",
                  (long long)k, (long long)m, kLargeMax);
        PTB_CHECK(nel[k] >= 0 && nel[k] / 2 <= m && Hpk[k] && Spk[k] && Ppk[k], PTBGPU_EINVAL,
                  "system %lld: bad electron count or arrays", (long long)k);
        PTB_CHECK(nel[k] % 2 == 0, PTBGPU_EINVAL,
                  "system %lld: odd electron count %lld (the T = 0 projector here is closed-shell)", (long long)k,
                  (long long)nel[k]);
        EigProbHost& q = pr[k];
        q.k = (int)k;
        q.m = (int)m;
        q.nown = 0;
        q.moff = nsum;
        q.eoff = nsum;
        q.o0 = 0;
        q.gbase = hsz;
        q.gld = m;
        q.mode = 2;
        q.nocc = (int)(nel[k] / 2);
        hsz += m * m;
        nsum += m;
        pkoff[k + 1] = pkoff[k] + m * (m + 1) / 2;
        (m > kEigBatchMax ? large : small).push_back(k);
    }
    struct Drain {   // a failing part leaves no copy into the caller's arrays on its way
        cudaStream_t s;
        ~Drain() { cudaStreamSynchronize(s); }
    } drain{s};
    struct Bufs {
        WorkBuf h, sm, pk, maps, e, dummy;
    } b;
    b.h.reserve(c, sizeof(double) * hsz);
    b.sm.reserve(c, sizeof(double) * hsz);
    b.pk.reserve(c, sizeof(double) * std::max<int64_t>(2 * pkoff[ninst], 1));
    b.maps.reserve(c, sizeof(int) * nsum);
    b.e.reserve(c, sizeof(double) * nsum);
    b.dummy.reserve(c, 64);
    std::vector<int> maps((size_t)nsum);
    for (const EigProbHost& q : pr)
        for (int i = 0; i < q.m; ++i) maps[q.moff + i] = i;
    PTB_CUDA(cudaMemcpyAsync(b.maps.ptr, maps.data(), sizeof(int) * nsum, cudaMemcpyHostToDevice, s));
    double* pkH = b.pk.as<double>();
    double* pkS = pkH + pkoff[ninst];
    auto upload = [&](const std::vector<int64_t>& ids) {
        for (int64_t k : ids) {
            const int64_t m = ndim[k], np = m * (m + 1) / 2;
            PTB_CUDA(cudaMemcpyAsync(pkH + pkoff[k], Hpk[k], sizeof(double) * np, cudaMemcpyHostToDevice, s));
            PTB_CUDA(cudaMemcpyAsync(pkS + pkoff[k], Spk[k], sizeof(double) * np, cudaMemcpyHostToDevice, s));
            unpack_sym(s, m, m, pkH + pkoff[k], b.h.as<double>() + pr[k].gbase, filter);
            unpack_sym(s, m, m, pkS + pkoff[k], b.sm.as<double>() + pr[k].gbase, filter);
        }
    };
    auto launch = [&](const std::vector<int64_t>& ids, int slot) {
        std::vector<EigProbHost> probs;
        for (int64_t k : ids) probs.push_back(pr[k]);
        double flops = 0.0;
        auto eb = eig_batch_launch(c, 0, b.h.as<double>(), b.sm.as<double>(), probs, b.maps.as<int>(),
                                   b.dummy.as<int>(), b.dummy.as<int>(), b.e.as<double>(), b.e.as<double>(), prl,
                                   &flops, slot);
        return eb;
    };
    auto download = [&](EigBatch& eb, const std::vector<int64_t>& ids) {
        for (size_t q = 0; q < ids.size(); ++q) {
            const int64_t k = ids[q], m = ndim[k], np = m * (m + 1) / 2;
            const int grid = (int)std::min<int64_t>((np + 255) / 256, 148 * 8);
            k_pack_scaled<<<grid, 256, 0, s>>>(m, eb.Ba.as<double>() + eb.hp[q].boff, 2.0, pkH + pkoff[k]);
            count_launch();
            PTB_CUDA(cudaGetLastError());
            PTB_CUDA(cudaMemcpyAsync(Ppk[k], pkH + pkoff[k], sizeof(double) * np, cudaMemcpyDeviceToHost, s));
        }
    };
    // parts of about equal work (m^3, which the copies follow at a distance)
    const size_t nparts =
        large.size() < kPartMin ? 1 : std::min<size_t>(kEigSlots, std::max<size_t>(2, large.size() / kPartMin));
    std::vector<std::vector<int64_t>> parts;
    double work = 0.0, done = 0.0;
    for (int64_t k : large) work += std::pow((double)ndim[k], 3);
    for (int64_t k : large) {
        const size_t part = std::min(nparts - 1, (size_t)(done / work * (double)nparts));
        if (parts.size() <= part) parts.resize(part + 1);
        parts[part].push_back(k);
        done += std::pow((double)ndim[k], 3);
    }
    // declared after b: released (side streams drained) before its buffers
    std::vector<std::shared_ptr<EigBatch>> ebl;
    std::shared_ptr<EigBatch> ebs;
    for (size_t i = 0; i < parts.size(); ++i) {
        upload(parts[i]);
        ebl.push_back(parts[i].empty() ? nullptr : launch(parts[i], (int)i));
    }
    upload(small);
    if (!small.empty()) ebs = launch(small, -1);
    // Results are copied out as their batch ends, while the next one is solved; after a
    // failure the others are waited for only, and the call's first failing system is named.
    EigFault fault;
    auto finish = [&](EigBatch& eb, const std::vector<int64_t>& ids) {
        eig_batch_join(c, eb);
        fault.merge(eig_batch_fault(c, eb));
        if (fault.status == kStOk) download(eb, ids);
    };
    if (ebs) finish(*ebs, small);
    for (size_t i = 0; i < parts.size(); ++i)
        if (ebl[i]) finish(*ebl[i], parts[i]);
    eig_fault_raise(fault, "system");
    PTB_CUDA(cudaStreamSynchronize(s));
    if (st)
        for (int64_t k = 0; k < ninst; ++k) st[k].flops += 7.0 * std::pow((double)ndim[k], 3);
}

// Kernel-level entry: dense host problems through the same stages.  Problem k's
// H and S sit at offset sum_{k'<k} m_k'^2 of the concatenated input (ld m_k);
// its owned columns are given by local index.
void sygv_batched_entry(ptbgpu_ctx* c, int64_t np, const int64_t* dims, const double* H, const double* S,
                        const int64_t* nown, const int64_t* owned, double mu, double* e, double* fe, double* Pcols) {
    struct Bufs {
        WorkBuf h, s, maps, own, ipos, e, fe, p;
    } b;
    cudaStream_t st = c->stream;
    std::vector<EigProbHost> probs;
    std::vector<int> maps, own, ipos;
    int64_t hsz = 0, nsum = 0, osum = 0, psz = 0;
    for (int64_t k = 0; k < np; ++k) {
        const int m = (int)dims[k];
        PTB_CHECK(dims[k] >= 1 && dims[k] <= kLargeMax && nown[k] >= 1 && nown[k] <= dims[k], PTBGPU_EINVAL,
                  "problem %lld: order %lld (1..%d) or owned count %lld out of range", (long long)k,
                  (long long)dims[k], kLargeMax, (long long)nown[k]);
        EigProbHost q{};
        q.k = (int)k;
        q.m = m;
        q.nown = (int)nown[k];
        q.moff = nsum;
        q.eoff = nsum;
        q.o0 = osum;
        q.gbase = hsz;
        q.gld = m;
        probs.push_back(q);
        for (int i = 0; i < m; ++i) {
            maps.push_back(i);
            ipos.push_back(i);
        }
        for (int64_t t = 0; t < nown[k]; ++t) {
            const int64_t li = owned[osum + t];
            PTB_CHECK(li >= 0 && li < m, PTBGPU_EINVAL, "problem %lld: owned index %lld out of range",
                      (long long)k, (long long)li);
            own.push_back((int)(nsum + li));
        }
        hsz += (int64_t)m * m;
        nsum += m;
        osum += nown[k];
        psz += (int64_t)m * nown[k];
    }
    b.h.reserve(c, sizeof(double) * hsz);
    b.s.reserve(c, sizeof(double) * hsz);
    b.maps.reserve(c, sizeof(int) * nsum);
    b.own.reserve(c, sizeof(int) * osum);
    b.ipos.reserve(c, sizeof(int) * nsum);
    b.e.reserve(c, sizeof(double) * nsum);
    b.fe.reserve(c, sizeof(double) * nsum);
    PTB_CUDA(cudaMemcpyAsync(b.h.ptr, H, sizeof(double) * hsz, cudaMemcpyHostToDevice, st));
    PTB_CUDA(cudaMemcpyAsync(b.s.ptr, S, sizeof(double) * hsz, cudaMemcpyHostToDevice, st));
    PTB_CUDA(cudaMemcpyAsync(b.maps.ptr, maps.data(), sizeof(int) * nsum, cudaMemcpyHostToDevice, st));
    PTB_CUDA(cudaMemcpyAsync(b.own.ptr, own.data(), sizeof(int) * osum, cudaMemcpyHostToDevice, st));
    PTB_CUDA(cudaMemcpyAsync(b.ipos.ptr, ipos.data(), sizeof(int) * nsum, cudaMemcpyHostToDevice, st));
    std::shared_ptr<EigBatch> eb =
        eig_batch_launch(c, 0, b.h.as<double>(), b.s.as<double>(), probs, b.maps.as<int>(), b.own.as<int>(),
                         b.ipos.as<int>(), b.e.as<double>(), b.fe.as<double>(), 0, nullptr);
    eig_batch_check(c, *eb);
    PTB_CUDA(cudaMemcpyAsync(e, b.e.ptr, sizeof(double) * nsum, cudaMemcpyDeviceToHost, st));
    PTB_CUDA(cudaMemcpyAsync(fe, b.fe.ptr, sizeof(double) * nsum, cudaMemcpyDeviceToHost, st));
    if (Pcols) {
        b.p.reserve(c, sizeof(double) * psz);
        eig_batch_final(c, *eb, mu, b.maps.as<int>(), b.own.as<int>(), nullptr, b.p.as<double>());
        PTB_CUDA(cudaMemcpyAsync(Pcols, b.p.ptr, sizeof(double) * psz, cudaMemcpyDeviceToHost, st));
    }
    PTB_CUDA(cudaStreamSynchronize(st));
}

}  // namespace ptb
