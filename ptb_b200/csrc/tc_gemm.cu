// tcgen05 tensor-core products for the trace-correcting purification.
//
// C = sum_p A_{a(p)} * B_{b(p)}^T over a short list of bf16 operand planes,
// accumulated in FP32 in tensor memory.  With planes {X_hi, X_lo} and the
// products (hi,hi) + (hi,lo) + (lo,hi) this is the "bf16x3" split product of
// an FP32 matrix (about 16 significant bits per operand; the dropped lo*lo
// term is 2^-16 relative).
//
// With three planes {hi, mid, lo} (hi = bf16(x), mid = bf16(x - hi),
// lo = bf16(x - hi - mid)) and the six products hh + hm + mh + hl + lh + mm the
// operands carry about 24 significant bits ("bf16x6").
//
// One CTA computes a 128 x BN tile (cta_group::1, UMMA 128xBNx16); BN = 256
// with two planes or BN = 128 with three planes.  K advances in blocks of KB:
// 64 (128B swizzle, two 96 KB stages) or 32 (64B swizzle, four 48 KB stages);
// the launcher times both on the first launch of a shape and keeps the faster.
//   warp 0      TMA producer: per K block, NP A tiles (128xKB) and NP B tiles
//               (BNxKB) into the stage ring, swizzled, completion on a "full"
//               mbarrier with a transaction count;
//   warp 1      MMA issuer (one thread): KB/16 K16 steps x the product list per
//               stage, tcgen05.commit releases the stage on its "empty" mbarrier;
//   warp 2      allocates / frees the BN TMEM columns of the accumulator;
//   warps 4..7  epilogue: tcgen05.ld of their 32 lanes (rows), fused update.
//
// Epilogues:
//   EPI_FULL  every tile; C written row-major as FP32 (general product).
//   EPI_SP2   symmetric X*X: only tiles touching the upper triangle run; the
//             element (r,c), c >= r, becomes X' = C (branch "square") or
//             2X - C, written to (r,c) and (c,r) as FP32 and as the bf16
//             hi/mid/lo planes of the next product; per-tile trace and sum of squares
//             (= tr X'^2 for symmetric X') go to a stats array that the
//             decision kernel reduces in a fixed order (deterministic).
//
// Every mbarrier wait is bounded (2 s of globaltimer); on expiry the CTA sets
// an error word, drains the copies it issued and frees its TMEM.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "common.cuh"
#include "tc_gemm.cuh"
#include "tc_ptx.cuh"

namespace ptb {
namespace tc {

namespace {

using namespace ptx;

constexpr int BM = 128;
constexpr int THREADS = 256;
constexpr int kSmemBudget = 196608;   // operand ring (192 KB); barriers and alignment come on top

// Tile configuration: BN output columns, NP operand planes, KB K elements per
// stage.  KB = 64 rows are 128 bytes (128B swizzle, 1024-byte atoms); KB = 32
// rows are 64 bytes (64B swizzle, 512-byte atoms).  The ring holds as many
// stages as fit in the 192 KB budget: 2 for KB = 64, 4 for KB = 32.
template <int BN, int NP, int KB>
struct Cfg {
    static constexpr int A_TILE_BYTES = BM * KB * 2;
    static constexpr int B_TILE_BYTES = BN * KB * 2;
    static constexpr int STAGE_BYTES = NP * (A_TILE_BYTES + B_TILE_BYTES);
    static constexpr int STAGES = kSmemBudget / STAGE_BYTES;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
    static constexpr uint32_t SWIZZLE_LAYOUT = KB == 64 ? 2u : 4u;      // UMMA layout type
    static constexpr uint32_t SBO = KB == 64 ? 1024u : 512u;            // bytes between 8-row groups
    // Instruction descriptor for kind::f16: D fp32, A/B bf16, both K-major, M=128, N=BN.
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                                      ((uint32_t)(BM >> 4) << 24);
    static_assert(KB == 64 || KB == 32, "K block of 64 or 32 elements");
    static_assert(STAGES >= 2 && STAGES <= 4, "2..4 pipeline stages");
    static_assert(STAGE_BYTES % 1024 == 0, "stages keep the swizzle atoms aligned");
};

__device__ __forceinline__ void split_bf16(float v, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
    h = __float2bfloat16_rn(v);
    const float r = v - __bfloat162float(h);
    m = __float2bfloat16_rn(r);
    l = __float2bfloat16_rn(r - __bfloat162float(m));
}

// ---- the kernel -----------------------------------------------------------
// Epilogue warps 4..7 (q = TMEM lane quarter) of a 128 x BN accumulator in this
// CTA's tensor memory: wait for it (bounded), drain it with the fused update,
// and reduce the per-tile trace / sum of squares into stats[2 * stat_index].
template <int EPI, int BN>
__device__ __forceinline__ void tc_epilogue(const EpiParams& ep, uint32_t tmem, uint32_t accum_bar,
                                            int* abort_flag, double* red, int bi, int bj, int q, int lane,
                                            int stat_index) {
    const int64_t ld = ep.ld;
    const int64_t r = (int64_t)bi * BM + q * 32 + lane;    // row of the (stacked) planes
    // stacked systems: the tile's system starts at row rb; rows and columns
    // below are local to it (rb = 0 for a single system)
    const int64_t rb = ep.stacked ? ((int64_t)bi * BM / ld) * ld : 0;
    const int64_t rl = r - rb;
    double tr = 0.0, ss = 0.0;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(accum_bar, 0));
    if (!ok && lane == 0) {
        set_err(ep.err, 31);
        *(volatile int*)abort_flag = 1;
    }
    const int aborted = __shfl_sync(0xffffffffu, *(volatile int*)abort_flag, 0);
    tc_fence_after();
    if (ok && !aborted) {
        const bool square = (EPI == EPI_SP2) ? (ep.sq_flag[rb / ld] != 0) : true;
        const bool w3 = ep.lo2 != nullptr;   // third plane written (kept only for three-plane products)
        for (int c0 = 0; c0 < BN; c0 += 32) {
            uint32_t v[32];
            __syncwarp();   // lanes may have taken different paths in the previous chunk
            tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)c0, v);
            const int64_t cbase = (int64_t)bj * BN - rb + c0;   // local column
            if (EPI == EPI_FULL) {
                float4* dst = reinterpret_cast<float4*>(ep.out + r * ld + cbase);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    dst[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                         __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
                continue;
            }
            if (cbase + 31 < rl) continue;      // chunk entirely below the diagonal
            if (cbase >= rl) {
                // whole chunk in the upper triangle: vector path
                const float4* xin = reinterpret_cast<const float4*>(ep.xcur + r * ld + cbase);
                float4* xo = reinterpret_cast<float4*>(ep.out + r * ld + cbase);
                uint4* ho = reinterpret_cast<uint4*>(ep.hi + r * ld + cbase);
                uint4* mo = reinterpret_cast<uint4*>(ep.lo + r * ld + cbase);
                uint4* lo = w3 ? reinterpret_cast<uint4*>(ep.lo2 + r * ld + cbase) : nullptr;
                // X is only needed for 2X - X^2: skip its read on the square branch.  The chunk's
                // eight reads go out together, before any store that could alias them holds
                // them back
                float4 xc[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) xc[q] = square ? make_float4(0.f, 0.f, 0.f, 0.f) : xin[q];
#pragma unroll
                for (int j8 = 0; j8 < 4; ++j8) {
                    float val[8];
                    const float4 x0 = xc[2 * j8], x1 = xc[2 * j8 + 1];
                    const float xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
                    __align__(16) __nv_bfloat16 hh[8], mm[8], ll[8];
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        const float cv = __uint_as_float(v[8 * j8 + t]);
                        val[t] = square ? cv : 2.0f * xs[t] - cv;
                        split_bf16(val[t], hh[t], mm[t], ll[t]);
                        const int64_t c = cbase + 8 * j8 + t;
                        const double dv = (double)val[t];
                        if (c == rl) {
                            tr += dv;
                            ss += dv * dv;
                        } else {
                            const int64_t m = (rb + c) * ld + rl;   // mirrored element
                            ss += 2.0 * dv * dv;
                            ep.out[m] = val[t];
                            ep.hi[m] = hh[t];
                            ep.lo[m] = mm[t];
                            if (w3) ep.lo2[m] = ll[t];
                        }
                    }
                    xo[2 * j8] = make_float4(val[0], val[1], val[2], val[3]);
                    xo[2 * j8 + 1] = make_float4(val[4], val[5], val[6], val[7]);
                    ho[j8] = *reinterpret_cast<const uint4*>(hh);
                    mo[j8] = *reinterpret_cast<const uint4*>(mm);
                    if (w3) lo[j8] = *reinterpret_cast<const uint4*>(ll);
                }
            } else {
                // chunk straddles the diagonal: scalar path, c >= r only
#pragma unroll 4
                for (int j = 0; j < 32; ++j) {
                    const int64_t c = cbase + j;
                    if (c < rl) continue;
                    const float cv = __uint_as_float(v[j]);
                    const float val = square ? cv : 2.0f * ep.xcur[r * ld + c] - cv;
                    __nv_bfloat16 h, m, l;
                    split_bf16(val, h, m, l);
                    const double dv = (double)val;
                    ep.out[r * ld + c] = val;
                    ep.hi[r * ld + c] = h;
                    ep.lo[r * ld + c] = m;
                    if (w3) ep.lo2[r * ld + c] = l;
                    if (c == rl) {
                        tr += dv;
                        ss += dv * dv;
                    } else {
                        const int64_t mi = (rb + c) * ld + rl;   // mirrored element
                        ss += 2.0 * dv * dv;
                        ep.out[mi] = val;
                        ep.hi[mi] = h;
                        ep.lo[mi] = m;
                        if (w3) ep.lo2[mi] = l;
                    }
                }
            }
        }
    }
    if (EPI == EPI_SP2) {
        for (int o = 16; o > 0; o >>= 1) {
            tr += __shfl_xor_sync(0xffffffffu, tr, o);
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
        }
        if (lane == 0) {
            red[2 * q] = tr;
            red[2 * q + 1] = ss;
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");   // epilogue warps only
        if (q == 0 && lane == 0) {
            ep.stats[2 * stat_index] = red[0] + red[2] + red[4] + red[6];
            ep.stats[2 * stat_index + 1] = red[1] + red[3] + red[5] + red[7];
        }
    }
}

template <int EPI, int BN, int NP, int KB>
__global__ void __launch_bounds__(THREADS, 1)
    k_tc_product(const __grid_constant__ TmaPlanes maps, const ProdList prods, const int2* __restrict__ tiles,
                 int nk, EpiParams ep) {
    // early exit of a converged system (uniform over the CTA)
    if (ep.active && ep.active[ep.stacked ? (int64_t)tiles[blockIdx.x].x * BM / ep.ld : 0] == 0) return;
    using C = Cfg<BN, NP, KB>;
    constexpr int STAGE_BYTES = C::STAGE_BYTES;
    constexpr int STAGES = C::STAGES;
    constexpr int A_TILE_BYTES = C::A_TILE_BYTES;
    constexpr int B_TILE_BYTES = C::B_TILE_BYTES;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t base_raw = smem_u32(smem_raw);
    const uint32_t base = (base_raw + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (base - base_raw);
    const uint32_t bar0 = base + STAGES * STAGE_BYTES;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (STAGES + s); };
    const uint32_t accum_bar = bar0 + 8u * (2 * STAGES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + STAGES * STAGE_BYTES + 8 * (2 * STAGES + 1));
    int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
    double* red = reinterpret_cast<double*>(gbase + STAGES * STAGE_BYTES + 128);   // 8 doubles

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int2 tile = tiles[blockIdx.x];
    const int bi = tile.x, bj = tile.y;

    auto a_tile = [&](int s, int p) { return base + s * STAGE_BYTES + p * A_TILE_BYTES; };
    auto b_tile = [&](int s, int p) {
        return base + s * STAGE_BYTES + NP * A_TILE_BYTES + p * B_TILE_BYTES;
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(accum_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"((uint32_t)BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // only the planes some product reads are loaded (the bytes the full barrier expects follow)
    uint32_t amask = 0, bmask = 0;
    for (int p = 0; p < prods.n; ++p) {
        amask |= 1u << prods.a[p];
        bmask |= 1u << prods.b[p];
    }
    const uint32_t stage_tx = (uint32_t)(__popc(amask) * A_TILE_BYTES + __popc(bmask) * B_TILE_BYTES);

    if (warp == 0 && lane == 0) {
        // ---------------- TMA producer ----------------
        int issued_phase[STAGES];
        for (int s = 0; s < STAGES; ++s) issued_phase[s] = -1;
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % STAGES, round = kb / STAGES;
            if (round > 0 && !mbar_wait(empty_bar(s), (round - 1) & 1)) {
                set_err(ep.err, 11);
                *(volatile int*)abort_flag = 1;
                break;
            }
            if (*(volatile int*)abort_flag) break;
            mbar_expect_tx(full_bar(s), stage_tx);
            for (int p = 0; p < NP; ++p)
                if ((amask >> p) & 1u) tma_load_2d(a_tile(s, p), &maps.a[p], full_bar(s), kb * KB, bi * BM);
            for (int p = 0; p < NP; ++p)
                if ((bmask >> p) & 1u) tma_load_2d(b_tile(s, p), &maps.b[p], full_bar(s), kb * KB, bj * BN);
            issued_phase[s] = round & 1;
        }
        // drain: every copy this thread issued has landed before the CTA may exit
        for (int s = 0; s < STAGES; ++s)
            if (issued_phase[s] >= 0 && !mbar_wait(full_bar(s), (uint32_t)issued_phase[s])) set_err(ep.err, 12);
    } else if (warp == 1 && lane == 0) {
        // ---------------- MMA issuer ----------------
        bool ok = true;
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % STAGES, round = kb / STAGES;
            if (!mbar_wait(full_bar(s), round & 1)) {
                set_err(ep.err, 21);
                *(volatile int*)abort_flag = 1;
                ok = false;
                break;
            }
            if (*(volatile int*)abort_flag) {
                ok = false;
                break;
            }
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < KB / 16; ++k) {
                for (int p = 0; p < prods.n; ++p) {
                    const uint64_t ad = sdesc(a_tile(s, prods.a[p]) + k * 32, C::SBO, C::SWIZZLE_LAYOUT);
                    const uint64_t bd = sdesc(b_tile(s, prods.b[p]) + k * 32, C::SBO, C::SWIZZLE_LAYOUT);
                    umma_bf16(tmem, ad, bd, C::IDESC, (kb | k | p) != 0);
                }
            }
            umma_commit(empty_bar(s));
        }
        umma_commit(accum_bar);   // also issued on abort so the wait below ends
        if (!ok) mbar_wait(accum_bar, 0);
    } else if (warp >= 4) {
        tc_epilogue<EPI, BN>(ep, tmem, accum_bar, abort_flag, red, bi, bj, warp - 4, lane, (int)blockIdx.x);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 2) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN));
    }
}

// ---- CTA-pair kernel (two planes) --------------------------------------------
// A cluster of two CTAs computes a 256 x 256 tile with cta_group::2 UMMA
// 256x256x16: CTA r holds rows 128r..128r+127 of A and of the accumulator, and
// columns 128r..128r+127 of the B operand, so every SM loads half the B panel
// of the one-CTA 128 x 256 tile: 1.5x fewer operand bytes per flop from L2.
// Each CTA's TMA loads count on the leader's (rank 0) "full" mbarrier, which
// the leader arms with both CTAs' bytes; the leader's single MMA thread issues
// the pair's MMAs and its commits arrive on the "empty" and accumulator
// barriers of both CTAs.  The epilogue is the one-CTA epilogue on each CTA's
// own 128 rows.
template <int NP, int KB>
struct CfgPair {
    static constexpr int A_TILE_BYTES = BM * KB * 2;          // this CTA's 128 rows of A
    static constexpr int B_TILE_BYTES = 128 * KB * 2;         // this CTA's 128 rows of B (half of N)
    static constexpr int STAGE_BYTES = NP * (A_TILE_BYTES + B_TILE_BYTES);
    static constexpr int STAGES = kSmemBudget / STAGE_BYTES > 6 ? 6 : kSmemBudget / STAGE_BYTES;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
    static constexpr uint32_t SWIZZLE_LAYOUT = KB == 64 ? 2u : 4u;
    static constexpr uint32_t SBO = KB == 64 ? 1024u : 512u;
    // kind::f16: D fp32, A/B bf16, K-major, M = 256 (the pair), N = 256
    static constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 3) << 17) |
                                      ((uint32_t)(256 >> 4) << 24);
    static_assert(KB == 64 || KB == 32, "K block of 64 or 32 elements");
    static_assert(STAGES >= 2, "at least two pipeline stages");
    static_assert(STAGE_BYTES % 1024 == 0, "stages keep the swizzle atoms aligned");
};

template <int EPI, int NP, int KB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
    k_tc_product_pair(const __grid_constant__ TmaPlanes maps, const ProdList prods, const int2* __restrict__ pairs,
                      int nk, EpiParams ep) {
    // early exit of a converged system: both CTAs of a pair hold rows of the same system
    if (ep.active && ep.active[ep.stacked ? (int64_t)pairs[blockIdx.x >> 1].x * 256 / ep.ld : 0] == 0) return;
    using C = CfgPair<NP, KB>;
    constexpr int STAGE_BYTES = C::STAGE_BYTES;
    constexpr int STAGES = C::STAGES;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t base_raw = smem_u32(smem_raw);
    const uint32_t base = (base_raw + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (base - base_raw);
    const uint32_t bar0 = base + STAGES * STAGE_BYTES;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (STAGES + s); };
    const uint32_t accum_bar = bar0 + 8u * (2 * STAGES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + STAGES * STAGE_BYTES + 8 * (2 * STAGES + 1));
    int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
    double* red = reinterpret_cast<double*>(gbase + STAGES * STAGE_BYTES + 128);   // 8 doubles

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int2 pt = pairs[blockIdx.x >> 1];
    const int bi = 2 * pt.x + (int)rank, bj = pt.y;   // this CTA's 128-row block; 256-column block

    auto a_tile = [&](int s, int p) { return base + s * STAGE_BYTES + p * C::A_TILE_BYTES; };
    auto b_tile = [&](int s, int p) { return base + s * STAGE_BYTES + NP * C::A_TILE_BYTES + p * C::B_TILE_BYTES; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(accum_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(256u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // both CTAs' barriers are initialised before any remote arrive
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    uint32_t amask = 0, bmask = 0;   // planes some product reads (both CTAs: the same list)
    for (int p = 0; p < prods.n; ++p) {
        amask |= 1u << prods.a[p];
        bmask |= 1u << prods.b[p];
    }
    const uint32_t stage_tx = (uint32_t)(__popc(amask) * C::A_TILE_BYTES + __popc(bmask) * C::B_TILE_BYTES);

    if (warp == 0 && lane == 0) {
        // ---------------- TMA producer (both CTAs) ----------------
        int issued_phase[STAGES];
        for (int s = 0; s < STAGES; ++s) issued_phase[s] = -1;
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % STAGES, round = kb / STAGES;
            if (round > 0 && !mbar_wait(empty_bar(s), (round - 1) & 1)) {
                set_err(ep.err, 41);
                *(volatile int*)abort_flag = 1;
                break;
            }
            if (*(volatile int*)abort_flag) break;
            if (rank == 0) mbar_expect_tx(full_bar(s), 2 * stage_tx);   // both CTAs' bytes
            const uint32_t fb = mapa_shared(full_bar(s), 0);
            for (int p = 0; p < NP; ++p)
                if ((amask >> p) & 1u) tma_load_2d_pair(a_tile(s, p), &maps.a[p], fb, kb * KB, bi * BM);
            for (int p = 0; p < NP; ++p)
                if ((bmask >> p) & 1u)
                    tma_load_2d_pair(b_tile(s, p), &maps.b[p], fb, kb * KB, bj * 256 + (int)rank * 128);
            issued_phase[s] = round & 1;
        }
        // drain: the leader sees every copy of the pair land on its full barriers;
        // the peer's copies have landed once the leader's MMAs consumed them,
        // which its accumulator barrier (waited by the epilogue) certifies
        if (rank == 0)
            for (int s = 0; s < STAGES; ++s)
                if (issued_phase[s] >= 0 && !mbar_wait(full_bar(s), (uint32_t)issued_phase[s]))
                    set_err(ep.err, 42);
    } else if (warp == 1 && lane == 0 && rank == 0) {
        // ---------------- MMA issuer (leader CTA) ----------------
        bool ok = true;
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % STAGES, round = kb / STAGES;
            if (!mbar_wait(full_bar(s), round & 1)) {
                set_err(ep.err, 51);
                *(volatile int*)abort_flag = 1;
                ok = false;
                break;
            }
            if (*(volatile int*)abort_flag) {
                ok = false;
                break;
            }
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < KB / 16; ++k) {
                for (int p = 0; p < prods.n; ++p) {
                    const uint64_t ad = sdesc(a_tile(s, prods.a[p]) + k * 32, C::SBO, C::SWIZZLE_LAYOUT);
                    const uint64_t bd = sdesc(b_tile(s, prods.b[p]) + k * 32, C::SBO, C::SWIZZLE_LAYOUT);
                    umma_bf16_pair(tmem, ad, bd, C::IDESC, (kb | k | p) != 0);
                }
            }
            umma_commit_pair(empty_bar(s), (uint16_t)0x3);
        }
        umma_commit_pair(accum_bar, (uint16_t)0x3);   // also on abort so the epilogues' waits end
        if (!ok) mbar_wait(accum_bar, 0);
    } else if (warp >= 4) {
        tc_epilogue<EPI, 256>(ep, tmem, accum_bar, abort_flag, red, bi, bj, warp - 4, lane, (int)blockIdx.x);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // the leader's MMAs have finished reading the peer's shared memory
    tc_fence_after();
    if (warp == 2) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u));
    }
}

// ---- host side ------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    PTB_CHECK(fn != nullptr, PTBGPU_ECUDA, "cuTensorMapEncodeTiled unavailable");
    return fn;
}

void encode_plane(CUtensorMap* map, const void* plane, int64_t ld, int64_t rows, int box_rows, int kb) {
    PTB_CHECK(((uintptr_t)plane & 15) == 0, PTBGPU_EINVAL, "operand plane not 16-byte aligned");
    PTB_CHECK(ld % 256 == 0, PTBGPU_EINVAL, "operand leading dimension must be a multiple of 256");
    cuuint64_t dims[2] = {(cuuint64_t)ld, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)kb, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUtensorMapSwizzle sw = kb == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    CUresult r = get_encode()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(plane), dims,
                              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    PTB_CHECK(r == CUDA_SUCCESS, PTBGPU_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
}

}  // namespace

int tile_n() { return 256; }

// Tile lists: row blocks of 128, column blocks of bn, grouped by 16 row
// blocks so that consecutive CTAs share operand panels in L2.
std::vector<int2> make_tiles(long long ld, bool upper_only, int bn) {
    const int nbi = (int)(ld / BM), nbj = (int)(ld / bn);
    std::vector<int2> t;
    const int G = 16;
    for (int g0 = 0; g0 < nbi; g0 += G)
        for (int bj = 0; bj < nbj; ++bj)
            for (int bi = g0; bi < std::min(nbi, g0 + G); ++bi)
                if (!upper_only || (int64_t)bj * bn + bn - 1 >= (int64_t)bi * BM) t.push_back(make_int2(bi, bj));
    return t;
}

// 256 x 256 tiles of the CTA-pair kernel, grouped by 8 tile rows.
std::vector<int2> make_pair_tiles(long long ld, bool upper_only) {
    const int nb = (int)(ld / 256);
    std::vector<int2> t;
    const int G = 8;
    for (int g0 = 0; g0 < nb; g0 += G)
        for (int pj = 0; pj < nb; ++pj)
            for (int pi = g0; pi < std::min(nb, g0 + G); ++pi)
                if (!upper_only || pj >= pi) t.push_back(make_int2(pi, pj));
    return t;
}

namespace {
template <int EPI, int BN, int NP, int KB>
void launch_t(cudaStream_t s, const TmaPlanes& maps, const ProdList& prods, const int2* tiles, int ntiles, int nk,
              const EpiParams& ep) {
    using C = Cfg<BN, NP, KB>;
    static const bool attr = [] {   // thread-safe one-time setup
        PTB_CUDA(cudaFuncSetAttribute(k_tc_product<EPI, BN, NP, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      C::SMEM_BYTES));
        return true;
    }();
    (void)attr;
    k_tc_product<EPI, BN, NP, KB><<<ntiles, THREADS, C::SMEM_BYTES, s>>>(maps, prods, tiles, nk, ep);
    count_launch();
}

template <int EPI, int KB>
void launch_pair(cudaStream_t s, const TmaPlanes& maps, const ProdList& prods, const int2* pairs, int npairs, int nk,
                 const EpiParams& ep) {
    using C = CfgPair<2, KB>;
    static const bool attr = [] {   // thread-safe one-time setup
        PTB_CUDA(cudaFuncSetAttribute(k_tc_product_pair<EPI, 2, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      C::SMEM_BYTES));
        return true;
    }();
    (void)attr;
    k_tc_product_pair<EPI, 2, KB><<<2 * npairs, THREADS, C::SMEM_BYTES, s>>>(maps, prods, pairs, nk, ep);
    count_launch();
}

template <int EPI>
void launch_epi(cudaStream_t s, int np, int kb, bool pair, bool narrow, const TmaPlanes& maps, const ProdList& prods,
                const int2* tiles, int ntiles, int nk, const EpiParams& ep) {
    if (pair) {
        if (kb == 64) launch_pair<EPI, 64>(s, maps, prods, tiles, ntiles, nk, ep);
        else launch_pair<EPI, 32>(s, maps, prods, tiles, ntiles, nk, ep);
    } else if (narrow) {
        launch_t<EPI, 128, 2, 64>(s, maps, prods, tiles, ntiles, nk, ep);
    } else if (np == 2) {
        if (kb == 64) launch_t<EPI, 256, 2, 64>(s, maps, prods, tiles, ntiles, nk, ep);
        else launch_t<EPI, 256, 2, 32>(s, maps, prods, tiles, ntiles, nk, ep);
    } else {
        if (kb == 64) launch_t<EPI, 128, 3, 64>(s, maps, prods, tiles, ntiles, nk, ep);
        else launch_t<EPI, 128, 3, 32>(s, maps, prods, tiles, ntiles, nk, ep);
    }
}

// Autotuned kernel choice per (device, epilogue, planes, leading dimension):
// the first launch of a shape runs every candidate (K block 64 / 32, one CTA
// or a CTA pair where pair tiles are given) back to back -- same inputs, same
// outputs, so running them all is harmless -- times them with CUDA events and
// keeps the fastest for the rest of the process.
std::mutex g_tune_mu;
std::map<std::tuple<int, int, int, long long, long long>, int> g_tuned;
}  // namespace

int tuned_kblock(int epi, int np, long long ld, long long rows) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(g_tune_mu);
    auto it = g_tuned.find(std::make_tuple(dev, epi, np, ld, rows == 0 ? ld : rows));
    return it == g_tuned.end() ? 0 : it->second;
}

int launch_product(cudaStream_t s, int epi, int np, long long ld, const void* const* a, const void* const* b,
                   const ProdList& prods, const int2* tiles_dev, int ntiles, const EpiParams& ep, int kblock,
                   const int2* pairs_dev, int npairs, long long rows) {
    if (rows == 0) rows = ld;
    PTB_CHECK(rows % ld == 0 && (ep.stacked || rows == ld), PTBGPU_EINVAL,
              "stacked planes: rows must be a multiple of ld and the epilogue told so");
    PTB_CHECK(np == 2 || np == 3, PTBGPU_EINVAL, "unsupported plane count %d", np);
    PTB_CHECK(kblock == 0 || kblock == 32 || kblock == 64 || kblock == kPairKernel + 32 ||
                  kblock == kPairKernel + 64 || kblock == kNarrowKernel,
              PTBGPU_EINVAL, "bad kernel choice %d", kblock);
    const bool narrow = kblock == kNarrowKernel;
    PTB_CHECK(!narrow || np == 2, PTBGPU_EINVAL, "the 128-column kernel takes two planes");
    PTB_CHECK(narrow || kblock < kPairKernel || (np == 2 && pairs_dev != nullptr), PTBGPU_EINVAL,
              "the CTA-pair kernel needs two planes and pair tiles");
    PTB_CHECK(ld % 256 == 0, PTBGPU_EINVAL, "leading dimension must be a multiple of 256");
    const int bn = np == 2 && !narrow ? 256 : 128;
    PTB_CHECK(prods.n >= 1 && prods.n <= 6, PTBGPU_EINVAL, "1 to 6 plane products (got %d)", prods.n);
    for (int p = 0; p < prods.n; ++p)
        PTB_CHECK(prods.a[p] >= 0 && prods.a[p] < np && prods.b[p] >= 0 && prods.b[p] < np, PTBGPU_EINVAL,
                  "product references a missing plane");
    PTB_CHECK(epi != EPI_SP2 || (ep.hi != nullptr && ep.lo != nullptr), PTBGPU_EINVAL,
              "the SP2 epilogue writes at least two planes");
    // returns the number of per-CTA stats partials the launch writes
    auto run = [&](int choice) {
        const bool pair = choice >= kPairKernel && !narrow;
        const int kb = narrow ? 64 : pair ? choice - kPairKernel : choice;
        TmaPlanes maps;
        for (int p = 0; p < np; ++p) {
            encode_plane(&maps.a[p], a[p], ld, rows, BM, kb);
            encode_plane(&maps.b[p], b[p], ld, rows, pair ? 128 : bn, kb);
        }
        const int nk = (int)(ld / kb);
        const int2* t = pair ? pairs_dev : tiles_dev;
        const int nt = pair ? npairs : ntiles;
        if (epi == EPI_SP2) launch_epi<EPI_SP2>(s, np, kb, pair, narrow, maps, prods, t, nt, nk, ep);
        else launch_epi<EPI_FULL>(s, np, kb, pair, narrow, maps, prods, t, nt, nk, ep);
        PTB_CUDA(cudaGetLastError());
        return pair ? 2 * npairs : ntiles;
    };
    if (kblock == 0) kblock = tuned_kblock(epi, np, ld, rows);
    if (kblock != 0 && (narrow || kblock < kPairKernel || pairs_dev)) return run(kblock);
    std::vector<int> cand = {64, 32};
    if (np == 2 && pairs_dev) {
        cand.push_back(kPairKernel + 64);
        cand.push_back(kPairKernel + 32);
    }
    std::vector<cudaEvent_t> e(cand.size() + 1);
    for (auto& x : e) PTB_CUDA(cudaEventCreate(&x));
    int parts = 0;
    PTB_CUDA(cudaEventRecord(e[0], s));
    for (size_t i = 0; i < cand.size(); ++i) {
        parts = run(cand[i]);
        PTB_CUDA(cudaEventRecord(e[i + 1], s));
    }
    PTB_CUDA(cudaEventSynchronize(e.back()));
    int best = cand[0];
    float tbest = 1e30f;
    for (size_t i = 0; i < cand.size(); ++i) {
        float t = 0.f;
        PTB_CUDA(cudaEventElapsedTime(&t, e[i], e[i + 1]));
        if (t < tbest) {
            tbest = t;
            best = cand[i];
        }
    }
    for (auto& x : e) cudaEventDestroy(x);
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_tuned[std::make_tuple(dev, epi, np, ld, rows)] = best;
    return parts;   // the buffers hold the last candidate's results
}

}  // namespace tc
}  // namespace ptb
