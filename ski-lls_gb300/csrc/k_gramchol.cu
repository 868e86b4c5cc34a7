// k_gramchol.cu -- preconditioner of a well-conditioned sketch from its Gram
// matrix: G = (S A)^T (S A), Cholesky G = R^T R and M = R^{-1} in one blocked
// sweep, and the explicit sketch solution's coefficients c.
//
// Pivoting a QR serves one purpose in the solve: finding the numerical rank
// (rnpre_sparse, src/ls_sparse_spqr.cpp:20-75, and the |R_ii| > rcond rule of
// src/ls_dense_hashing_blendenpik.cpp:79-89).  It is also what the pivoted
// factorization spends its time on: a chain of dependent 64-column panels
// (sample pivoting, column moves, CholeskyQR2) at ~330 us each.  When the
// sketch is well conditioned every pivot order finds rank d, and that can be
// proven afterwards from M:
//   * |R_ii| >= sigma_min(S A) >= 1 / ||M||_F for every pivot of every column
//     order, and |R_00| <= max_j ||S A e_j||, so 1 / ||M||_F > the rank rule's
//     threshold means that the pivoted factorization keeps all columns;
//   * Cholesky of a Gram matrix loses the square of the condition number, so
//     eps ||M D||_F^2 <= 1/16 is asked for as well (D = diag(||S A e_j||), which
//     makes the bound independent of the column scaling, as Cholesky is): R is
//     then within a few percent of an orthogonal change of basis of the QR's
//     R, far inside what moves LSQR's iteration count.
// Columns whose pivot falls below 2048 eps of their mass are dropped from the
// sweep (zero row and column of M) where the caller carries such columns in
// LSQR's basis (the mixed sparse path); the small singular values they stand
// for, taken from S A itself, must then lie below a quarter of the rank rule's
// threshold, as the pivoted factorization's trailing pivots would.
// On the dense mixed path a failed pivot is raised to the bound instead and the
// same is done again on Q = S A M (at most twice): each pass takes the condition
// number to about the root of what exceeds ~300.  40,000 x 4,000 (S A 6,800 x 4,000):
// QR and inverse 20.2 + 1.4 ms, one pass ~3.3 ms, two (condition number 1e3 to
// 1e4) 7.4 ms, three (to 1e6) 11.4 with LSQR's iterations, x and residual unchanged.
// From ~3e6 on at that size (12,007 x 1,201: 1e7) M is too large for the rank proof,
// and the QR comes on top of two passes.
// The sparse path takes the later passes where no pivot failed but the bound on M D
// does, or where the dropped columns are all at least four thresholds away from
// dependence (120,000 x 5,000, S A 8,500 x 5,000: 11.2 and 16 to 19 ms; the QR and
// inverse 26.9 + 2 ms).  Columns between a quarter of the threshold and four of
// them, and more than 512 failed pivots, end in the QR after an attempt of 0.2 to
// 7.5 ms.
// A sketch that fails a test keeps the QR: S A is not touched here.
//
// Sweep (outer blocks of 256 rows, inner blocks of 64): the same row
// operations that turn G into R turn I into E = R^{-T}, so one trailing update
// per block carries both:
//   diag    R_ss, X_s = R_ss^{-1} of a 64-block (one CTA), then one launch for
//           the block row and the updates inside the 256-block (k_gc_step)
//   row     [R_k* | E_k*] = M_kk^T [G_k* | E'_k*]     (K = 256)
//   update  [G | E'] -= R_k*^T [R_k* | E_k*]          (K = 256, upper tiles)
// All three are products A^T B with both operands contiguous along K.  FP32:
// tcgen05 (k_tc_tn); FP64: k_gemm.  E column-major is M row-major, the layout
// the LSQR's forward product reads; M column-major is its transpose.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <mutex>
#include <type_traits>

#include "skl_internal.hpp"
#include "launch.cuh"
#include "common.cuh"
#include "k_gemm.cuh"
#include "chol_small.cuh"
#include "tc_ptx.cuh"

namespace skl {

using namespace tc;

namespace {

constexpr int kOB = 256;   // outer block
constexpr int kIB = 64;    // inner block

// ---- C = alpha A^T B + beta C on the tensor cores (FP32, 3xTF32) -------------
// 128 x 128 tiles of C, one per CTA; K in stages of 32 rows.  Both operands
// are column-major with K contiguous, loaded by TMA with the 128-byte swizzle
// and split into hi and lo TF32 parts: A's go to tensor memory, from where the
// MMAs take them, B's stay in shared memory (hi in place).  The accumulator lives
// in tensor memory for 64 rows of K and is then added into registers, because the
// tensor core's own FP32 accumulation over thousands of rows is several times
// less accurate than FP32 adds.  A stage is 12 MMAs of 128 x 128 x 8 (~768
// cycles) against ~1,125 cycles of shared-memory traffic (TMA write, split, MMA
// reads of B); with A's parts in shared memory too that was ~1,750.  The Gram
// matrix of 15,000 x 10,000: 7.5 ms, 1,500 cycles a stage; 1,990 with A in shared
// memory, 1,650 with conversions instead of integer rounding for the hi parts.
constexpr int kNT = 128;
constexpr int kNStages = 4;
constexpr int kNTile = kNT * kBK * 4;               // 16 KB
constexpr int kNStage = 3 * kNTile;                 // A, B (then its hi), B lo
constexpr int kNThreads = 512;                      // producer, MMA, 6 splitter, 8 drainer warps
constexpr int kNSplit = 192;                        // splitter threads (16 warps in all: 128 registers each)
constexpr int kNGroup = 2;                          // stages per accumulation
constexpr int kNSmem = kNStages * kNStage + 1024 + 1024;
constexpr unsigned kNTmemCols = 2 * kNT + kNStages * 2 * kBK;   // accumulators; A hi and lo by stage

// Output tiles: blockIdx.y = row tile, blockIdx.x = column tile, first nE tiles
// of the E part (columns from 0), then the G part (columns from g0).  A row
// tile covers A's columns a0 + 128 y and C's rows r0 + 128 y.
struct TnArgs {
    int kA, kB, nkb;        // first K row in A's and in B's map, stages
    int a0, r0, g0, nE;
    int rows, cols;         // C is written for row < rows, column < cols
    int cols_e;             // E part: columns < cols_e
    int e_add;              // E part: tiles below this index add to C, others overwrite
    int g_add;              // G part adds to C
    int upper;              // skip G tiles that lie below the diagonal
    int tri;                // 1: B is upper triangular (K ends at the tile's last column);
                            // 2: A^T is too (K starts at the tile's first row)
    float alpha;
    float* Cg; int64_t ldg;
    float* Ce; int64_t lde;
};

__global__ void __launch_bounds__(kNThreads, 1)
k_tc_tn(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapBg,
        const __grid_constant__ CUtensorMap mapBe, const TnArgs t, const int* __restrict__ bad,
        unsigned* __restrict__ status)
{
    pdl_wait();
    const bool is_e = (int)blockIdx.x < t.nE;
    const int row0 = t.r0 + blockIdx.y * kNT;
    const int col0 = is_e ? (int)blockIdx.x * kNT : t.g0 + ((int)blockIdx.x - t.nE) * kNT;
    if (!is_e && t.upper && col0 < row0) return;
    __shared__ int s_bad;
    if (threadIdx.x == 0) s_bad = bad ? *bad : 0;
    __syncthreads();
    if (s_bad) return;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kNStages * kNStage);
    // bars: full, conv, empty [kNStages each], tfull[2], tempty[2], done; then the TMEM address
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 3 * kNStages + 5);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kb0 = t.tri == 2 ? row0 / kBK : 0;
    const int nkb = (t.tri ? min(t.nkb, (col0 + kNT) / kBK) : t.nkb) - kb0;
    const int ngroups = (nkb + kNGroup - 1) / kNGroup;
    auto full = [&](int s) { return smem_u32(bars + s); };
    auto conv = [&](int s) { return smem_u32(bars + kNStages + s); };
    auto empty = [&](int s) { return smem_u32(bars + 2 * kNStages + s); };
    auto tfull = [&](int q) { return smem_u32(bars + 3 * kNStages + q); };
    auto tempty = [&](int q) { return smem_u32(bars + 3 * kNStages + 2 + q); };
    const unsigned done = smem_u32(bars + 3 * kNStages + 4);
    auto raw_a = [&](int s) { return smem + s * kNStage; };
    auto hi_b = [&](int s) { return smem + s * kNStage + kNTile; };
    auto lo_b = [&](int s) { return smem + s * kNStage + 2 * kNTile; };
    auto tmem_a = [&](unsigned base, int s) { return base + 2 * kNT + (unsigned)(s * 2 * kBK); };   // hi, then lo

    if (threadIdx.x == 0) {
        for (int s = 0; s < kNStages; ++s) {
            mbar_init(full(s), 1);
            mbar_init(conv(s), kNSplit);
            mbar_init(empty(s), 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(tfull(q), 1);
            mbar_init(tempty(q), 256);
        }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kNTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            const CUtensorMap* mapB = is_e ? &mapBe : &mapBg;
            bool ok = true;
            int issued = 0;
            for (int kb = 0; kb < nkb && ok; ++kb) {
                const int s = kb % kNStages;
                if (kb >= kNStages) ok = mbar_wait(empty(s), ((kb / kNStages) - 1) & 1, status);
                if (!ok) break;
                mbar_expect_tx(full(s), 2 * kNTile);
                tma_load_2d(smem_u32(raw_a(s)), &mapA, t.kA + (kb0 + kb) * kBK, t.a0 + blockIdx.y * kNT, full(s));
                tma_load_2d(smem_u32(hi_b(s)), mapB, t.kB + (kb0 + kb) * kBK, col0, full(s));
                ++issued;
            }
            // the copies this CTA issued have landed before it may exit
            for (int kb = std::max(0, issued - kNStages); kb < issued; ++kb)
                mbar_wait(full(kb % kNStages), (kb / kNStages) & 1, status);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = tf32_idesc(kNT, kNT);
            bool ok = true;
            for (int kb = 0; kb < nkb && ok; ++kb) {
                const int s = kb % kNStages;
                const int g = kb / kNGroup, buf = g & 1;
                const bool first = (kb % kNGroup) == 0;
                if (first && g >= 2) ok = mbar_wait(tempty(buf), ((g >> 1) - 1) & 1, status);
                if (ok) ok = mbar_wait(conv(s), (kb / kNStages) & 1, status);
                if (!ok) break;
                tc_fence_after();
                const unsigned d = tmem + (unsigned)(buf * kNT);
                const unsigned ah = tmem_a(tmem, s), al = ah + kBK;
                const unsigned bh = smem_u32(hi_b(s)), bl = smem_u32(lo_b(s));
#pragma unroll
                for (int k8 = 0; k8 < kBK / 8; ++k8) {
                    const unsigned off = k8 * 32;   // 8 TF32 values along K
                    mma_tf32_ta(d, al + k8 * 8, sw128_desc(bh + off), idesc, (first && k8 == 0) ? 0u : 1u);
                    mma_tf32_ta(d, ah + k8 * 8, sw128_desc(bl + off), idesc, 1u);
                    mma_tf32_ta(d, ah + k8 * 8, sw128_desc(bh + off), idesc, 1u);
                }
                mma_commit(empty(s));
                if ((kb % kNGroup) == kNGroup - 1 || kb == nkb - 1) mma_commit(tfull(buf));
            }
            // every MMA issued here has completed before the TMEM is freed
            mma_commit(done);
            mbar_wait(done, 0, status);
        }
    } else if (warp < 8) {
        // warps 2..7 split into hi / lo.  Warps 4..7: their quadrant's 32 rows of A
        // to tensor memory; warps 2 to 5 share B's 32 groups of 32 float4.
        constexpr int kShare = 6;   // of warps 4, 5, whose schedulers have no other splitter
        const int quad = warp & 3;
        const int g0 = warp < 4 ? 2 * kShare + (warp - 2) * (16 - kShare) : warp < 6 ? (warp - 4) * kShare : 0;
        const int ng = warp < 4 ? 16 - kShare : warp < 6 ? kShare : 0;
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % kNStages;
            if (!__all_sync(0xffffffffu, mbar_wait(full(s), (kb / kNStages) & 1, status))) break;
            if (warp >= 4) {
                tc_fence_after();
                const unsigned char* rowp = raw_a(s) + (quad * 32 + lane) * 128;
                float h[kBK], l[kBK];
#pragma unroll
                for (int c = 0; c < kBK / 4; ++c) {
                    const float4 v = *reinterpret_cast<const float4*>(rowp + ((c ^ (lane & 7)) << 4));
                    const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        h[4 * c + q] = tf32_hi_int(x[q]);
                        l[4 * c + q] = tf32_hi(x[q] - h[4 * c + q]);
                    }
                }
                const unsigned ta = tmem_a(tmem, s) + ((unsigned)(quad * 32) << 16);
                tmem_st32(ta, h);
                tmem_st32(ta + kBK, l);
            }
            float4* h = reinterpret_cast<float4*>(hi_b(s)) + g0 * 32 + lane;
            float4* l = reinterpret_cast<float4*>(lo_b(s)) + g0 * 32 + lane;
#pragma unroll 4
            for (int e = 0; e < ng; ++e) {
                const float4 v = h[e * 32];
                float4 a, b;
                a.x = tf32_hi_int(v.x); b.x = tf32_hi(v.x - a.x);
                a.y = tf32_hi_int(v.y); b.y = tf32_hi(v.y - a.y);
                a.z = tf32_hi_int(v.z); b.z = tf32_hi(v.z - a.z);
                a.w = tf32_hi_int(v.w); b.w = tf32_hi(v.w - a.w);
                h[e * 32] = a;
                l[e * 32] = b;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (warp >= 4) {
                tmem_st_wait();
                tc_fence_before();
            }
            mbar_arrive(conv(s));
        }
    } else {
        // warps 8..15: this warp's 32-lane quadrant = 32 rows of C, `half` =
        // which 64 of the tile's columns
        const int quad = warp & 3;
        const int half = (warp - 8) >> 2;
        float sum[64];
#pragma unroll
        for (int q = 0; q < 64; ++q) sum[q] = 0.f;
        bool ok = true;
        for (int g = 0; g < ngroups; ++g) {
            const int buf = g & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(tfull(buf), (g >> 1) & 1, status));
            if (!ok) break;   // warp-uniform: tcgen05.ld is warp-collective
            tc_fence_after();
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                float v[32];
                tmem_ld32(tmem + ((unsigned)(quad * 32) << 16) + (unsigned)(buf * kNT + half * 64 + p * 32), v);
#pragma unroll
                for (int q = 0; q < 32; ++q) sum[p * 32 + q] += v[q];
            }
            tc_fence_before();
            mbar_arrive(tempty(buf));
        }
        const int row = row0 + quad * 32 + lane;
        const int cb = col0 + half * 64;
        if (ok && row < t.rows) {
            const int nc = min(64, (is_e ? t.cols_e : t.cols) - cb);
            const int64_t ldc = is_e ? t.lde : t.ldg;
            float* c = (is_e ? t.Ce : t.Cg) + row + (int64_t)cb * ldc;
            const bool add = is_e ? (int)blockIdx.x < t.e_add : t.g_add != 0;
            if (add) {
#pragma unroll
                for (int p = 0; p < 64; p += 16) {
                    float old[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) old[q] = p + q < nc ? c[(p + q) * ldc] : 0.f;
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        if (p + q < nc) c[(p + q) * ldc] = fmaf(t.alpha, sum[p + q], old[q]);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 64; ++q)
                    if (q < nc) c[q * ldc] = t.alpha * sum[q];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kNTmemCols)
                     : "memory");
    }
}

// ---- the 64 x 64 diagonal block ----------------------------------------------
// diag(G), saved before the sweep overwrites it (also the pivots' masses, but
// for the columns an earlier attempt excluded: first = 0 keeps an infinite
// mass, which fails every pivot); the identity column order
template <typename T>
__global__ void k_gc_init(const T* __restrict__ G, int64_t ldg, int d, T* __restrict__ gdiag,
                          T* __restrict__ mass, int first, T* __restrict__ mkk, int* __restrict__ jpvt,
                          int* __restrict__ bad, int* __restrict__ ndrop)
{
    pdl_wait();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e == 0) *bad = *ndrop = 0;
    for (int j = e; j < d; j += gridDim.x * blockDim.x) {
        const T v = G[j + (int64_t)j * ldg];
        gdiag[j] = v;
        if (first || !(mass[j] > std::numeric_limits<T>::max())) mass[j] = v;
        jpvt[j] = j;
    }
    for (int j = e; j < kOB * kOB; j += gridDim.x * blockDim.x) mkk[j] = T(0);
}

// What the sweep's small kernels share.
template <typename T>
struct GcArgs {
    T* G; T* R; int64_t ldg;
    T* Ew; T* E; int64_t lde;
    T* mkk;                 // inverse of the 256-block (ld 256), column-major
    const T* mass;          // a pivot is measured against its column's entry
    int* bad; int* ndrop; int* drop; int drop_cap;
    int d;
    T pivot;                // pivots at or below pivot * mass fail
    int boost;              // a failed pivot becomes that bound (counted in ndrop)
};

constexpr int kSL = kIB + 4;   // row-major 64 x 64 shared-memory blocks

// rows r0.., columns c0.. of a column-major matrix (zeros outside nr x nc) to S[row][col]
template <typename T>
SKL_DEV void tile_load(const T* __restrict__ X, int64_t ld, int r0, int c0, int nr, int nc, T* S)
{
#pragma unroll
    for (int q = 0; q < kIB * kIB / kSmallThreads; ++q) {
        const int e = threadIdx.x + q * kSmallThreads;
        const int r = e % kIB, c = e / kIB;
        S[r * kSL + c] = (r < nr && c < nc) ? X[(r0 + r) + (int64_t)(c0 + c) * ld] : T(0);
    }
}

// V -= U^T U (64 x 64).  FP64: 2 x 2 tiles of the upper triangle on 17 full warps,
// mirrored: the FP64 pipe bounds it (134,000 cycles with all tiles).
template <typename T>
SKL_DEV void sub_gram(const T* U, T* V)
{
    if constexpr (std::is_same<T, float>::value) {
        blk_mul<T, true, kMFull, false, kMFull, true>(kIB, kIB, kIB, U, kSL, U, kSL, nullptr, T(-1), V, kSL);
    } else {
        // tile t of the triangle: row i of tiles holds columns i .. 31
        int t = threadIdx.x, i = 0;
        if (t < 32 * 33 / 2) {
            while (t >= 32 - i) t -= 32 - i++;
            const int r0 = 2 * i, c0 = 2 * (i + t);
            T a00 = 0, a01 = 0, a10 = 0, a11 = 0;
#pragma unroll 4
            for (int k = 0; k < kIB; ++k) {
                const T x0 = U[k * kSL + r0], x1 = U[k * kSL + r0 + 1];
                const T y0 = U[k * kSL + c0], y1 = U[k * kSL + c0 + 1];
                a00 += x0 * y0;
                a01 += x0 * y1;
                a10 += x1 * y0;
                a11 += x1 * y1;
            }
            auto sub = [&](int r, int c, T v) {
                const T w = V[r * kSL + c] - v;
                V[r * kSL + c] = w;
                V[c * kSL + r] = w;
            };
            sub(r0, c0, a00);
            sub(r0, c0 + 1, a01);
            if (c0 > r0) sub(r0 + 1, c0, a10);
            sub(r0 + 1, c0 + 1, a11);
        }
        __syncthreads();
    }
}

// R_ss and X = R_ss^{-1} of the b x b (b <= 64) diagonal block S0 (symmetric,
// identity beyond b) at row q: R to R, X^T to E, X to mkk at offset ql.  A
// failed pivot drops the column: its row of
// R and its row and column of X are zero, so that the sweep runs on as if the
// column were not there, and its index joins the list; more than drop_cap of
// them set *bad.
template <typename T>
SKL_DEV void diag_block(const GcArgs<T>& g, int q, int b, int ql, T* S0, T* S1, T* mass)
{
    __shared__ int s_any;
    const int np = small_np(b);
    if (threadIdx.x == 0) s_any = 0;
    for (int k = threadIdx.x; k < np; k += kSmallThreads) mass[k] = k < b ? g.mass[q + k] : T(1);
    __syncthreads();
    // chol_inv_small asks for a pivot above 32 x its eps x mass
    if (g.boost) chol_inv_small<T, true>(S0, kSL, np, mass, g.pivot / T(32), S1, &s_any);
    else chol_inv_small<T>(S0, kSL, np, mass, g.pivot / T(32), S1, &s_any);
    for (int e = threadIdx.x; e < b * b; e += kSmallThreads) {
        const int i = e % b, c = e / b;
        g.R[(q + i) + (int64_t)(q + c) * g.ldg] = S0[i * kSL + c];
        g.mkk[(ql + i) + (ql + c) * kOB] = S1[i * kSL + c];
        g.E[(q + i) + (int64_t)(q + c) * g.lde] = S1[c * kSL + i];
    }
    if (g.boost) {
        if (threadIdx.x == 0 && s_any) {
            *g.ndrop = 1;
            if (s_any > 1) *g.bad = 1;   // a zero (or NaN) column
        }
        return;
    }
    if (s_any && threadIdx.x < 32) {
        int n = *g.ndrop;
        for (int h = 0; h < 2; ++h) {
            const int k = h * 32 + (int)threadIdx.x;
            const bool z = k < b && S0[k * kSL + k] == T(0);
            const unsigned m = __ballot_sync(0xffffffffu, z);
            const int at = n + __popc(m & ((1u << threadIdx.x) - 1u));
            if (z && at < g.drop_cap) g.drop[at] = q + k;
            n += __popc(m);
        }
        __syncwarp();
        if (threadIdx.x == 0) {
            *g.ndrop = n;
            if (n > g.drop_cap) *g.bad = 1;
        }
    }
}

// The first diagonal block of a 256-block.
template <typename T>
__global__ void __launch_bounds__(kSmallThreads, 1) k_gc_diag(const GcArgs<T> g, int q, int b)
{
    pdl_wait();
    __shared__ int s_bad;
    if (threadIdx.x == 0) s_bad = *g.bad;
    __syncthreads();
    if (s_bad) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* S0 = (T*)smem_raw;
    T* S1 = S0 + kIB * kSL;
    // both triangles from G's upper one, identity beyond b
    for (int e = threadIdx.x; e < kIB * kIB; e += kSmallThreads) {
        const int i = e % kIB, c = e / kIB;
        if (i > c) continue;
        const T v = c < b ? g.G[(q + i) + (int64_t)(q + c) * g.ldg] : (i == c ? T(1) : T(0));
        S0[i * kSL + c] = v;
        S0[c * kSL + i] = v;
    }
    diag_block<T>(g, q, b, 0, S0, S1, S1 + kIB * kSL);
}

// ---- one inner step of a 256-block ---------------------------------------------
// With X = R_ss^{-1} of inner block s: the block row R(s, J) = X^T G(s, J)
// (J > s) and E(s, J) = X^T E'(s, J) (J < s), the updates
// G(I, J) -= R(s, I)^T R(s, J), E'(I, J) -= R(s, I)^T E(s, J) of the rows I > s
// inside the 256-block, and (CTA 0) the factorization of the next diagonal
// block, which needs only its own update.  One CTA per 64 x 64 target; an
// update forms the block-row factors it needs itself (64^3 products on the
// warps' tensor cores) instead of waiting for a second launch, so the chain is
// one launch per 64 columns, bound by CTA 0: 20.7 us, of 40,000 cycles half the
// block's elimination (FP64: 125 us, 243 before its products kept to triangles).
template <typename T>
__global__ void __launch_bounds__(kSmallThreads, 1) k_gc_step(const GcArgs<T> g, int j0, int s, int nb)
{
    pdl_wait();
    __shared__ int s_bad;
    if (threadIdx.x == 0) s_bad = *g.bad;
    __syncthreads();
    if (s_bad) return;
    // block index -> (I, J): the next diagonal block, the nb - 1 blocks of row s,
    // then the updates row by row (E' columns 0..s, G columns I..nb-1 without
    // the next diagonal block)
    int I, J, t = blockIdx.x;
    bool is_e = false, diag = false;
    if (s + 1 < nb && t == 0) {
        I = J = s + 1;
        diag = true;
    } else {
        t -= s + 1 < nb ? 1 : 0;
        if (t < nb - 1) {
            I = s;
            J = t < s ? t : t + 1;
            is_e = J < s;
        } else {
            t -= nb - 1;
            for (I = s + 1; I < nb; ++I) {
                const int w = s + 1 + nb - I - (I == s + 1 ? 1 : 0);
                if (t < w) break;
                t -= w;
            }
            is_e = t <= s;
            J = is_e ? t : I + (t - s - 1) + (I == s + 1 ? 1 : 0);
        }
    }
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* X = (T*)smem_raw;
    T* P = X + kIB * kSL;
    T* U = P + kIB * kSL;
    T* V = U + kIB * kSL;
    const int q = j0 + s * kIB;
    auto width = [&](int blk) { return min(kIB, g.d - (j0 + blk * kIB)); };
    const int bs = width(s), bI = width(I), bJ = width(J);
    const int cI = j0 + I * kIB, cJ = j0 + J * kIB;
    tile_load<T>(g.mkk, kOB, s * kIB, s * kIB, bs, bs, X);
    if (diag) {
        tile_load<T>(g.G, g.ldg, q, cI, bs, bI, P);
        // the block itself: both triangles from the upper one, identity beyond bI
        for (int e = threadIdx.x; e < kIB * kIB; e += kSmallThreads) {
            const int i = e % kIB, c = e / kIB;
            if (i > c) continue;
            const T v = c < bI ? g.G[(cI + i) + (int64_t)(cI + c) * g.ldg] : (i == c ? T(1) : T(0));
            V[i * kSL + c] = v;
            V[c * kSL + i] = v;
        }
        __syncthreads();
        blk_mul<T, true, kMLower, false, kMFull>(kIB, kIB, kIB, X, kSL, P, kSL, nullptr, T(1), U, kSL);
        sub_gram<T>(U, V);
        diag_block<T>(g, cI, bI, I * kIB, V, P, V + kIB * kSL);
        return;
    }
    // V = row s of the target's columns
    if (is_e && J == s) {
        __syncthreads();
        for (int e = threadIdx.x; e < kIB * kIB; e += kSmallThreads)
            V[(e / kIB) * kSL + e % kIB] = X[(e % kIB) * kSL + e / kIB];   // E(s, s) = X^T
    } else {
        tile_load<T>(is_e ? g.Ew : g.G, is_e ? g.lde : g.ldg, q, cJ, bs, bJ, P);
        __syncthreads();
        blk_mul<T, true, kMLower, false, kMFull>(kIB, kIB, kIB, X, kSL, P, kSL, nullptr, T(1), V, kSL);
    }
    if (I == s) {
        for (int e = threadIdx.x; e < kIB * kIB; e += kSmallThreads) {
            const int r = e % kIB, c = e / kIB;
            if (r >= bs || c >= bJ) continue;
            const T v = V[r * kSL + c];
            if (is_e) {
                g.E[(q + r) + (int64_t)(cJ + c) * g.lde] = v;
                g.mkk[(J * kIB + c) + (s * kIB + r) * kOB] = v;
            } else {
                g.R[(q + r) + (int64_t)(cJ + c) * g.ldg] = v;
                g.E[(q + r) + (int64_t)(cJ + c) * g.lde] = T(0);
            }
        }
        return;
    }
    // U = R(s, I), then P = U^T V
    const T* u = V;
    if (is_e || I != J) {
        __syncthreads();
        tile_load<T>(g.G, g.ldg, q, cI, bs, bI, P);
        __syncthreads();
        blk_mul<T, true, kMLower, false, kMFull>(kIB, kIB, kIB, X, kSL, P, kSL, nullptr, T(1), U, kSL);
        u = U;
    }
    blk_mul<T, true, kMFull, false, kMFull>(kIB, kIB, kIB, u, kSL, V, kSL, nullptr, T(1), P, kSL);
    T* C = is_e ? g.Ew : g.G;
    const int64_t ldc = is_e ? g.lde : g.ldg;
    const bool add = !(is_e && J == s);
    for (int e = threadIdx.x; e < kIB * kIB; e += kSmallThreads) {
        const int r = e % kIB, c = e / kIB;
        if (r >= bI || c >= bJ) continue;
        T* p = C + (cI + r) + (int64_t)(cJ + c) * ldc;
        *p = add ? *p - P[r * kSL + c] : -P[r * kSL + c];
    }
}

// ---- M column-major from E (= M row-major); norms --------------------------------
// Also per-block sums of M(i, j)^2 and gdiag[i] M(i, j)^2.
constexpr int kTrTile = 64;
template <typename T>
__global__ void __launch_bounds__(256)
k_gc_transpose(const T* __restrict__ E, int64_t lde, int d, T* __restrict__ M, int64_t ldm,
               const T* __restrict__ gdiag, double* __restrict__ part, const int* __restrict__ bad)
{
    pdl_wait();
    __shared__ T tile[kTrTile][kTrTile + 1];
    __shared__ double red[8];
    const int bi = blockIdx.x, bj = blockIdx.y;   // E rows bi, E columns bj (bj <= bi)
    const int64_t slot = (int64_t)blockIdx.y * gridDim.x + blockIdx.x;
    const int nparts = gridDim.x * gridDim.y;
    if (bj > bi || *bad) {   // uniform in the block: *bad is final here
        if (threadIdx.x == 0) part[slot] = part[slot + nparts] = 0.0;
        return;
    }
    double s0 = 0.0, s1 = 0.0;
    for (int e = threadIdx.x; e < kTrTile * kTrTile; e += 256) {
        const int r = e % kTrTile, c = e / kTrTile;
        const int j = bi * kTrTile + r, i = bj * kTrTile + c;   // M(i, j) = E(j, i)
        T v = T(0);
        if (j < d && i <= j) {
            v = E[j + (int64_t)i * lde];
            const double v2 = (double)(v * v);
            s0 += v2;
            s1 += (double)(v * v * gdiag[i]);
        }
        tile[c][r] = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kTrTile * kTrTile; e += 256) {
        const int c = e % kTrTile, r = e / kTrTile;
        const int j = bi * kTrTile + r, i = bj * kTrTile + c;
        if (j < d && i <= j) M[i + (int64_t)j * ldm] = tile[c][r];
    }
    s0 = block_sum(s0, red);
    s1 = block_sum(s1, red);
    if (threadIdx.x == 0) {
        part[slot] = s0;
        part[slot + nparts] = s1;
    }
}

// out[2] = ||M||_F^2, out[3] = ||M D||_F^2, out[4] = max diag(G), out[5] = *bad,
// out[6] = the status word, out[7] = number of dropped columns
template <typename T>
__global__ void __launch_bounds__(1024)
k_gc_finish(const double* __restrict__ part, int nparts, const T* __restrict__ gdiag, int d,
            const int* __restrict__ bad, const int* __restrict__ ndrop,
            const unsigned* __restrict__ status, double* __restrict__ out)
{
    pdl_wait();
    __shared__ double red[32];
    double a = 0.0, b = 0.0, mx = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        a += part[i];
        b += part[nparts + i];
    }
    for (int j = threadIdx.x; j < d; j += blockDim.x) mx = fmax(mx, (double)gdiag[j]);
    a = block_sum(a, red);
    b = block_sum(b, red);
    mx = block_max(mx, red);
    if (threadIdx.x == 0) {
        out[2] = a;
        out[3] = b;
        out[4] = mx;
        out[5] = (double)*bad;
        out[6] = (double)*status;
        out[7] = (double)*ndrop;
    }
}

// out(c, r) = X(r, c) for the rows x cols matrix X; upper: entries below X's
// diagonal count as zero, and become zero in X.
__global__ void __launch_bounds__(256)
k_gc_tr(float* __restrict__ X, int64_t ldx, int rows, int cols, int upper, float* __restrict__ out, int64_t ldo)
{
    pdl_wait();
    __shared__ float tile[32][33];
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int q = ty; q < 32; q += 8) {
        const int r = r0 + tx, c = c0 + q;
        float v = 0.f;
        if (r < rows && c < cols) {
            if (upper && r > c) X[r + (int64_t)c * ldx] = 0.f;
            else v = X[r + (int64_t)c * ldx];
        }
        tile[q][tx] = v;
    }
    __syncthreads();
    for (int q = ty; q < 32; q += 8) {
        const int c = c0 + tx, r = r0 + q;
        if (r < rows && c < cols) out[c + (int64_t)r * ldo] = tile[tx][q];
    }
}

// ---- c = argmin || S A M c - S b ||: normal equations and refinement -----------
// Products of FP32 matrices with FP64-class vectors: float-float accumulation
// (FP64 FMAs would take 5x as long here); vectors as (hi, lo) pairs.
template <typename T> struct GV { using type = float2; };
template <> struct GV<double> { using type = double; };
SKL_DEV void gv_store(float2& o, double x)
{
    const ff f = ff_from_double(x);
    o = make_float2(f.hi, f.lo);
}
SKL_DEV void gv_store(double& o, double x) { o = x; }
struct GAccF {
    ff a{0.f, 0.f};
    SKL_DEV void fma(float m, float2 x) { ff_fma_f(a, m, ff{x.x, x.y}); }
    SKL_DEV double value() const { return ff_to_double(a); }
};
struct GAccD {
    double a = 0.0;
    SKL_DEV void fma(double m, double x) { a = ::fma(m, x, a); }
    SKL_DEV double value() const { return a; }
};
template <typename T> using GAcc = typename std::conditional<std::is_same<T, float>::value, GAccF, GAccD>::type;

constexpr int kDotThreads = 128;

// y[j] (+)= sum_{i = lo..hi-1} X[i + j ld] v[i] for columns j, one block each:
// MODE 0: all m rows; 1: rows 0..j (M^T t); 2: rows j..m-1 (M y, X = M row-major)
template <typename T, int MODE>
__global__ void __launch_bounds__(kDotThreads)
k_gc_dot(const T* __restrict__ X, int64_t ld, int m, const typename GV<T>::type* __restrict__ v,
         double* __restrict__ y, int add, typename GV<T>::type* __restrict__ ysplit)
{
    pdl_wait();
    __shared__ double red[kDotThreads / 32];
    const int j = blockIdx.x;
    const T* x = X + (int64_t)j * ld;
    const int lo = MODE == 2 ? j : 0, hi = MODE == 1 ? j + 1 : m;
    GAcc<T> a0, a1;
    int i = lo + threadIdx.x;
    for (; i + kDotThreads < hi; i += 2 * kDotThreads) {
        a0.fma(x[i], v[i]);
        a1.fma(x[i + kDotThreads], v[i + kDotThreads]);
    }
    if (i < hi) a0.fma(x[i], v[i]);
    const double s = block_sum(a0.value() + a1.value(), red);
    if (threadIdx.x == 0) {
        const double o = add ? y[j] + s : s;
        if (y) y[j] = o;
        if (ysplit) gv_store(ysplit[j], o);
    }
}

// part[c][i] = sum over the columns of chunk c of X[i + j ld] w[j]
constexpr int kResCols = 64;
template <typename T>
__global__ void __launch_bounds__(256)
k_gc_rows(const T* __restrict__ X, int64_t ld, int m, int d, const typename GV<T>::type* __restrict__ w,
          double* __restrict__ part)
{
    pdl_wait();
    const int i = blockIdx.x * 256 + threadIdx.x;
    const int j0 = blockIdx.y * kResCols, j1 = min(d, j0 + kResCols);
    if (i >= m) return;
    GAcc<T> a;
    int j = j0;
    for (; j + 8 <= j1; j += 8) {
        T x[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) x[q] = X[i + (int64_t)(j + q) * ld];
#pragma unroll
        for (int q = 0; q < 8; ++q) a.fma(x[q], w[j + q]);
    }
    for (; j < j1; ++j) a.fma(X[i + (int64_t)j * ld], w[j]);
    part[(int64_t)blockIdx.y * m + i] = a.value();
}

// r = b - sum of the chunks (nchunks = 0: r = b)
template <typename T>
__global__ void k_gc_res(const double* __restrict__ b, const double* __restrict__ part, int nchunks,
                         int m, typename GV<T>::type* __restrict__ r)
{
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    double s = b[i];
    for (int c = 0; c < nchunks; ++c) s -= part[(int64_t)c * m + i];
    gv_store(r[i], s);
}

// ---- columns the sweep dropped -----------------------------------------------
// Their coefficients R(0:j, j) on the kept columns to W (zeros elsewhere),
// their columns of S A to P; their columns of R become zero.
__global__ void k_gc_drop_gather(const int* __restrict__ drop, float* __restrict__ R, int64_t ldr, int d,
                                 const float* __restrict__ SA, int64_t ld, int m, float* __restrict__ W,
                                 int64_t ldw, float* __restrict__ P, int64_t ldp)
{
    pdl_wait();
    const int t = blockIdx.y, j = drop[t];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < max(d, m); i += gridDim.x * blockDim.x) {
        if (i < d) {
            W[i + t * ldw] = i < j ? R[i + (int64_t)j * ldr] : 0.f;
            if (i <= j) R[i + (int64_t)j * ldr] = 0.f;
        }
        if (i < m) P[i + t * ldp] = SA[i + (int64_t)j * ld];
    }
}

// Zeros below Mc's and above Mr's diagonal (operands of full products).
__global__ void k_gc_zero_other(float* __restrict__ Mc, float* __restrict__ Mr, int64_t ldm, int d)
{
    pdl_wait();
    const int j = blockIdx.x;
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        if (i > j) Mc[i + (int64_t)j * ldm] = 0.f;
        if (i < j) Mr[i + (int64_t)j * ldm] = 0.f;
    }
}

// ||X(:, t)||^2 of column t, one block each
__global__ void __launch_bounds__(256)
k_gc_colnorm(const float* __restrict__ X, int64_t ld, int m, float* __restrict__ out)
{
    pdl_wait();
    __shared__ float red[8];
    const float* x = X + blockIdx.x * ld;
    float s = 0.f;
    for (int i = threadIdx.x; i < m; i += 256) s = fmaf(x[i], x[i], s);
    s = block_sum(s, red);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// *out = max(*out, ||upper triangle of X||_1); one block per column
template <typename T>
__global__ void __launch_bounds__(256)
k_gc_one_norm(const T* __restrict__ X, int64_t ld, double* __restrict__ out)
{
    pdl_wait();
    __shared__ double red[8];
    const T* x = X + (int64_t)blockIdx.x * ld;
    double s = 0.0;
    for (int i = threadIdx.x; i <= (int)blockIdx.x; i += 256) s += fabs((double)x[i]);
    s = block_sum(s, red);
    // sums >= 0 compare like their bits
    if (threadIdx.x == 0) atomicMax((unsigned long long*)out, (unsigned long long)__double_as_longlong(s));
}

// out[0] = max_t p[t] / (1 + w[t]) (a NaN counts as infinity), out[1] = the smallest
// (as 0); one block
__global__ void __launch_bounds__(256)
k_gc_ratio_max(const float* __restrict__ p, const float* __restrict__ w, int k, double* __restrict__ out)
{
    pdl_wait();
    __shared__ double red[8];
    double mx = 0.0, mi = 0.0;   // of r and 1 / r
    for (int t = threadIdx.x; t < k; t += 256) {
        const float r = p[t] / (1.f + w[t]);
        mx = fmax(mx, r >= 0.f ? (double)r : HUGE_VAL);
        mi = fmax(mi, r > 0.f ? 1.0 / (double)r : HUGE_VAL);
    }
    mx = block_max(mx, red);
    mi = block_max(mi, red);
    if (threadIdx.x == 0) {
        out[0] = mx;
        out[1] = 1.0 / mi;
    }
}

// The block's largest |x_i| of n entries and its smallest index (n if all are zero or
// not numbers), in thread 0.
SKL_DEV void block_argmax(const float* __restrict__ x, int n, float& w, int& at)
{
    __shared__ float s_w[8];
    __shared__ int s_i[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    w = 0.f;
    at = n;
    auto take = [&](float v, int i) {
        if (v > w || (v == w && i < at)) {
            w = v;
            at = i;
        }
    };
    for (int i = threadIdx.x; i < n; i += 256) take(fabsf(x[i]), i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float v = __shfl_xor_sync(0xffffffffu, w, o);
        const int i = __shfl_xor_sync(0xffffffffu, at, o);
        take(v, i);
    }
    if (lane == 0) {
        s_w[warp] = w;
        s_i[warp] = at;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int q = 1; q < 8; ++q) take(s_w[q], s_i[q]);
    __syncthreads();
}

// The sweep drops the last of a set of dependent columns, whose coefficients w on the
// others (a column of W per dropped one) may be large: those that stay are then
// nearly dependent themselves.  In another attempt the column with the largest |w_i|
// goes instead if that exceeds 1, and j stays, which multiplies the volume of those
// that stay by |w_i|; a pivoted QR chooses so.  LSQR, which carries the dropped
// columns, pays for the difference where they are not exactly dependent, which FP32
// cannot tell below ~3e-7 (120,000 x 5,000, 50 columns at a distance of 1e-6: 2,650
// iterations, 1,026 with the exchange, 1,028 with the QR).
// want[t] = the column to leave out, *big = max |w_i| (bits of a float >= 0).
__global__ void __launch_bounds__(256)
k_gc_exchange(const int* __restrict__ drop, const float* __restrict__ W, int64_t ldw, int d, int* __restrict__ want,
              int* __restrict__ big)
{
    pdl_wait();
    const int t = blockIdx.x;
    float w;
    int at;
    block_argmax(W + t * ldw, d, w, at);
    if (threadIdx.x != 0) return;
    want[t] = w > 1.02f && at < d ? at : drop[t];   // 2 % above 1: equal ones stay
    atomicMax(big, __float_as_int(w));
}
__global__ void k_gc_leave_out(const int* __restrict__ want, int k, float* __restrict__ mass)
{
    pdl_wait();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < k) mass[want[t]] = std::numeric_limits<float>::infinity();
}

// Excludes (infinite mass) a column for each with ||M e_j||^2 >= limit from the next
// attempt: a dependent column that follows two nearly parallel ones has the
// Gram matrix's noise amplified in its pivot, which then passes, but its column
// of M, (-w, 1) / R_jj, is as large as the noise is small.  The largest entry's column
// goes, by 2 % as above.
__global__ void __launch_bounds__(256)
k_gc_exclude(const float* __restrict__ Mc, int64_t ldm, float limit, float* __restrict__ mass)
{
    pdl_wait();
    __shared__ float red[8];
    const int j = blockIdx.x;
    const float* m = Mc + (int64_t)j * ldm;
    float s = 0.f;
    for (int i = threadIdx.x; i <= j; i += 256) s = fmaf(m[i], m[i], s);
    s = block_sum(s, red);
    if (s < limit) return;   // the same in every thread
    float w;
    int at;
    block_argmax(m, j, w, at);
    if (threadIdx.x == 0) mass[w > 1.02f * fabsf(m[j]) && at < j ? at : j] = std::numeric_limits<float>::infinity();
}

__global__ void __launch_bounds__(256)
k_gc_narrow(const double* __restrict__ X, int64_t ld, int rows, float* __restrict__ out)
{
    pdl_wait();
    const int64_t o = blockIdx.y * ld;
    for (int i = blockIdx.x * 256 + threadIdx.x; i < rows; i += gridDim.x * 256) out[o + i] = (float)X[o + i];
}

// M's diagonal entries of the dropped columns
__global__ void k_gc_drop_unit(const int* __restrict__ drop, int k, float* __restrict__ Mc,
                               float* __restrict__ Mr, int64_t ldm)
{
    pdl_wait();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= k) return;
    const int64_t j = drop[t];
    Mc[j + j * ldm] = 1.f;
    Mr[j + j * ldm] = 1.f;
}

template <typename T>
struct GramBuffers {
    int64_t ldg;
    T* G; T* R; T* mkk; T* gdiag; T* mass; T* partial; int64_t partial_cap;
    int* bad; int* ndrop; double* part; double* out;
    T* Gkeep; T* dw; T* dt; T* dp; T* dn; int* want; int64_t ldp;
    T* Q; T* QT; T* M2c; T* M2r; T* Racc; int64_t ldq;
    typename GV<T>::type* rv; typename GV<T>::type* tv; typename GV<T>::type* cv; typename GV<T>::type* wv;
    double* rows_part; double* c;
    size_t bytes;
};

template <typename T>
GramBuffers<T> gram_carve(void* work, int64_t m, int64_t d, bool multi, bool drops)
{
    GramBuffers<T> B;
    size_t used = 0;
    auto take = [&](size_t bytes) {
        void* p = (char*)work + used;
        used += (bytes + 255) & ~(size_t)255;
        return p;
    };
    using V = typename GV<T>::type;
    const int64_t nt = (d + kTrTile - 1) / kTrTile;
    B.ldg = (d + 31) / 32 * 32;
    B.G = (T*)take((size_t)B.ldg * d * sizeof(T));
    B.R = (T*)take((size_t)B.ldg * d * sizeof(T));
    B.mkk = (T*)take((size_t)kOB * kOB * sizeof(T));
    B.gdiag = (T*)take((size_t)d * sizeof(T));
    B.mass = (T*)take((size_t)d * sizeof(T));
    // FP64: the Gram product's split-K partials (the FP32 products need none)
    B.partial_cap = std::is_same<T, double>::value ? 4 * d * d : 0;
    B.partial_cap = std::min<int64_t>(B.partial_cap, (int64_t)1 << 25);
    B.partial = (T*)take((size_t)B.partial_cap * sizeof(T));
    B.bad = (int*)take(sizeof(int));
    B.ndrop = (int*)take(sizeof(int));
    // dropped columns: their coefficients and two rounds' scratch (d x k), their
    // residuals (m x k)
    const int64_t kd = std::is_same<T, float>::value && drops ? std::min<int64_t>(kGramDropMax, d / 4) : 0;
    B.ldp = (m + 31) / 32 * 32;
    B.Gkeep = (T*)take(kd > 0 ? (size_t)B.ldg * d * sizeof(T) : 0);
    B.dw = (T*)take((size_t)B.ldg * kd * sizeof(T));
    B.dt = (T*)take((size_t)B.ldg * kd * sizeof(T));
    B.dp = (T*)take((size_t)B.ldp * kd * sizeof(T));
    B.dn = (T*)take((size_t)2 * kd * sizeof(T));
    B.want = (int*)take((size_t)kd * sizeof(int));
    B.part = (double*)take((size_t)2 * nt * nt * sizeof(double));
    B.out = (double*)take(8 * sizeof(double));
    B.rv = (V*)take((size_t)m * sizeof(V));
    B.tv = (V*)take((size_t)d * sizeof(V));
    B.cv = (V*)take((size_t)d * sizeof(V));
    B.wv = (V*)take((size_t)d * sizeof(V));
    B.rows_part = (double*)take((size_t)((d + kResCols - 1) / kResCols) * m * sizeof(double));
    B.c = (double*)take((size_t)d * sizeof(double));
    if (multi) {   // later passes: Q, its transpose, the pass's inverse (both layouts), R so far
        B.ldq = (m + 31) / 32 * 32;
        B.Q = (T*)take((size_t)B.ldq * d * sizeof(T));
        B.QT = (T*)take((size_t)B.ldg * m * sizeof(T));
        B.M2c = (T*)take((size_t)B.ldg * d * sizeof(T));
        B.M2r = (T*)take((size_t)B.ldg * d * sizeof(T));
        B.Racc = (T*)take((size_t)B.ldg * d * sizeof(T));
    }
    B.bytes = used;
    return B;
}

// C = A^T B products of the sweep.  Each has an E part (nE columns of E' / E,
// starting at column 0) and a G part (columns from g0).
template <typename T>
struct Sweep {
    const T* SA; int64_t m, d, ld;
    GramBuffers<T> B;
    T* Ew; T* E; int64_t lde;
    unsigned* status;
};

void tn_launch(const CUtensorMap& a, const CUtensorMap& bg, const CUtensorMap& be, const TnArgs& t,
               int row_tiles, int g_tiles, const int* bad, unsigned* status, cudaStream_t st)
{
    if (row_tiles <= 0 || t.nE + g_tiles <= 0) return;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaFuncSetAttribute((const void*)k_tc_tn, cudaFuncAttributeMaxDynamicSharedMemorySize, kNSmem);
    });
    launch_k(k_tc_tn, dim3((unsigned)(t.nE + g_tiles), (unsigned)row_tiles), kNThreads, kNSmem, st, a, bg, be, t,
             bad, status);
    SKL_LAUNCHED();
}

int tiles(int64_t n) { return (int)((n + kNT - 1) / kNT); }

// G = (S A)^T (S A), upper tiles
void sweep_gram(const Sweep<float>& S, cudaStream_t st)
{
    const CUtensorMap ma = map_f32(S.SA, S.m, S.d, S.ld, kNT);
    TnArgs t{};
    t.nkb = (int)((S.m + kBK - 1) / kBK);
    t.rows = t.cols = (int)S.d;
    t.upper = 1;
    t.alpha = 1.f;
    t.Cg = S.B.G;
    t.ldg = S.B.ldg;
    tn_launch(ma, ma, ma, t, tiles(S.d), tiles(S.d), nullptr, S.status, st);
}

void sweep_gram(const Sweep<double>& S, cudaStream_t st)
{
    gemm_upper<double>((int)S.d, (int)S.d, (int)S.m, 1.0, S.SA, S.ld, S.SA, S.ld, 0.0, S.B.G, S.B.ldg,
                       S.B.partial, S.B.partial_cap, st);
}

// [R | E] rows j0..j0+b-1 = M_kk^T [G | E'] (columns right of the block / left of it)
void sweep_row(const Sweep<float>& S, int64_t j0, int b, cudaStream_t st)
{
    const int64_t j1 = j0 + b;
    const CUtensorMap ma = map_f32(S.B.mkk, b, b, kOB, kNT);
    const CUtensorMap mg = map_f32(S.B.G, S.d, S.d, S.B.ldg, kNT);
    const CUtensorMap me = map_f32(S.Ew, S.d, S.d, S.lde, kNT);
    TnArgs t{};
    t.kB = (int)j0;
    t.nkb = (b + kBK - 1) / kBK;
    t.r0 = (int)j0;
    t.g0 = (int)j1;
    t.nE = tiles(j0);
    t.rows = (int)j1;
    t.cols = (int)S.d;
    t.cols_e = (int)j0;
    t.alpha = 1.f;
    t.Cg = S.B.R;
    t.ldg = S.B.ldg;
    t.Ce = S.E;
    t.lde = S.lde;
    tn_launch(ma, mg, me, t, tiles(b), tiles(S.d - j1), S.B.bad, S.status, st);
}

void sweep_row(const Sweep<double>& S, int64_t j0, int b, cudaStream_t st)
{
    const int64_t j1 = j0 + b;
    gemm<double>(true, false, b, (int)(S.d - j1), b, 1.0, S.B.mkk, kOB, S.B.G + j0 + j1 * S.B.ldg, S.B.ldg, 0.0,
                 S.B.R + j0 + j1 * S.B.ldg, S.B.ldg, nullptr, 0, st);
    gemm<double>(true, false, b, (int)j0, b, 1.0, S.B.mkk, kOB, S.Ew + j0, S.lde, 0.0, S.E + j0, S.lde, nullptr,
                 0, st);
}

// rows i0..i1-1 (below block k = [j0, j1)): G -= R_k^T R_k (upper), E' -= R_k^T E_k;
// the columns of E' inside the block start here (overwritten, not added to)
void sweep_update(const Sweep<float>& S, int64_t j0, int64_t j1, int64_t i0, int64_t i1, cudaStream_t st)
{
    if (i1 <= i0) return;
    const CUtensorMap mr = map_f32(S.B.R, S.d, S.d, S.B.ldg, kNT);
    const CUtensorMap me = map_f32(S.E, S.d, S.d, S.lde, kNT);
    TnArgs t{};
    t.kA = t.kB = (int)j0;
    t.nkb = (int)((j1 - j0 + kBK - 1) / kBK);
    t.a0 = t.r0 = t.g0 = (int)i0;
    t.nE = tiles(j1);
    t.rows = (int)i1;
    t.cols = (int)S.d;
    t.cols_e = (int)j1;
    t.e_add = (int)(j0 / kNT);
    t.g_add = 1;
    t.upper = 1;
    t.alpha = -1.f;
    t.Cg = S.B.G;
    t.ldg = S.B.ldg;
    t.Ce = S.Ew;
    t.lde = S.lde;
    tn_launch(mr, mr, me, t, tiles(i1 - i0), tiles(S.d - i0), S.B.bad, S.status, st);
}

void sweep_update(const Sweep<double>& S, int64_t j0, int64_t j1, int64_t i0, int64_t i1, cudaStream_t st)
{
    if (i1 <= i0) return;
    const int K = (int)(j1 - j0), rows = (int)(i1 - i0);
    const double* Ra = S.B.R + j0 + i0 * S.B.ldg;
    gemm_upper<double>(rows, (int)(S.d - i0), K, -1.0, Ra, S.B.ldg, Ra, S.B.ldg, 1.0, S.B.G + i0 + i0 * S.B.ldg,
                       S.B.ldg, nullptr, 0, st);
    if (j0 > 0)
        gemm<double>(true, false, rows, (int)j0, K, -1.0, Ra, S.B.ldg, S.E + j0, S.lde, 1.0, S.Ew + i0, S.lde,
                     nullptr, 0, st);
    gemm<double>(true, false, rows, K, K, -1.0, Ra, S.B.ldg, S.E + j0 + j0 * S.lde, S.lde, 0.0,
                 S.Ew + i0 + j0 * S.lde, S.lde, nullptr, 0, st);
}

// C (M x N) = A^T B, A K x M, B K x N; tri as in TnArgs (2: C's upper tiles only)
void tn_product(int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, const float* B, int64_t ldb, float* C,
                int64_t ldc, unsigned* status, cudaStream_t st, int tri = 0)
{
    const CUtensorMap ma = map_f32(A, K, M, lda, kNT);
    const CUtensorMap mb = map_f32(B, K, N, ldb, kNT);
    TnArgs t{};
    t.nkb = (int)((K + kBK - 1) / kBK);
    t.rows = (int)M;
    t.cols = (int)N;
    t.alpha = 1.f;
    t.Cg = C;
    t.ldg = ldc;
    t.tri = tri;
    t.upper = tri == 2;
    tn_launch(ma, mb, mb, t, tiles(M), tiles(N), nullptr, status, st);
}

// W (dt, zeros at the dropped columns) = the dropped columns' coefficients on the
// columns before them that stay; P (dp) = the dropped columns of S A.
void drop_coefs(const Sweep<float>& S, const int* drop, int k, cudaStream_t st)
{
    const GramBuffers<float>& B = S.B;
    const int m = (int)S.m, d = (int)S.d;
    launch_k(k_gc_drop_gather, dim3(16, (unsigned)k), 256, 0, st, drop, B.R, B.ldg, d, S.SA, S.ld, m, B.dw, B.ldg,
             B.dp, B.ldp);
    launch_k(k_gc_zero_other, (unsigned)d, 256, 0, st, S.Ew, S.E, S.lde, d);
    SKL_LAUNCHED();
    SKL_LAUNCHED();
    tn_product(d, k, d, S.E, S.lde, B.dw, B.ldg, B.dt, B.ldg, S.status, st);
}
void drop_coefs(const Sweep<double>&, const int*, int, cudaStream_t)
{
    fail(SKL_ERR_INVALID, "dropped columns: FP32 only");
}

// Whether the k dropped columns of S A depend on the others at FP32 resolution
// (after drop_coefs).  From S A itself (the Gram matrix cannot tell 1e-4 from 0):
// p = the residual of column j against the columns that stay, with coefficients w
// from the normal equations.  (w, -1) is then a vector that S A maps to p, so the
// dropped columns' singular values are about ||p|| / (1 + ||w||^2)^(1/2), which is
// what the trailing pivots of a pivoted QR show; out[0] = the largest such ratio
// squared.  W is a good start where only columns before j matter; a column that an
// exchange left out depends on later ones too, and takes two steps from zero.
void drop_check(const Sweep<float>& S, int k, bool from_w, cudaStream_t st)
{
    const GramBuffers<float>& B = S.B;
    const int m = (int)S.m, d = (int)S.d;
    float* Mc = S.Ew;
    float* Mr = S.E;
    float* part = (float*)B.rows_part;
    const int64_t cap = (int64_t)((d + kResCols - 1) / kResCols) * m * 2;
    auto norms = [&](const float* X, int64_t ld, int rows, float* out) {
        launch_k(k_gc_colnorm, (unsigned)k, 256, 0, st, X, ld, rows, out);
        SKL_LAUNCHED();
    };
    auto residual = [&](const float* W) {
        gemm<float>(false, false, m, k, d, -1.f, S.SA, S.ld, W, B.ldg, 1.f, B.dp, B.ldp, part, cap, st);
    };
    if (from_w) {
        norms(B.dt, B.ldg, d, B.dn);
        residual(B.dt);
    }
    for (int s = from_w ? 1 : 0; s < 2; ++s) {
        tn_product(d, k, m, S.SA, S.ld, B.dp, B.ldp, B.dw, B.ldg, S.status, st);
        tn_product(d, k, d, Mc, S.lde, B.dw, B.ldg, B.dt, B.ldg, S.status, st);
        tn_product(d, k, d, Mr, S.lde, B.dt, B.ldg, B.dw, B.ldg, S.status, st);
        residual(B.dw);
        if (s == 0) norms(B.dw, B.ldg, d, B.dn);
    }
    norms(B.dp, B.ldp, m, B.dn + k);
    launch_k(k_gc_ratio_max, 1, 256, 0, st, B.dn + k, B.dn, k, B.out);
    SKL_LAUNCHED();
}
void drop_check(const Sweep<double>&, int, bool, cudaStream_t) {}

// After drop_coefs: the columns that another attempt would leave out, to B.want, and
// the largest |w| of a dropped column (its bits to the low half of out[0]).
void drop_exchange(const Sweep<float>& S, const int* drop, int k, cudaStream_t st)
{
    const GramBuffers<float>& B = S.B;
    SKL_CUDA(cudaMemsetAsync(B.out, 0, sizeof(double), st));
    launch_k(k_gc_exchange, (unsigned)k, 256, 0, st, drop, (const float*)B.dt, B.ldg, (int)S.d, B.want, (int*)B.out);
    SKL_LAUNCHED();
}
void drop_exchange(const Sweep<double>&, const int*, int, cudaStream_t) {}
void leave_out(const Sweep<float>& S, int k, cudaStream_t st)
{
    launch_k(k_gc_leave_out, (unsigned)((k + 127) / 128), 128, 0, st, (const int*)S.B.want, k, S.B.mass);
    SKL_LAUNCHED();
}
void leave_out(const Sweep<double>&, int, cudaStream_t) {}

void tr_launch(float* X, int64_t ldx, int64_t rows, int64_t cols, int upper, float* out, int64_t ldo, cudaStream_t st)
{
    launch_k(k_gc_tr, dim3((unsigned)((rows + 31) / 32), (unsigned)((cols + 31) / 32)), 256, 0, st, X, ldx, (int)rows,
             (int)cols, upper, out, ldo);
    SKL_LAUNCHED();
}

// After pass 1 (S.SA = S A, its inverse in Mc / Mr): S becomes the sweep of
// Q = S A M, with the pass's own inverse in M2c / M2r.
void next_pass(Sweep<float>& S, float* Mc, float* Mr, int64_t ldm, bool first, cudaStream_t st)
{
    GramBuffers<float>& B = S.B;
    // the last pass's inverse, zeros in its other triangles
    float* Pc = first ? Mc : B.M2c;
    float* Pr = first ? Mr : B.M2r;
    const int64_t ldp = first ? ldm : B.ldg;
    launch_k(k_gc_zero_other, (unsigned)S.d, 256, 0, st, Pc, Pr, ldp, (int)S.d);
    SKL_LAUNCHED();
    if (first) SKL_CUDA(cudaMemcpyAsync(B.Racc, B.R, (size_t)B.ldg * S.d * sizeof(float), cudaMemcpyDeviceToDevice, st));
    // Q = (last Q) P by products with both operands contiguous along K
    tr_launch(const_cast<float*>(S.SA), S.ld, S.m, S.d, 0, B.QT, B.ldg, st);
    tn_product(S.m, S.d, S.d, B.QT, B.ldg, Pc, ldp, B.Q, B.ldq, S.status, st, 1);
    S.SA = B.Q;
    S.ld = B.ldq;
    S.Ew = B.M2c;
    S.E = B.M2r;
    S.lde = B.ldg;
}
void next_pass(Sweep<double>&, double*, double*, int64_t, bool, cudaStream_t)
{
    fail(SKL_ERR_INVALID, "Gram passes: FP32 only");
}

// M = M (pass's inverse), R = (pass's R) R after a sweep of a later pass.
void join_pass(Sweep<float>& S, float* Mc, float* Mr, int64_t ldm, cudaStream_t st)
{
    GramBuffers<float>& B = S.B;
    const int64_t d = S.d;
    launch_k(k_gc_zero_other, (unsigned)d, 256, 0, st, B.M2c, B.M2r, B.ldg, (int)d);
    SKL_LAUNCHED();
    tn_product(d, d, d, Mr, ldm, B.M2c, B.ldg, Mc, ldm, S.status, st, 2);
    transpose_upper<float>(Mc, ldm, d, Mr, st);
    tr_launch(B.R, B.ldg, d, d, 1, B.QT, B.ldg, st);
    tr_launch(B.Racc, B.ldg, d, d, 1, B.G, B.ldg, st);   // zeros below R's diagonal
    tn_product(d, d, d, B.QT, B.ldg, B.Racc, B.ldg, B.G, B.ldg, S.status, st, 2);
    SKL_CUDA(cudaMemcpyAsync(B.Racc, B.G, (size_t)B.ldg * d * sizeof(float), cudaMemcpyDeviceToDevice, st));
}
void join_pass(Sweep<double>&, double*, double*, int64_t, cudaStream_t) {}

void drop_exclude(const Sweep<float>& S, double limit, cudaStream_t st)
{
    launch_k(k_gc_exclude, (unsigned)S.d, 256, 0, st, S.Ew, S.lde, (float)limit, S.B.mass);
    SKL_LAUNCHED();
}
void drop_exclude(const Sweep<double>&, double, cudaStream_t) {}

}  // namespace

template <typename T>
size_t gram_workspace_bytes(int64_t m, int64_t d, bool multi, bool drops)
{
    return gram_carve<T>(nullptr, m, d, multi && std::is_same<T, float>::value, drops).bytes;
}

bool gram_enabled()
{
    static const bool v = [] {
        const char* e = std::getenv("SKILLS_GRAM");
        return !(e && e[0] == '0');
    }();
    return v;
}

template <typename T>
bool gram_precond(const T* SA, int64_t m, int64_t d, int64_t ld, double* c, int* jpvt, T* Mc, T* Mr, int64_t ldm,
                  double abs_thresh, double rel_thresh, double rcond_min, GramResult& res, int* drop, bool multi, void* work,
                  unsigned* status, void* host_pinned, cudaStream_t st)
{
    // columns the sweep may drop: only where the caller carries them (FP32)
    const int drop_cap = drop ? (int)std::min<int64_t>(kGramDropMax, d / 4) : 0;
    // A dependent column leaves a pivot of up to ~2e-5 of its mass in the FP32
    // Gram matrix (measured at 120,000 x 5,000), and boosted pivots have to stand
    // clear of the noise around them: with rows of noise / bound ~ 0.1 above them
    // the inverse grows exponentially (128 eps overflowed at 200 columns).  With
    // neither, a failed pivot only ends the attempt early, which the bound on M D
    // below would do.
    // Where columns may be dropped, pivots are only raised for sketches that turn out
    // to need later passes.
    const bool passes = multi && std::is_same<T, float>::value;
    bool boost = passes && !drop;
    const T eps = std::is_same<T, float>::value ? T(5.9604644775390625e-08) : T(1.1102230246251565e-16);
    const T pivot = (drop || passes ? T(2048) : T(128)) * eps;
    Sweep<T> S{SA, m, d, ld, gram_carve<T>(work, m, d, passes, drop != nullptr), Mc, Mr, ldm, status};
    GramBuffers<T>& B = S.B;
    const size_t dsm = (2 * (size_t)kIB * kSL + kIB) * sizeof(T);
    const size_t ssm = (4 * (size_t)kIB * kSL + kIB) * sizeof(T);
    GcArgs<T> ga{B.G, B.R, B.ldg, Mc, Mr, ldm, B.mkk, B.mass, B.bad, B.ndrop, drop, drop_cap, (int)d, pivot, boost ? 1 : 0};
    allow_max_dynamic_smem((const void*)k_gc_diag<T>);
    allow_max_dynamic_smem((const void*)k_gc_step<T>);

    // Side stream for the bulk of the trailing updates: block k + 1's rows are
    // updated first on the main stream, so its chain of diagonal blocks runs
    // while the rows below it are updated.  Worth its events only when the
    // bulk is more than a few blocks.
    const bool lookahead = d > 4 * kOB;
    cudaStream_t side = nullptr;
    cudaEvent_t evT = nullptr, evB = nullptr;
    struct Guard {
        cudaStream_t& s;
        cudaEvent_t& a;
        cudaEvent_t& b;
        ~Guard()
        {
            if (a) cudaEventDestroy(a);
            if (b) cudaEventDestroy(b);
            if (s) cudaStreamDestroy(s);
        }
    } guard{side, evT, evB};
    if (lookahead) {
        SKL_CUDA(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
        SKL_CUDA(cudaEventCreateWithFlags(&evT, cudaEventDisableTiming));
        SKL_CUDA(cudaEventCreateWithFlags(&evB, cudaEventDisableTiming));
    }

    // again: on the first sweep's Gram matrix
    auto factor = [&](bool again, bool all_columns) {
        // the sweep works in place; a copy of the Gram matrix (30 us at 5,000 columns, the
        // product 1.5 ms) is there for attempts without some of the columns
        const size_t gbytes = (size_t)B.ldg * d * sizeof(T);
        if (!again) sweep_gram(S, st);
        if (drop_cap > 0 && (again || !ga.boost))
            SKL_CUDA(cudaMemcpyAsync(again ? B.G : B.Gkeep, again ? B.Gkeep : B.G, gbytes, cudaMemcpyDeviceToDevice, st));
        launch_k(k_gc_init<T>, 64, 256, 0, st, B.G, B.ldg, (int)d, B.gdiag, B.mass, all_columns, B.mkk, jpvt, B.bad, B.ndrop);
        SKL_LAUNCHED();
        bool bulk_pending = false;
        for (int64_t j0 = 0; j0 < d; j0 += kOB) {
            const int b = (int)std::min<int64_t>(kOB, d - j0);
            const int64_t j1 = j0 + b;
            const int nb = (b + kIB - 1) / kIB;
            launch_k(k_gc_diag<T>, 1, kSmallThreads, dsm, st, ga, (int)j0, (int)std::min<int64_t>(kIB, d - j0));
            SKL_LAUNCHED();
            for (int s = 0; s < nb; ++s) {
                int blocks = nb - 1;   // the block row, the next diagonal block (in the G updates), the updates
                for (int I = s + 1; I < nb; ++I) blocks += s + 1 + nb - I;
                if (blocks == 0) break;
                launch_k(k_gc_step<T>, blocks, kSmallThreads, ssm, st, ga, (int)j0, s, nb);
                SKL_LAUNCHED();
            }
            if (j0 > 0 || j1 < d) sweep_row(S, j0, b, st);
            if (j1 >= d) break;
            const int64_t i1 = std::min<int64_t>(d, j1 + kOB);
            if (lookahead && i1 < d) {
                SKL_CUDA(cudaEventRecord(evT, st));
                if (bulk_pending) SKL_CUDA(cudaStreamWaitEvent(st, evB, 0));
                SKL_CUDA(cudaStreamWaitEvent(side, evT, 0));
                sweep_update(S, j0, j1, j1, i1, st);
                sweep_update(S, j0, j1, i1, d, side);
                SKL_CUDA(cudaEventRecord(evB, side));
                bulk_pending = true;
            } else {
                if (bulk_pending) SKL_CUDA(cudaStreamWaitEvent(st, evB, 0));
                bulk_pending = false;
                sweep_update(S, j0, j1, j1, d, st);
            }
        }
        const int nt = (int)((d + kTrTile - 1) / kTrTile);
        launch_k(k_gc_transpose<T>, dim3(nt, nt), 256, 0, st, S.E, S.lde, (int)d, S.Ew, S.lde, B.gdiag, B.part, B.bad);
        SKL_LAUNCHED();
        launch_k(k_gc_finish<T>, 1, 1024, 0, st, B.part, nt * nt, B.gdiag, (int)d, B.bad, B.ndrop, status, B.out);
        SKL_LAUNCHED();
    };
    auto solve_c = [&] {
        if (c) {
            // c = M M^T-normal equations of the sketched problem, then two steps of
            // refinement against its residual: each contracts the error by the
            // factor's departure from orthogonality (a few percent at the acceptance
            // bound, ~1e-4 usually), which leaves c at the accuracy of an FP32 QR's
            // or better
            const unsigned gm = (unsigned)((m + 255) / 256);
            const int nch = (int)((d + kResCols - 1) / kResCols);
            auto correct = [&](bool add, auto* split) {
                launch_k(k_gc_dot<T, 0>, (unsigned)d, kDotThreads, 0, st, SA, ld, (int)m, B.rv, (double*)nullptr, 0,
                         B.tv);
                launch_k(k_gc_dot<T, 1>, (unsigned)d, kDotThreads, 0, st, (const T*)Mc, ldm, (int)d, B.tv, B.c,
                         add ? 1 : 0, split);
                SKL_LAUNCHED();
                SKL_LAUNCHED();
            };
            launch_k(k_gc_res<T>, gm, 256, 0, st, c, (const double*)nullptr, 0, (int)m, B.rv);
            SKL_LAUNCHED();
            correct(false, B.cv);
            for (int s = 0; s < 2; ++s) {
                launch_k(k_gc_dot<T, 2>, (unsigned)d, kDotThreads, 0, st, (const T*)Mr, ldm, (int)d, B.cv,
                         (double*)nullptr, 0, B.wv);
                launch_k(k_gc_rows<T>, dim3(gm, nch), 256, 0, st, SA, ld, (int)m, (int)d, B.wv, B.rows_part);
                launch_k(k_gc_res<T>, gm, 256, 0, st, c, B.rows_part, nch, (int)m, B.rv);
                for (int q = 0; q < 3; ++q) SKL_LAUNCHED();
                correct(true, B.cv);
            }
        }
    };
    double* hp = (double*)host_pinned;
    auto read_out = [&](int count) {
        SKL_CUDA(cudaMemcpyAsync(hp, B.out, count * sizeof(double), cudaMemcpyDeviceToHost, st));
        SKL_CUDA(cudaStreamSynchronize(st));
    };
    double mf2 = 0.0, mdf2 = 0.0, gmax = 0.0, thresh = 0.0;
    int ndrop = 0;
    auto read_sweep = [&] {
        read_out(8);
        mf2 = hp[2];
        mdf2 = hp[3];
        gmax = hp[4];
        ndrop = (int)hp[7];
        if ((unsigned)hp[6] & kStatusTcTimeout)
            fail(SKL_ERR_TIMEOUT, "a tensor-core product's bounded wait gave up");
        // the rank rule's threshold (below: with a factor 2 for M's own error)
        thresh = std::max(abs_thresh, rel_thresh * std::sqrt(gmax));
        return hp[5] == 0.0 && std::isfinite(mf2) && std::isfinite(mdf2) && mf2 > 0.0;
    };
    // sigma_min > 2 thresh: from ||M||_F, or where many small singular values make that
    // too large, from ||M||_2^2 <= ||M||_1 ||M||_inf
    auto resolves = [&] {
        if (1.0 / std::sqrt(mf2) > 2.0 * thresh) return true;
        if (!drop || !std::isfinite(mf2)) return false;
        SKL_CUDA(cudaMemsetAsync(B.out, 0, 2 * sizeof(double), st));
        inf_norm_upper<T>(Mc, ldm, d, B.rows_part, B.out, st);
        launch_k(k_gc_one_norm<T>, (unsigned)d, 256, 0, st, (const T*)Mc, ldm, B.out + 1);
        SKL_LAUNCHED();
        read_out(2);
        return 1.0 / std::sqrt(hp[0] * hp[1]) > 2.0 * thresh;
    };
    for (int attempt = 0;; ++attempt) {
        factor(attempt > 0, attempt == 0);
        if (!read_sweep()) return false;
        if (boost) break;
        const bool well = (double)eps * mdf2 <= 1.0 / 16;
        if (ndrop == 0) {
            if (well) break;
            // condition number beyond ~1e3: later passes, as on the dense path
            if (!passes || !resolves()) return false;
            ga.boost = boost = true;
            break;
        }
        drop_coefs(S, drop, ndrop, st);
        bool again = !well;
        if (attempt == 0) {
            // a sweep more (a tenth of a rank-deficient solve) where a choice is worse
            // than the best by more than 2
            drop_exchange(S, drop, ndrop, st);
            read_out(1);
            float w;
            std::memcpy(&w, hp, sizeof w);
            again = again || w > 2.f;
            if (again) leave_out(S, ndrop, st);
        }
        if (!again) {
            drop_check(S, ndrop, attempt == 0, st);
            read_out(2);
            if (std::sqrt(hp[0]) <= 0.25 * thresh) break;
            // none of them dependent, nor close to what the rule decides on: later
            // passes with all columns resolve them
            if (!passes || !(std::sqrt(hp[1]) >= 4.0 * thresh)) return false;
            ga.boost = boost = true;
            factor(true, true);
            if (!read_sweep()) return false;
            break;
        }
        if (attempt == 2) return false;
        // and without dependent columns whose pivots passed
        if (!well) drop_exclude(S, 1.0 / (64.0 * (double)eps), st);
    }
    const T* R = B.R;
    if (boost && !((double)eps * mdf2 <= 1.0 / 16 && ndrop == 0)) {
        // Too ill-conditioned for its Gram matrix, or with boosted pivots: the same
        // on Q = S A M, whose condition number is about the root of the excess, at
        // most twice; M and R are the passes' products.  Boosted pivots can make a
        // pass's inverse grow, which costs the product its digits: the limit of 64 on
        // eps ||S A|| ||M_1|| ||M_2|| stands above what accepted attempts showed (1,500
        // x 100 to 40,000 x 4,000, condition numbers to 3e7: at most 15; 30 to 257
        // where the rank rule below refused) and keeps a runaway from a third pass.
        const double unit = (double)eps * std::sqrt(gmax);
        if (unit * std::sqrt(mf2 * (double)d) > 64.0) return false;
        for (int pass = 2;; ++pass) {
            const double before = mf2;
            next_pass(S, Mc, Mr, ldm, pass == 2, st);
            ga.Ew = S.Ew;
            ga.E = S.E;
            ga.lde = S.lde;
            factor(false, true);
            read_out(8);
            if ((unsigned)hp[6] & kStatusTcTimeout)
                fail(SKL_ERR_TIMEOUT, "a tensor-core product's bounded wait gave up");
            if (hp[5] != 0.0 || !std::isfinite(hp[2]) || !std::isfinite(hp[3]) || !(hp[2] > 0.0)) return false;
            if (unit * std::sqrt(before * hp[2]) > 64.0) return false;
            const bool last = (double)eps * hp[3] <= 1.0 / 16 && hp[7] == 0.0;
            join_pass(S, Mc, Mr, ldm, st);
            // ||M||_F of the product (the masses stay the pass's: only out[2] counts)
            const int nt = (int)((d + kTrTile - 1) / kTrTile);
            launch_k(k_gc_transpose<T>, dim3(nt, nt), 256, 0, st, Mr, ldm, (int)d, Mc, ldm, B.gdiag, B.part, B.bad);
            launch_k(k_gc_finish<T>, 1, 1024, 0, st, B.part, nt * nt, B.gdiag, (int)d, B.bad, B.ndrop, status, B.out);
            SKL_LAUNCHED();
            SKL_LAUNCHED();
            read_out(8);
            mf2 = hp[2];
            if (!std::isfinite(mf2) || !resolves()) return false;
            if (last) break;
            // raised pivots understate M: with 0.28 and more of the FP32 resolution here,
            // all of ten third passes ended beyond it (12,007 x 1,201 to 40,000 x 4,000);
            // 12,000 x 4,500, condition number 1e7: a refusal costs 8.1 ms instead of 12
            if (hp[7] != 0.0 && unit * std::sqrt(mf2) > 0.3) return false;
            if (pass == 3) return false;
        }
        R = B.Racc;
        ndrop = 0;
    }
    if (!resolves()) return false;
    SKL_CUDA(cudaMemsetAsync(B.out, 0, 2 * sizeof(double), st));
    inf_norm_upper<T>(R, B.ldg, d, B.rows_part, B.out, st);
    inf_norm_upper<T>(Mc, ldm, d, B.rows_part, B.out + 1, st);
    read_out(2);
    const double nr = hp[0], nm = hp[1];
    if (!(nr > 0 && nm > 0) || !(1.0 / (nr * nm) > rcond_min)) return false;
    res.norm_r = nr;
    res.norm_m = nm;
    res.dropped = ndrop;
    solve_c();
    if (c) SKL_CUDA(cudaMemcpyAsync(c, B.c, d * sizeof(double), cudaMemcpyDeviceToDevice, st));
    return true;
}

static size_t up256(size_t b) { return (b + 255) & ~(size_t)255; }

size_t gram_probe_bytes(int64_t m, int64_t d, int64_t ld)
{
    if (d < kGramProbeCols) return 0;
    return up256((size_t)ld * d * sizeof(float)) + up256(kGramDropMax * sizeof(int)) +
           gram_workspace_bytes<float>(m, d, true, true);
}

bool gram_probe(const double* SA, int64_t m, int64_t d, int64_t ld, int* jpvt, double* Mc, double* Mr, void* work,
                unsigned* status, void* host_pinned, cudaStream_t st)
{
    if (d < kGramProbeCols) return true;
    float* SAf = (float*)work;
    int* drop = (int*)((char*)work + up256((size_t)ld * d * sizeof(float)));
    void* rest = (char*)drop + up256(kGramDropMax * sizeof(int));
    launch_k(k_gc_narrow, dim3((unsigned)((m + 1023) / 1024), (unsigned)d), 256, 0, st, SA, ld, (int)m, SAf);
    SKL_LAUNCHED();
    const double eps = 5.960464477539063e-08;
    GramResult res;
    auto attempt = [&](double rel, int* dropped) {
        return gram_precond<float>(SAf, m, d, ld, nullptr, jpvt, (float*)Mc, (float*)Mr, (d + 3) / 4 * 4, 0.0, rel, 0.0,
                                   res, dropped, true, rest, status, host_pinned, st);
    };
    if (attempt(2.0 * std::sqrt((double)m) * eps, drop)) return res.dropped == 0;
    // too ill-conditioned for that: as far as FP32 passes resolve it (~1e6) the FP64
    // Gram matrix (~1e7) does
    return attempt(eps, nullptr);
}

void gram_unit_dropped(const int* drop, int64_t k, float* Mc, float* Mr, int64_t ldm, cudaStream_t st)
{
    if (k <= 0) return;
    launch_k(k_gc_drop_unit, (unsigned)((k + 127) / 128), 128, 0, st, drop, (int)k, Mc, Mr, ldm);
    SKL_LAUNCHED();
}
void gram_unit_dropped(const int*, int64_t, double*, double*, int64_t, cudaStream_t) {}

template size_t gram_workspace_bytes<float>(int64_t, int64_t, bool, bool);
template size_t gram_workspace_bytes<double>(int64_t, int64_t, bool, bool);
template bool gram_precond<float>(const float*, int64_t, int64_t, int64_t, double*, int*, float*, float*, int64_t, double,
                                  double, double, GramResult&, int*, bool, void*, unsigned*, void*, cudaStream_t);
template bool gram_precond<double>(const double*, int64_t, int64_t, int64_t, double*, int*, double*, double*, int64_t,
                                   double, double, double, GramResult&, int*, bool, void*, unsigned*, void*, cudaStream_t);

}  // namespace skl
