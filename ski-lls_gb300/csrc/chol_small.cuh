// chol_small.cuh -- b x b (b <= 64) dense algebra of one CTA: Cholesky with
// the inverse of its factor, modified LU with both inverses, and their block
// products, on row-major shared-memory blocks.
#pragma once
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "skl_internal.hpp"
#include "common.cuh"

namespace skl {

constexpr int kSmallThreads = 1024;

// ---- small dense algebra on b x b (b <= 64) row-major shared-memory blocks --
// The modified LU is blocked by 16: the 16 x 16 diagonal blocks are factored and
// inverted by one warp (a step is a __syncwarp, not a block barrier), and
// everything else is a block product over the whole CTA (blk_mul).  Matrices are padded to
// np = round_up(b, 16) rows/columns (identity for the Cholesky, zeros for the
// LU input, which the modified LU turns into identity factors).
constexpr int kDB = 16;   // diagonal block

// Warp-level 16 x 16 routines: lane l holds row l >> 1, columns 8 (l & 1) ..
// +7 of the block in registers; row k reaches the other lanes by shuffles, so
// a step is ~25 instructions with no shared-memory round trip.  The step
// loops stay rolled (register elements picked by selects): a one-warp
// straight-line version would wait on instruction fetch.
template <typename T>
SKL_DEV void row_load(const T* A, int ld, T (&a)[8])
{
    const int lane = threadIdx.x & 31, r = lane >> 1, cb = (lane & 1) * 8;
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] = A[r * ld + cb + e];
}

template <typename T>
SKL_DEV T t_rcp(T x);
template <> SKL_DEV float t_rcp<float>(float x) { return __frcp_rn(x); }
template <> SKL_DEV double t_rcp<double>(double x) { return __drcp_rn(x); }

// Pivot reciprocal on the elimination's dependency chain: the hardware
// approximation (relative error ~2^-23, like one more rounding of the
// pivot) instead of the correctly rounded multi-instruction sequence.
template <typename T>
SKL_DEV T t_rcp_chain(T x);
template <> SKL_DEV float t_rcp_chain<float>(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <> SKL_DEV double t_rcp_chain<double>(double x) { return __drcp_rn(x); }

// X = U^{-1} for the upper 16 x 16 block U (entries below its diagonal never
// read): X's upper triangle, and zeros below it when zero_lower.  A zero
// diagonal entry leaves its row and column of X zero: X is then the inverse of
// the rest.
template <typename T>
SKL_DEV void warp16_inv_upper(const T* U, int ldu, T* X, int ldx, bool zero_lower)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, r = lane >> 1, cb = (lane & 1) * 8;
    const T dv = lane < kDB ? U[lane * ldu + lane] : T(0);
    const T iv = dv != T(0) ? t_rcp(dv) : T(0);
    T x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = (cb + e == r) ? T(1) : T(0);
#pragma unroll 1
    for (int k = kDB - 1; k >= 0; --k) {
        const T ik = __shfl_sync(full, iv, k);
        const T u = U[r * ldu + k];
        if (r == k) {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] *= ik;
        }
        T xk[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) xk[e] = __shfl_sync(full, x[e], 2 * k + (lane & 1));
        if (r < k) {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] -= u * xk[e];
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int c = cb + e;
        if (c >= r) X[r * ldx + c] = x[e];
        else if (zero_lower) X[r * ldx + c] = T(0);
    }
    __syncwarp();
}

// Y = L^{-1} for the unit lower 16 x 16 block L (strict lower part read):
// Y's strict lower part only (unit diagonal implied).
template <typename T>
SKL_DEV void warp16_inv_unit_lower(const T* L, int ldl, T* Y, int ldy)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, r = lane >> 1, cb = (lane & 1) * 8;
    T y[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) y[e] = T(0);
#pragma unroll 1
    for (int k = 0; k < kDB - 1; ++k) {
        const T l = L[r * ldl + k];
        T yk[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) yk[e] = __shfl_sync(full, y[e], 2 * k + (lane & 1));
        if (r > k) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int c = cb + e;
                if (c < k) y[e] -= l * yk[e];
                else if (c == k) y[e] -= l;
            }
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e)
        if (cb + e < r) Y[r * ldy + cb + e] = y[e];
    __syncwarp();
}

// Modified LU without pivoting of the 16 x 16 block A in place: S_k =
// -sign(pivot), U_kk = pivot - S_k (|U_kk| >= 1); L's multipliers below the
// diagonal, U on and above; S to sg.
template <typename T>
SKL_DEV void warp16_mlu(T* A, int ld, T* sg)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, r = lane >> 1, cb = (lane & 1) * 8;
    T a[8];
    row_load(A, ld, a);
#pragma unroll 1
    for (int kh = 0; kh < 2; ++kh) {
#pragma unroll
        for (int kl = 0; kl < 8; ++kl) {
            const int k = kh * 8 + kl;
            const T p = __shfl_sync(full, a[kl], 2 * k + kh);
            const T sk = p >= T(0) ? T(-1) : T(1);
            const T ukk = p - sk;
            const T iu = t_rcp_chain(ukk);
            T rk[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) rk[e] = __shfl_sync(full, a[e], 2 * k + (lane & 1));
            const T other = __shfl_xor_sync(full, a[kl], 1);
            const T l = (kh == (lane & 1) ? a[kl] : other) * iu;
            if (r > k) {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int c = cb + e;
                    if (c > k) a[e] -= l * rk[e];
                    else if (c == k) a[e] = l;
                }
            } else if (r == k) {
                if (kh == (lane & 1)) a[kl] = ukk;
            }
            if (lane == 0) sg[k] = sk;
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) A[r * ld + cb + e] = a[e];
    __syncwarp();
}

// Operand views for blk_mul, in the coordinates (r, s) of op(X):
// kMLower: zeros are stored above the diagonal.
enum : int { kMFull = 0, kMUpper = 1, kMUpperUnit = 2, kMLowerUnit = 3, kMLower = 4 };

template <typename T, bool TR, int MASK>
SKL_DEV T op_at(const T* X, int ld, int r, int s)
{
    if (MASK == kMUpper && s < r) return T(0);
    if (MASK == kMUpperUnit && s <= r) return s == r ? T(1) : T(0);
    if (MASK == kMLowerUnit && s >= r) return s == r ? T(1) : T(0);
    return TR ? X[s * ld + r] : X[r * ld + s];
}

// k range of a product term for masked operands: A upper restricts k >= i,
// B upper / upper-unit restricts k <= c, A lower-unit restricts k <= i.
template <int MA, int MB>
SKL_DEV void k_range(int i0, int c0, int tr, int tc, int kk, int& klo, int& khi)
{
    klo = 0;
    khi = kk;
    if (MA == kMUpper) klo = i0;
    if (MA == kMLowerUnit || MA == kMLower) khi = min(khi, i0 + tr);
    if (MB == kMUpper || MB == kMUpperUnit) khi = min(khi, c0 + tc);
    if (MB == kMLowerUnit) klo = max(klo, c0);
}

// C (m x n) = alpha * op(A) (m x kk) * op(B) (kk x n) [* diag(sB) on B's
// rows] (+ C when ACC), row-major shared memory; TR x TR register tiles, one
// per thread (m * n <= TR * TR * kSmallThreads); k runs only over the range
// the operand masks leave nonzero.  Results wait for a block barrier, so C may
// alias A or B.  With Cg set, C goes to global memory column-major (ldg)
// instead and its diagonal also to tau.
template <typename T, bool TA, int MA, bool TB, int MB, bool ACC, int TR>
SKL_DEV void blk_mul_t(int m, int n, int kk, const T* A, int lda, const T* B, int ldb,
                       const T* __restrict__ sB, T alpha, T* C, int ldc, T* __restrict__ Cg, int ldg,
                       T* __restrict__ tau)
{
    const int ntc = (n + TR - 1) / TR;
    const int t = threadIdx.x;
    const int i0 = (t / ntc) * TR, c0 = (t % ntc) * TR;
    const bool act = i0 < m;
    T acc[TR][TR];
#pragma unroll
    for (int r = 0; r < TR; ++r)
#pragma unroll
        for (int q = 0; q < TR; ++q) acc[r][q] = T(0);
    if (act) {
        int klo, khi;
        k_range<MA, MB>(i0, c0, TR, TR, kk, klo, khi);
#pragma unroll 4
        for (int k = klo; k < khi; ++k) {
            T av[TR], bv[TR];
#pragma unroll
            for (int r = 0; r < TR; ++r) av[r] = (i0 + r < m) ? op_at<T, TA, MA>(A, lda, i0 + r, k) : T(0);
            const T sc = sB ? sB[k] : T(1);
#pragma unroll
            for (int q = 0; q < TR; ++q) bv[q] = (c0 + q < n) ? sc * op_at<T, TB, MB>(B, ldb, k, c0 + q) : T(0);
#pragma unroll
            for (int r = 0; r < TR; ++r)
#pragma unroll
                for (int q = 0; q < TR; ++q) acc[r][q] += av[r] * bv[q];
        }
    }
    __syncthreads();
    if (act) {
#pragma unroll
        for (int r = 0; r < TR; ++r) {
            const int i = i0 + r;
            if (i >= m) continue;
#pragma unroll
            for (int q = 0; q < TR; ++q) {
                const int c = c0 + q;
                if (c >= n) continue;
                const T v = alpha * acc[r][q];
                if (Cg) {
                    Cg[i + (int64_t)c * ldg] = v;
                    if (i == c) tau[i] = v;
                } else if (ACC) {
                    C[i * ldc + c] += v;
                } else {
                    C[i * ldc + c] = v;
                }
            }
        }
    }
    __syncthreads();
}

// FP32: the same product on the warps' tensor cores, one 16 x 8 tile of C per
// warp (mma.sync m16n8k8 TF32; a 64 x 64 result is the CTA's 32 warps), k
// over the range the masks leave nonzero.  3xTF32 with round-to-nearest
// splits, hi = rna(a) and lo = rna(a - hi), so hi*hi + hi*lo + lo*hi carries
// each product to ~2^-24 like an FP32 FMA.  A 64 x 64 x 64 product is ~200
// instructions per warp instead of ~770 per thread for the 2 x 2 register
// tiles, and these products are most of the panel's serial b x b algebra.
// (For a single-CTA product this small the warp-level MMA beats a tcgen05
// launch: no tensor-memory allocation, descriptors or commit round trip.)
SKL_DEV unsigned tf32_rna(float a)
{
    unsigned r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(a));
    return r;
}

SKL_DEV void mma_tf32_16x8x8(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2])
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
        "{%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// One warp's 16 x 8 tile w of C = op(A) op(B) (m x n, k over the masks'
// range), accumulated in acc; false when the product has no tile w.
template <bool TA, int MA, bool TB, int MB>
SKL_DEV bool tc_tile(int w, int m, int n, int kk, const float* A, int lda, const float* B, int ldb,
                     const float* __restrict__ sB, float (&acc)[4], int& i0, int& c0)
{
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int ntn = (n + 7) >> 3;
    acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
    if (w < 0 || w >= ((m + 15) >> 4) * ntn) return false;
    i0 = (w / ntn) * 16;
    c0 = (w % ntn) * 8;
    int klo, khi;
    k_range<MA, MB>(i0, c0, 16, 8, kk, klo, khi);
    klo &= ~7;
    const int ra0 = i0 + g, ra1 = i0 + g + 8, cb = c0 + g;
    for (int k0 = klo; k0 < khi; k0 += 8) {
        const int ka0 = k0 + tig, ka1 = k0 + tig + 4;
        // fragments: A (g, tig) (g+8, tig) (g, tig+4) (g+8, tig+4); B (tig, g) (tig+4, g)
        float av[4], bv[2];
        av[0] = (ra0 < m && ka0 < kk) ? op_at<float, TA, MA>(A, lda, ra0, ka0) : 0.f;
        av[1] = (ra1 < m && ka0 < kk) ? op_at<float, TA, MA>(A, lda, ra1, ka0) : 0.f;
        av[2] = (ra0 < m && ka1 < kk) ? op_at<float, TA, MA>(A, lda, ra0, ka1) : 0.f;
        av[3] = (ra1 < m && ka1 < kk) ? op_at<float, TA, MA>(A, lda, ra1, ka1) : 0.f;
        bv[0] = (ka0 < kk && cb < n) ? (sB ? sB[ka0] : 1.f) * op_at<float, TB, MB>(B, ldb, ka0, cb) : 0.f;
        bv[1] = (ka1 < kk && cb < n) ? (sB ? sB[ka1] : 1.f) * op_at<float, TB, MB>(B, ldb, ka1, cb) : 0.f;
        unsigned ah[4], al[4], bh[2], bl[2];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            ah[e] = tf32_rna(av[e]);
            al[e] = tf32_rna(av[e] - __uint_as_float(ah[e]));
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            bh[e] = tf32_rna(bv[e]);
            bl[e] = tf32_rna(bv[e] - __uint_as_float(bh[e]));
        }
        mma_tf32_16x8x8(acc, al, bh);
        mma_tf32_16x8x8(acc, ah, bl);
        mma_tf32_16x8x8(acc, ah, bh);
    }
    return true;
}

// C fragment: (g, 2 tig) (g, 2 tig + 1) (g + 8, 2 tig) (g + 8, 2 tig + 1)
template <bool ACC>
SKL_DEV void tc_tile_store(int m, int n, int i0, int c0, const float (&acc)[4], float alpha, float* C, int ldc,
                           float* __restrict__ Cg, int ldg, float* __restrict__ tau)
{
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int i = i0 + g + (e >> 1) * 8, c = c0 + 2 * tig + (e & 1);
        if (i >= m || c >= n) continue;
        const float v = alpha * acc[e];
        if (Cg) {
            Cg[i + (int64_t)c * ldg] = v;
            if (i == c) tau[i] = v;
        } else if (ACC) {
            C[i * ldc + c] += v;
        } else {
            C[i * ldc + c] = v;
        }
    }
}

template <bool TA, int MA, bool TB, int MB, bool ACC>
SKL_DEV void blk_mul_tc(int m, int n, int kk, const float* A, int lda, const float* B, int ldb,
                        const float* __restrict__ sB, float alpha, float* C, int ldc,
                        float* __restrict__ Cg, int ldg, float* __restrict__ tau)
{
    float acc[4];
    int i0 = 0, c0 = 0;
    const bool act = tc_tile<TA, MA, TB, MB>(threadIdx.x >> 5, m, n, kk, A, lda, B, ldb, sB, acc, i0, c0);
    __syncthreads();
    if (act) tc_tile_store<ACC>(m, n, i0, c0, acc, alpha, C, ldc, Cg, ldg, tau);
    __syncthreads();
}

// Tiles of a product: the warps a phase gives it.
SKL_DEV int tc_tiles(int m, int n) { return ((m + 15) >> 4) * ((n + 7) >> 3); }

// Off-diagonal blocks of X = U^{-1} (upper) and, when L is given, of Y =
// L^{-1} (unit lower), np x np (np a multiple of 16, at most 64), once the
// 16 x 16 diagonal blocks hold the inverses: recursive doubling,
//   [A B; 0 C]^{-1} = [A^{-1}, -A^{-1} B C^{-1}; 0, C^{-1}],
//   [A 0; B C]^{-1} = [A^{-1}, 0; -C^{-1} B A^{-1}, C^{-1}],
// with every pair of a level (and the U and L pairs) in one phase of warp
// tiles: two block barriers per product level instead of two per product.
// tmp holds 64 x 36 (ldt = 36): U pairs in rows 0..31, L pairs in 32..63,
// pair q of a level at column 16 q.
SKL_DEV void inv_offdiag_tc(const float* U, int ldu, float* X, int ldx, const float* L, int ldl, float* Y,
                            int ldy, int np, float* tmp, int ldt)
{
    const int warp = threadIdx.x >> 5;
    for (int w = kDB; w < np; w *= 2) {
        // phase 1: tmp_U = U_12 X_22, tmp_L = L_21 Y_11 for every pair
        {
            float acc[4];
            int i0 = 0, c0 = 0, m = 0, n = 0;
            float* C = nullptr;
            bool act = false;
            int base = 0;
            for (int p0 = 0; p0 + w < np; p0 += 2 * w) {
                const int n2 = min(w, np - p0 - w), q = p0 / (2 * w);
                const int tU = tc_tiles(w, n2);
                if (warp >= base && warp < base + tU) {
                    act = tc_tile<false, kMFull, false, kMUpper>(warp - base, w, n2, n2, U + p0 * ldu + p0 + w,
                                                                 ldu, X + (p0 + w) * ldx + p0 + w, ldx,
                                                                 nullptr, acc, i0, c0);
                    C = tmp + 16 * q;
                    m = w;
                    n = n2;
                }
                base += tU;
                if (L) {
                    const int tL = tc_tiles(n2, w);
                    if (warp >= base && warp < base + tL) {
                        act = tc_tile<false, kMFull, false, kMLowerUnit>(warp - base, n2, w, w,
                                                                         L + (p0 + w) * ldl + p0, ldl,
                                                                         Y + p0 * ldy + p0, ldy, nullptr, acc,
                                                                         i0, c0);
                        C = tmp + 32 * ldt + 16 * q;
                        m = n2;
                        n = w;
                    }
                    base += tL;
                }
            }
            __syncthreads();
            if (act) tc_tile_store<false>(m, n, i0, c0, acc, 1.f, C, ldt, nullptr, 0, nullptr);
            __syncthreads();
        }
        // phase 2: X_12 = -X_11 tmp_U, Y_21 = -Y_22 tmp_L
        {
            float acc[4];
            int i0 = 0, c0 = 0, m = 0, n = 0, ldc = 0;
            float* C = nullptr;
            bool act = false;
            int base = 0;
            for (int p0 = 0; p0 + w < np; p0 += 2 * w) {
                const int n2 = min(w, np - p0 - w), q = p0 / (2 * w);
                const int tU = tc_tiles(w, n2);
                if (warp >= base && warp < base + tU) {
                    act = tc_tile<false, kMUpper, false, kMFull>(warp - base, w, n2, w, X + p0 * ldx + p0, ldx,
                                                                 tmp + 16 * q, ldt, nullptr, acc, i0, c0);
                    C = X + p0 * ldx + p0 + w;
                    ldc = ldx;
                    m = w;
                    n = n2;
                }
                base += tU;
                if (L) {
                    const int tL = tc_tiles(n2, w);
                    if (warp >= base && warp < base + tL) {
                        act = tc_tile<false, kMLowerUnit, false, kMFull>(warp - base, n2, w, n2,
                                                                         Y + (p0 + w) * ldy + p0 + w, ldy,
                                                                         tmp + 32 * ldt + 16 * q, ldt, nullptr,
                                                                         acc, i0, c0);
                        C = Y + (p0 + w) * ldy + p0;
                        ldc = ldy;
                        m = n2;
                        n = w;
                    }
                    base += tL;
                }
            }
            __syncthreads();
            if (act) tc_tile_store<false>(m, n, i0, c0, acc, -1.f, C, ldc, nullptr, 0, nullptr);
            __syncthreads();
        }
    }
}

// 2 x 2 tiles for FP64: 4 x 4 tiles measured slower inside the small kernels
// (their k ranges trim less under the triangular masks).
template <typename T, bool TA, int MA, bool TB, int MB, bool ACC = false>
SKL_DEV void blk_mul(int m, int n, int kk, const T* A, int lda, const T* B, int ldb,
                     const T* __restrict__ sB, T alpha, T* C, int ldc, T* __restrict__ Cg = nullptr,
                     int ldg = 0, T* __restrict__ tau = nullptr)
{
    if constexpr (std::is_same<T, float>::value)
        blk_mul_tc<TA, MA, TB, MB, ACC>(m, n, kk, A, lda, B, ldb, sB, alpha, C, ldc, Cg, ldg, tau);
    else
        blk_mul_t<T, TA, MA, TB, MB, ACC, 2>(m, n, kk, A, lda, B, ldb, sB, alpha, C, ldc, Cg, ldg, tau);
}

// Off-diagonal blocks of X = U^{-1} (np x np upper, np a multiple of 16)
// once X's 16 x 16 diagonal blocks hold the inverses of U's: recursive
// doubling, [A B; 0 C]^{-1} = [A^{-1}, -A^{-1} B C^{-1}; 0, C^{-1}].  tmp holds
// 32 x 32 (ldt).
template <typename T>
SKL_DEV void inv_upper_offdiag(const T* U, int ldu, T* X, int ldx, int np, T* tmp, int ldt)
{
    for (int w = kDB; w < np; w *= 2) {
        for (int p0 = 0; p0 + w < np; p0 += 2 * w) {
            const int n2 = min(w, np - p0 - w);
            blk_mul<T, false, kMFull, false, kMUpper>(w, n2, n2, U + p0 * ldu + p0 + w, ldu,
                                                     X + (p0 + w) * ldx + p0 + w, ldx, nullptr, T(1),
                                                     tmp, ldt);
            blk_mul<T, false, kMUpper, false, kMFull>(w, n2, w, X + p0 * ldx + p0, ldx, tmp, ldt,
                                                     nullptr, T(-1), X + p0 * ldx + p0 + w, ldx);
        }
    }
}

// Strict lower off-diagonal blocks of Y = L^{-1} (np x np unit lower) once
// Y's diagonal blocks hold the inverses of L's:
// [A 0; B C]^{-1} = [A^{-1}, 0; -C^{-1} B A^{-1}, C^{-1}].
template <typename T>
SKL_DEV void inv_unit_lower_offdiag(const T* L, int ldl, T* Y, int ldy, int np, T* tmp, int ldt)
{
    for (int w = kDB; w < np; w *= 2) {
        for (int p0 = 0; p0 + w < np; p0 += 2 * w) {
            const int n2 = min(w, np - p0 - w);
            blk_mul<T, false, kMFull, false, kMLowerUnit>(n2, w, w, L + (p0 + w) * ldl + p0, ldl,
                                                         Y + p0 * ldy + p0, ldy, nullptr, T(1), tmp,
                                                         ldt);
            blk_mul<T, false, kMLowerUnit, false, kMFull>(n2, w, n2, Y + (p0 + w) * ldy + p0 + w, ldy,
                                                         tmp, ldt, nullptr, T(-1),
                                                         Y + (p0 + w) * ldy + p0, ldy);
        }
    }
}

// Cholesky G = R^T R (np x np, np a multiple of 16, both triangles given) with
// X = R^{-1}: R (upper, zeros below) over G, X (upper, zeros below) to Xs.
// Gaussian elimination of [G | I] on 16 warps, in place: row i of the work
// matrix holds G's Schur complement at the columns not yet eliminated and row i
// of R^{-T} at the others (unnormalised until the end).  Warp w keeps rows 4 w ..
// 4 w + 3 in registers, two columns per lane.  In round r warp r eliminates its
// four rows among themselves with shuffles and publishes them with their
// multiples by the pivots' reciprocals; one barrier later the warps below
// subtract the four products, whose row factors are the same published rows (the
// complement is symmetric).  Bound by the chain through warp r in FP32, by the
// FP64 pipe and that chain in FP64.  64 x 64: 20,600 cycles (FP64 157,000); with
// blocks of 16 factored and inverted by one warp and block products over 32
// warps between them ~37,000 (260,000); with a rolled loop of one pivot per
// barrier 31,000 (144,000).
// A pivot that is not above 32 eps times its mass sets *bad to 1 and leaves zeros
// in its row of R and its row and column of X.  BOOST: it is replaced by that
// bound (by 1 if the mass is not positive, which sets *bad to 2).
template <typename T, bool BOOST = false>
SKL_DEV void chol_inv_small(T* G, int ldx, int np, const T* __restrict__ mass, T eps, T* Xs, int* bad)
{
    constexpr int kRows = 4, kWarps = 64 / kRows;
    struct alignas(16) Quad { T v[kRows]; };
    // by column: the four rows of a round, and those times their pivots' reciprocals
    __shared__ Quad s_row[2][64], s_mul[2][64];
    const unsigned full = 0xffffffffu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i0 = kRows * warp;
    __syncthreads();
    if (warp < kWarps) {
        T a[kRows][2];
#pragma unroll
        for (int j = 0; j < kRows; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = lane + 32 * h;
                a[j][h] = i0 < np && c < np ? G[(i0 + j) * ldx + c] : T(0);
            }
#pragma unroll 1
        for (int r = 0; kRows * r < np; ++r) {
            const int k0 = kRows * r;
            const bool up = k0 >= 32;             // the half that holds the round's columns
            const int rl = lane - (k0 & 31);      // 0..3: the lane's column of that half is k0 + rl
            T dd[kRows];
            int flag = 0;
            if (warp == r) {
                T l[kRows][2];
#pragma unroll
                for (int j = 0; j < kRows; ++j) {
                    const int src = (k0 & 31) + j;
                    const T cur = up ? a[j][1] : a[j][0];
                    const T d = __shfl_sync(full, cur, src);
                    const T ms = mass[k0 + j], bound = T(32) * eps * ms;
                    const bool pos = ms > T(0), ok = pos && d > bound;
                    dd[j] = ok ? d : BOOST ? (pos ? bound : T(1)) : T(0);
                    const T inv = ok || BOOST ? t_rcp_chain(dd[j]) : T(0);
                    flag = max(flag, ok ? 0 : BOOST && !pos ? 2 : 1);
                    // from here on the pivot's column belongs to R^{-T}: 1 in its row
                    if (rl == j) {
#pragma unroll
                        for (int q = j; q < kRows; ++q) {
                            const T v = q == j ? T(1) : T(0);
                            if (up) a[q][1] = v;
                            else a[q][0] = v;
                        }
                    }
                    l[j][0] = a[j][0] * inv;
                    l[j][1] = a[j][1] * inv;
#pragma unroll
                    for (int q = j + 1; q < kRows; ++q) {
                        const T f = __shfl_sync(full, cur, src + q - j);
                        a[q][0] -= f * l[j][0];
                        a[q][1] -= f * l[j][1];
                    }
                }
                // the round's columns right of a pivot: eliminated in the rows below
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    Quad vr, vl;
#pragma unroll
                    for (int j = 0; j < kRows; ++j) {
                        vr.v[j] = a[j][h];
                        vl.v[j] = (h == 1) == up && rl > j && rl < kRows ? T(0) : l[j][h];
                    }
                    s_row[r & 1][lane + 32 * h] = vr;
                    s_mul[r & 1][lane + 32 * h] = vl;
                }
            }
            asm volatile("bar.sync 1, 512;" ::: "memory");
            if (warp == r) {
                if (flag && lane == 0) atomicMax(bad, flag);
                T sc[kRows];
#pragma unroll
                for (int j = 0; j < kRows; ++j) sc[j] = dd[j] > T(0) ? t_rcp(t_sqrt(dd[j])) : T(0);
#pragma unroll
                for (int j = 0; j < kRows; ++j)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int k = k0 + j, c = lane + 32 * h;
                        if (c >= np) continue;
                        const T v = a[j][h] * sc[j];
                        G[k * ldx + c] = c < k ? T(0) : c == k ? dd[j] * sc[j] : v;
                        Xs[c * ldx + k] = c > k ? T(0) : v;
                    }
            } else if (warp > r && i0 < np) {
                if (rl >= 0 && rl < kRows) {
#pragma unroll
                    for (int q = 0; q < kRows; ++q) {
                        if (up) a[q][1] = T(0);
                        else a[q][0] = T(0);
                    }
                }
                const Quad m0 = s_mul[r & 1][lane], m1 = s_mul[r & 1][lane + 32];
#pragma unroll
                for (int q = 0; q < kRows; ++q) {
                    const Quad f = s_row[r & 1][i0 + q];
#pragma unroll
                    for (int j = 0; j < kRows; ++j) {
                        a[q][0] -= f.v[j] * m0.v[j];
                        a[q][1] -= f.v[j] * m1.v[j];
                    }
                }
            }
        }
    }
    __syncthreads();
}

// Modified LU of A (np x np) in place (L strict lower, U upper), signs to
// sg, and in Z: L^{-1} (strict lower, unit diagonal implied) and U^{-1}
// (upper).  Blocked right-looking by 16: warp 0 factors the diagonal block,
// warps 0 and 1 invert its L and U factors into Z, then U12 = L11^{-1} A12,
// L21 = A21 U11^{-1} and A22 -= L21 U12 as block products.
template <typename T>
SKL_DEV void mlu_inv_small(T* A, int ldx, int np, T* sg, T* Z, T* tmp, int ldt)
{
    for (int k0 = 0; k0 < np; k0 += kDB) {
        const int rest = np - k0 - kDB;
        T* A11 = A + k0 * ldx + k0;
        T* Z11 = Z + k0 * ldx + k0;
        if (threadIdx.x < 32) warp16_mlu<T>(A11, ldx, sg + k0);
        __syncthreads();
        if (threadIdx.x < 32) warp16_inv_unit_lower<T>(A11, ldx, Z11, ldx);
        else if (threadIdx.x < 64) warp16_inv_upper<T>(A11, ldx, Z11, ldx, false);
        __syncthreads();
        if (rest > 0) {
            T* A12 = A11 + kDB;
            T* A21 = A11 + kDB * ldx;
            if constexpr (std::is_same<T, float>::value) {
                // U12 = L11^{-1} A12 and L21 = A21 U11^{-1} in one phase
                const int warp = threadIdx.x >> 5, t12 = tc_tiles(kDB, rest);
                float acc[4];
                int i0 = 0, c0 = 0;
                bool act;
                if (warp < t12)
                    act = tc_tile<false, kMLowerUnit, false, kMFull>(warp, kDB, rest, kDB, Z11, ldx, A12, ldx,
                                                                     nullptr, acc, i0, c0);
                else
                    act = tc_tile<false, kMFull, false, kMUpper>(warp - t12, rest, kDB, kDB, A21, ldx, Z11,
                                                                 ldx, nullptr, acc, i0, c0);
                __syncthreads();
                if (act) {
                    if (warp < t12) tc_tile_store<false>(kDB, rest, i0, c0, acc, 1.f, A12, ldx, nullptr, 0, nullptr);
                    else tc_tile_store<false>(rest, kDB, i0, c0, acc, 1.f, A21, ldx, nullptr, 0, nullptr);
                }
                __syncthreads();
            } else {
                blk_mul<T, false, kMLowerUnit, false, kMFull>(kDB, rest, kDB, Z11, ldx, A12, ldx, nullptr,
                                                             T(1), A12, ldx);
                blk_mul<T, false, kMFull, false, kMUpper>(rest, kDB, kDB, A21, ldx, Z11, ldx, nullptr, T(1),
                                                         A21, ldx);
            }
            blk_mul<T, false, kMFull, false, kMFull, true>(rest, rest, kDB, A21, ldx, A12, ldx, nullptr,
                                                           T(-1), A11 + kDB * ldx + kDB, ldx);
        }
    }
    if constexpr (std::is_same<T, float>::value) {
        inv_offdiag_tc(A, ldx, Z, ldx, A, ldx, Z, ldx, np, tmp, ldt);
    } else {
        inv_upper_offdiag<T>(A, ldx, Z, ldx, np, tmp, ldt);
        inv_unit_lower_offdiag<T>(A, ldx, Z, ldx, np, tmp, ldt);
    }
}

// Padded size of the b x b algebra and the workspace layout of the small
// kernels: four np x np blocks (row-major, ld = np + 4), a 64 x 36 product
// scratch, and 3 np entries.
__host__ __device__ inline int small_np(int b) { return (b + kDB - 1) / kDB * kDB; }
template <typename T>
size_t chol_small_smem_bytes(int b)
{
    const size_t np = (size_t)small_np(b);
    return (4 * np * (np + 4) + 64 * 36 + 3 * np) * sizeof(T) + 256;
}

}  // namespace skl
