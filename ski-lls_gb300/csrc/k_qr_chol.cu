// k_qr_chol.cu -- the CholeskyQR2 panel of the randomized QR (FP32): the
// tall products as GEMMs over the whole GPU and the b x b algebra
// (Cholesky, triangular inverses, modified LU) in single-CTA kernels.  The
// algorithm and its failure rule are described with the panel loop in
// k_qr.cu.
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "skl_internal.hpp"
#include "launch.cuh"
#include "common.cuh"
#include "k_gemm.cuh"
#include "chol_small.cuh"

namespace skl {

// Pass 1: R1 and X1 = R1^{-1} from G1 (column-major b x b, ldg = b).  Sets
// *fail (1 on a Cholesky breakdown, else 0).
template <typename T>
__global__ void __launch_bounds__(kSmallThreads, 1)
k_chol_small1(const T* __restrict__ G, int b, T* __restrict__ R1, T* __restrict__ X1,
              int* __restrict__ fail)
{
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int np = small_np(b);
    const int LDX = np + 4;
    T* S0 = (T*)smem_raw;
    T* S1 = S0 + (size_t)np * LDX;
    T* mass = S1 + (size_t)np * LDX;
    __shared__ int s_bad;
    const T eps = std::is_same<T, float>::value ? T(5.9604645e-08) : T(1.1102230246251565e-16);
    if (threadIdx.x == 0) s_bad = 0;
    // G padded with the identity beyond b
    for (int e = threadIdx.x; e < np * np; e += kSmallThreads) {
        const int i = e % np, c = e / np;
        S0[i * LDX + c] = (i < b && c < b) ? G[i + c * b] : (i == c ? T(1) : T(0));
    }
    for (int k = threadIdx.x; k < np; k += kSmallThreads) mass[k] = k < b ? G[k * b + k] : T(1);
    __syncthreads();
    chol_inv_small<T>(S0, LDX, np, mass, eps, S1, &s_bad);
    for (int e = threadIdx.x; e < b * b; e += kSmallThreads) {
        const int i = e / b, c = e % b;
        R1[e] = S0[i * LDX + c];     // row-major b x b
        X1[c * b + i] = S1[i * LDX + c];   // column-major (a GEMM operand)
    }
    if (threadIdx.x == 0) *fail = s_bad ? 1 : 0;
}

// Pass 2 and the reconstruction: from G2 (column-major), R1 (row-major) and
// the first b rows of Q (column-major, ldq) writes W = R2^{-1} U^{-1}
// (column-major b x b), T (ldt), tau, the panel's first b rows of A (R_H on
// and above the diagonal, L below) and of V (unit lower L).  Does nothing if
// pass 1 failed; sets *fail on a pass-2 breakdown (A untouched).
template <typename T>
__global__ void __launch_bounds__(kSmallThreads, 1)
k_chol_small2(const T* __restrict__ G, int b, const T* __restrict__ R1g, const T* __restrict__ Q,
              int64_t ldq, T* __restrict__ A, int64_t ld, int j0, T* __restrict__ V, int64_t ldv,
              T* __restrict__ Tout, int ldt, T* __restrict__ tau_out, T* __restrict__ Wg,
              int* __restrict__ fail)
{
    pdl_wait();
    if (*fail) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int np = small_np(b);
    const int LDX = np + 4;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T* S0 = (T*)smem_raw;                        // R1 -> R = R2 R1
    T* S1 = S0 + (size_t)np * LDX;               // G2 -> R2 -> L^{-1} \ U^{-1}
    T* S2 = S1 + (size_t)np * LDX;               // X2 -> W
    T* S3 = S2 + (size_t)np * LDX;               // Q(0:b,:) -> Q1 -> L \ U
    T* tmp = S3 + (size_t)np * LDX;              // 64 x 36 product scratch
    T* Sg = tmp + 64 * 36;
    T* mass = Sg + np;
    __shared__ int s_bad;
    const T eps = std::is_same<T, float>::value ? T(5.9604645e-08) : T(1.1102230246251565e-16);
    if (threadIdx.x == 0) s_bad = 0;
    // G2 padded with the identity, Q(0:b,:) with zeros, beyond b
    for (int e = threadIdx.x; e < np * np; e += kSmallThreads) {
        const int i = e % np, c = e / np;
        const bool in = i < b && c < b;
        S1[i * LDX + c] = in ? G[i + c * b] : (i == c ? T(1) : T(0));
        S3[i * LDX + c] = in ? Q[i + (int64_t)c * ldq] : T(0);
        S0[c * LDX + i] = in ? R1g[c * b + i] : (i == c ? T(1) : T(0));   // row-major source
    }
    for (int k = threadIdx.x; k < np; k += kSmallThreads) mass[k] = T(1);
    __syncthreads();
    // Gershgorin distance of G2 from the identity
    for (int i = wid; i < b; i += kSmallThreads / 32) {
        T sabs = T(0);
        for (int c = lane; c < b; c += 32) sabs += t_abs(S1[i * LDX + c] - (c == i ? T(1) : T(0)));
        sabs = warp_sum(sabs);
        if (lane == 0 && !(sabs <= T(0.5))) s_bad = 1;
    }
    __syncthreads();
    if (s_bad) {
        if (threadIdx.x == 0) *fail = 1;
        return;
    }
    chol_inv_small<T>(S1, LDX, np, mass, eps, S2, &s_bad);  // R2 over S1, X2 -> S2
    if (s_bad) {
        if (threadIdx.x == 0) *fail = 1;
        return;
    }
    blk_mul<T, false, kMFull, false, kMUpper>(b, b, b, S3, LDX, S2, LDX, nullptr, T(1), S3, LDX);   // Q1 = Q(0:b,:) X2
    blk_mul<T, false, kMUpper, false, kMUpper>(b, b, b, S1, LDX, S0, LDX, nullptr, T(1), S0, LDX);  // R = R2 R1
    mlu_inv_small<T>(S3, LDX, np, Sg, S1, tmp, 36);              // Q1 - S = L U; S1 = L^{-1} \ U^{-1}
    blk_mul<T, false, kMUpper, false, kMUpper>(b, b, b, S2, LDX, S1, LDX, nullptr, T(1), S2, LDX);  // W = X2 U^{-1}
    blk_mul<T, false, kMUpper, true, kMUpperUnit>(b, b, b, S3, LDX, S1, LDX, Sg, T(-1), nullptr, 0,
                                                   Tout, ldt, tau_out + j0);   // T = -U S L^{-T}
    for (int e = threadIdx.x; e < b * b; e += kSmallThreads) {
        const int g = e % b, c = e / b;          // column-major targets
        Wg[e] = S2[g * LDX + c];
        const T l = (g > c) ? S3[g * LDX + c] : T(0);
        A[(int64_t)(j0 + g) + (int64_t)(j0 + c) * ld] = (g <= c) ? Sg[g] * S0[g * LDX + c] : l;
        V[(int64_t)g + (int64_t)c * ldv] = (g > c) ? l : (g == c ? T(1) : T(0));
    }
}

// A(j0+b : j0+M, j0 : j0+b) = V(b : M, :) once the panel succeeded.
template <typename T>
__global__ void k_chol_copy_down(const T* __restrict__ V, int64_t ldv, T* __restrict__ A, int64_t ld,
                                 int j0, int M, int b, const int* __restrict__ fail)
{
    pdl_wait();
    if (*fail) return;
    const int rows = M - b;
    const int c = blockIdx.y;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x)
        A[(int64_t)(j0 + b + r) + (int64_t)(j0 + c) * ld] = V[(int64_t)(b + r) + (int64_t)c * ldv];
}

// Host side: one panel P (M x b, column-major, ld) = A(j0:m, j0:j0+b).
template <typename T>
void chol_panel(T* P, int64_t ld, int M, int b, int j0, T* A, T* cg, T* cr1, T* cx1, T* cw, T* tmp,
                T* V, int64_t ldv, T* Tm, int ldt, T* tau, T* part, int64_t part_cap, int* fail,
                cudaStream_t st)
{
    const size_t ssm = chol_small_smem_bytes<T>(b);
    allow_max_dynamic_smem((const void*)k_chol_small1<T>);
    allow_max_dynamic_smem((const void*)k_chol_small2<T>);
    gemm<T>(true, false, b, b, M, T(1), P, ld, P, ld, T(0), cg, b, part, part_cap, st);
    launch_k(k_chol_small1<T>, 1, kSmallThreads, ssm, st, cg, b, cr1, cx1, fail);
    SKL_CUDA(cudaGetLastError());
    SKL_LAUNCHED();
    gemm<T>(false, false, M, b, b, T(1), P, ld, cx1, b, T(0), tmp, M, nullptr, 0, st);
    gemm<T>(true, false, b, b, M, T(1), tmp, M, tmp, M, T(0), cg, b, part, part_cap, st);
    launch_k(k_chol_small2<T>, 1, kSmallThreads, ssm, st, cg, b, cr1, tmp, M, A, ld, j0, V, ldv, Tm, ldt,
                                                    tau, cw, fail);
    SKL_CUDA(cudaGetLastError());
    SKL_LAUNCHED();
    gemm<T>(false, false, M - b, b, b, T(1), tmp + b, M, cw, b, T(0), V + b, ldv, nullptr, 0, st);
    dim3 gc((unsigned)std::max<int64_t>(1, std::min<int64_t>((M - b + 255) / 256, 64)), b);
    launch_k(k_chol_copy_down<T>, gc, 256, 0, st, V, ldv, A, ld, j0, M, b, fail);
    SKL_LAUNCHED();
}

template <>
void chol_panel<double>(double*, int64_t, int, int, int, double*, double*, double*, double*, double*,
                        double*, double*, int64_t, double*, int, double*, double*, int64_t, int*,
                        cudaStream_t)
{
    fail(SKL_ERR_INVALID, "CholeskyQR2 panel: FP32 only");
}

template void chol_panel<float>(float*, int64_t, int, int, int, float*, float*, float*, float*, float*,
                                float*, float*, int64_t, float*, int, float*, float*, int64_t, int*,
                                cudaStream_t);

}  // namespace skl
