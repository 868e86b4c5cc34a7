// k_dense.cu -- randomized Hartley transform + hashing sketch for dense A.
//
// Reference: rand_hashing_dct (src/dense_helpers.cpp:83-112):
//   D = random signs (gen_scaled_rand_signs, :7-16),
//   Y = DHT_N( D * A / sqrt(N) ) column by column (fast_unitary_transform,
//       src/fast_unitary_transform.cpp:42-121, FFTW_DHT via fftw_r2r.cpp:33-51),
//   SA = (1/sqrt(k)) * S * Y  with S's values +-1/sqrt(k)  (sketch(),
//       src/sketching.cpp:39-62), same for b.
//
// GB300 mapping: one CTA per column.  The column is read once from HBM
// (multiplied by D/sqrt(N) on load), transformed in shared memory, and hashed
// into its m sketch rows by a fixed-order gather over S's bucket lists, so
// HDA never exists in HBM.  The DHT of a real length-N vector is computed from
// a complex FFT of half length L = N/2 (even/odd packing) and H = Re F - Im F.
// FP32 columns run a decimation-in-frequency FFT in place in shared memory; FP64
// columns, or lengths beyond shared memory, Stockham passes with radices 7, 5, 4,
// 3, 2 through a global scratch slab per CTA; the right-hand side (one FP64
// column) the same passes over the whole GPU.
#include <cmath>

#include "skl_internal.hpp"
#include "launch.cuh"
#include "common.cuh"

namespace skl {

constexpr int kFftThreads = 1024;
constexpr int kFftMaxRadices = 32;
constexpr int kFftSmemMaxL = 25 * 1024;        // shared-memory path limit

template <typename T> struct Cplx;
template <> struct Cplx<float> { using type = float2; };
template <> struct Cplx<double> { using type = double2; };

template <typename C> SKL_DEV C cmk(double re, double im);
template <> SKL_DEV float2 cmk<float2>(double re, double im) { return make_float2((float)re, (float)im); }
template <> SKL_DEV double2 cmk<double2>(double re, double im) { return make_double2(re, im); }
template <typename C> SKL_DEV C cadd(C a, C b) { a.x += b.x; a.y += b.y; return a; }
template <typename C> SKL_DEV C csub(C a, C b) { a.x -= b.x; a.y -= b.y; return a; }
template <typename C> SKL_DEV C cmul(C a, C b)
{
    C r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}

// exp(-2 pi i * num / den) in the working precision, 0 <= num < den < 2^31
// (32-bit operands: a 64-bit remainder or division per twiddle is a long
// emulated sequence).
template <typename T>
SKL_DEV typename Cplx<T>::type twiddle(int num, int den)
{
    if constexpr (std::is_same<T, float>::value) {
        float s, c;
        sincospif(-2.0f * (float)num / (float)den, &s, &c);
        return make_float2(c, s);
    } else {
        double s, c;
        sincospi(-2.0 * (double)num / (double)den, &s, &c);
        return make_double2(c, s);
    }
}

// The R-th roots of unity of the small DFTs, exp(-2 pi i j / R), as compile-
// time constants: cos and sin by their Taylor series (the argument reduced to
// [-pi, pi], 30 terms: far below double rounding there), so the radix-3/5/7
// butterflies carry no runtime trigonometry.
constexpr double kPiD = 3.14159265358979323846;
constexpr double cx_sin(double x)
{
    double term = x, sum = x;
    for (int n = 1; n < 30; ++n) {
        term *= -x * x / ((2.0 * n) * (2.0 * n + 1.0));
        sum += term;
    }
    return sum;
}
constexpr double cx_cos(double x)
{
    double term = 1.0, sum = 1.0;
    for (int n = 1; n < 30; ++n) {
        term *= -x * x / ((2.0 * n - 1.0) * (2.0 * n));
        sum += term;
    }
    return sum;
}
constexpr double root_angle(int j, int R)
{
    const double a = -2.0 * kPiD * (double)(j % R) / (double)R;
    return a < -kPiD ? a + 2.0 * kPiD : a;
}
template <int R>
struct Roots {
    double re[R], im[R];
    constexpr Roots() : re(), im()
    {
        for (int j = 0; j < R; ++j) {
            re[j] = cx_cos(root_angle(j, R));
            im[j] = cx_sin(root_angle(j, R));
        }
    }
};
template <typename T, int R>
SKL_DEV typename Cplx<T>::type small_root(int j)
{
    constexpr Roots<R> w{};
    typename Cplx<T>::type r;
    r.x = (T)w.re[j % R];
    r.y = (T)w.im[j % R];
    return r;
}

// In-register R-point DFT (forward) of v[0..R).
template <typename T, int R>
SKL_DEV void dft_small(typename Cplx<T>::type* v)
{
    using C = typename Cplx<T>::type;
    if constexpr (R == 2) {
        C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (R == 4) {
        C a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
        C b0 = cadd(v[1], v[3]), b1 = csub(v[1], v[3]);
        // -i * b1
        C mb1;
        mb1.x = b1.y;
        mb1.y = -b1.x;
        v[0] = cadd(a0, b0);
        v[2] = csub(a0, b0);
        v[1] = cadd(a1, mb1);
        v[3] = csub(a1, mb1);
    } else {
        C out[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            C acc = v[0];
#pragma unroll
            for (int t = 1; t < R; ++t) acc = cadd(acc, cmul(v[t], small_root<T, R>(q * t)));
            out[q] = acc;
        }
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = out[q];
    }
}

// Butterfly i of a radix-R Stockham pass with parameter p (product of the
// radices already applied): inputs x[i + q*L/R], twiddles exp(-2 pi i q k/(pR)),
// outputs y[(i-k)*R + k + q*p], k = i mod p.
template <typename T, int R>
SKL_DEV void butterfly_load(const typename Cplx<T>::type* x, int L, int p, int i,
                            typename Cplx<T>::type* v)
{
    const int T_ = L / R;
    const int k = i % p;
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = x[i + q * T_];
    if (p > 1 && k > 0) {
        // w^q for w = exp(-2 pi i k / (pR)): one sincospi, then powers
        const typename Cplx<T>::type w = twiddle<T>(k, p * R);
        typename Cplx<T>::type wq = w;
#pragma unroll
        for (int q = 1; q < R; ++q) {
            v[q] = cmul(v[q], wq);
            if (q + 1 < R) wq = cmul(wq, w);
        }
    }
    dft_small<T, R>(v);
}

template <typename T, int R>
SKL_DEV void butterfly_store(typename Cplx<T>::type* y, int p, int i, const typename Cplx<T>::type* v)
{
    const int k = i % p;
    const int j = (i - k) * R + k;
#pragma unroll
    for (int q = 0; q < R; ++q) y[j + q * p] = v[q];
}

template <typename T, int R>
SKL_DEV void pass_pingpong(const typename Cplx<T>::type* x, typename Cplx<T>::type* y, int L, int p)
{
    using C = typename Cplx<T>::type;
    const int nb = L / R;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        C v[R];
        butterfly_load<T, R>(x, L, p, i, v);
        butterfly_store<T, R>(y, p, i, v);
    }
    __syncthreads();
}

struct FftPlan {
    int L;
    int nr;
    int radix[kFftMaxRadices];
};

// Complex forward FFT of length L, ping-pong between buf and alt; the result's buffer.
template <typename T>
SKL_DEV typename Cplx<T>::type* fft_run(const FftPlan& P, typename Cplx<T>::type* buf,
                                        typename Cplx<T>::type* alt)
{
    using C = typename Cplx<T>::type;
    int p = 1;
    C* x = buf;
    C* y = alt;
    for (int s = 0; s < P.nr; ++s) {
        const int R = P.radix[s];
        switch (R) {
        case 2: pass_pingpong<T, 2>(x, y, P.L, p); break;
        case 3: pass_pingpong<T, 3>(x, y, P.L, p); break;
        case 4: pass_pingpong<T, 4>(x, y, P.L, p); break;
        case 5: pass_pingpong<T, 5>(x, y, P.L, p); break;
        default: pass_pingpong<T, 7>(x, y, P.L, p); break;
        }
        C* t = x;
        x = y;
        y = t;
        p *= R;
    }
    return x;
}

// z[t] = x[2t] + i x[2t+1] of the column a (n entries, zeros beyond) times D scale.
template <typename T>
SKL_DEV typename Cplx<T>::type dht_packed(const double* __restrict__ a, int n, const double* __restrict__ D, T sc,
                                          int t)
{
    const int i0 = 2 * t, i1 = 2 * t + 1;
    T x0 = i0 < n ? (T)a[i0] : T(0);
    T x1 = i1 < n ? (T)a[i1] : T(0);
    if (i0 < n && D[i0] < 0) x0 = -x0;
    if (i1 < n && D[i1] < 0) x1 = -x1;
    typename Cplx<T>::type z;
    z.x = x0 * sc;
    z.y = x1 * sc;
    return z;
}

// H[k] and H[N-k] from Z[k] = zk, Z[L-k] = zc and w = exp(-2 pi i k / N):
// X[k] = (Z[k] + conj(Z[L-k]))/2 - i/2 w (Z[k] - conj(Z[L-k])),
// H[k] = Re X[k] - Im X[k], H[N-k] = Re X[k] + Im X[k]; also H[0], H[L] for k = 0.
template <typename T>
SKL_DEV void dht_pair(typename Cplx<T>::type zk, typename Cplx<T>::type zc, typename Cplx<T>::type w, T& hk, T& hnk)
{
    const T er = (zk.x + zc.x) * T(0.5), ei = (zk.y - zc.y) * T(0.5);   // even part
    const T or_ = (zk.y + zc.y) * T(0.5), oi = -(zk.x - zc.x) * T(0.5); // odd part
    const T xr = er + (w.x * or_ - w.y * oi);
    const T xi = ei + (w.x * oi + w.y * or_);
    hk = xr - xi;
    hnk = xr + xi;
}

// Bucket sums of one transformed column: SA[h] = sum over the bucket of h
// (increasing source row) of alpha * (+-1/sqrt(k)) * H[i], the order of csc_mv 'n'.
template <typename T>
SKL_DEV T bucket_sum(const T* H, const int* __restrict__ bptr, const unsigned* __restrict__ bent, int h, T av)
{
    T acc = T(0);
    for (int q = bptr[h]; q < bptr[h + 1]; ++q) {
        const unsigned e = bent[q];
        const T hv = H[e & 0x7fffffffu];
        acc += (e & 0x80000000u) ? -av * hv : av * hv;
    }
    return acc;
}

// FP64 columns, or lengths beyond shared memory: a CTA per column, ping-pong in gscratch.
template <typename T>
__global__ void __launch_bounds__(kFftThreads)
k_dht_hash(const double* __restrict__ A, int64_t lda, int n, int d, const double* __restrict__ D,
           FftPlan P, double scale, const int* __restrict__ bptr, const unsigned* __restrict__ bent,
           int m, double alpha_v, T* __restrict__ SA, int64_t ld, double* __restrict__ Yout,
           int64_t ldy, typename Cplx<T>::type* __restrict__ gscratch)
{
    pdl_wait();
    using C = typename Cplx<T>::type;
    C* buf = gscratch + (size_t)blockIdx.x * 2 * P.L;
    C* alt = buf + P.L;
    const int L = P.L, N = 2 * L;
    for (int j = blockIdx.x; j < d; j += gridDim.x) {
        for (int t = threadIdx.x; t < L; t += blockDim.x)
            buf[t] = dht_packed<T>(A + (int64_t)j * lda, n, D, (T)scale, t);
        __syncthreads();
        const C* Z = fft_run<T>(P, buf, alt);
        T* H = reinterpret_cast<T*>(Z == buf ? alt : buf);
        for (int kk = threadIdx.x; kk < L; kk += blockDim.x) {
            T hk, hnk;
            dht_pair<T>(Z[kk], Z[(L - kk) % L], twiddle<T>(kk, N), hk, hnk);
            H[kk] = hk;
            if (kk != 0) H[N - kk] = hnk;
        }
        if (threadIdx.x == 0) H[L] = Z[0].x - Z[0].y;
        __syncthreads();
        if (Yout) {
            for (int k = threadIdx.x; k < N; k += blockDim.x) Yout[k + (int64_t)j * ldy] = (double)H[k];
        }
        if (SA) {
            for (int h = threadIdx.x; h < m; h += blockDim.x)
                SA[h + (int64_t)j * ld] = bucket_sum<T>(H, bptr, bent, h, (T)alpha_v);
        }
        __syncthreads();
    }
}

// One column over the whole GPU (the right-hand side, FP64): a launch per pass.
// A single CTA takes 1,380 us for 40,000 rows, these ~10 launches 58 us.
__global__ void k_dht_load(const double* __restrict__ a, int n, const double* __restrict__ D, double scale, int L,
                           double2* __restrict__ z)
{
    pdl_wait();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < L) z[t] = dht_packed<double>(a, n, D, scale, t);
}
template <int R>
__global__ void k_dht_pass(const double2* __restrict__ x, double2* __restrict__ y, int L, int p)
{
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= L / R) return;
    double2 v[R];
    butterfly_load<double, R>(x, L, p, i, v);
    butterfly_store<double, R>(y, p, i, v);
}
__global__ void k_dht_unpack(const double2* __restrict__ Z, int L, double* __restrict__ H)
{
    pdl_wait();
    const int kk = blockIdx.x * blockDim.x + threadIdx.x;
    if (kk >= L) return;
    double hk, hnk;
    dht_pair<double>(Z[kk], Z[(L - kk) % L], twiddle<double>(kk, 2 * L), hk, hnk);
    H[kk] = hk;
    if (kk != 0) H[2 * L - kk] = hnk;
    else H[L] = Z[0].x - Z[0].y;
}
__global__ void k_dht_gather(const double* __restrict__ H, const int* __restrict__ bptr,
                             const unsigned* __restrict__ bent, int m, double alpha_v, double* __restrict__ Sb)
{
    pdl_wait();
    const int h = blockIdx.x * blockDim.x + threadIdx.x;
    if (h < m) Sb[h] = bucket_sum<double>(H, bptr, bent, h, alpha_v);
}

// ---- FP32 columns in shared memory ----------------------------------------------
// A CTA per column at a time.  The FFT is decimation in frequency in place: a pass
// of radix R = R1 R2 (two radices in registers between one load and one store of
// shared memory) reads and writes the same places, so no thread holds more than
// R values and no second buffer is needed; the results end in digit-reversed
// order, which the last two steps undo through tables made once per call: the
// places of each pair of frequencies for the unpacking, done in place, and the
// bucket entries with source rows replaced by places.
// The transform without a sketch computes places where it needs them (two per
// frequency and column): it uses no scratch, so that calls which share one may
// overlap.  40,000 x 1,000: 489 us; 1,342 with a division per digit, 711 for the
// autosorted passes before this kernel.
// The column is read once, with the next column's lines on their way to L2; the
// signs are bits in shared memory, and the FP64 values are rounded to FP32 on
// their bits (a warp's FP64 conversion holds the pipe for 16 cycles: 10 us of a
// column of 40,000).  Passes with odd R come last: their short strides then meet
// each bank once.  40,000 x 4,000: 1,350 us (cycles of a column: load 14,000, FFT
// 20,000, the rest unpacking and buckets), 2,690 with one radix per pass,
// autosorted through local memory (floor: 188 us for the read).
constexpr int kDifThreads = 512;
constexpr int kDifMaxPasses = 16;
struct DifPlan {
    int L, np;
    int r1[kDifMaxPasses], r2[kDifMaxPasses];
    // the digits of a frequency, first pass's first: radix, stride of its place, and
    // ceil(2^32 / radix) (quotients exact below 2^16)
    int nd;
    int dr[kFftMaxRadices], ds[kFftMaxRadices];
    unsigned dm[kFftMaxRadices];
};

// Forward DFT of the R values v[off + q step].
template <int R, int NV>
SKL_DEV void dft_at(float2 (&v)[NV], int off, int step)
{
    if constexpr (R == 2 || R == 4) {
        float2 w[R];
#pragma unroll
        for (int q = 0; q < R; ++q) w[q] = v[off + q * step];
        dft_small<float, R>(w);
#pragma unroll
        for (int q = 0; q < R; ++q) v[off + q * step] = w[q];
    } else if constexpr (R > 1) {
        // symmetric halves: X_q, X_{R-q} = x0 + sum cos a_h -+ i sum sin b_h
        constexpr int H = (R - 1) / 2;
        constexpr Roots<R> w{};
        const float2 x0 = v[off];
        float2 a[H], b[H];
        float2 s = x0;
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const float2 u = v[off + (h + 1) * step], t = v[off + (R - 1 - h) * step];
            a[h] = cadd(u, t);
            b[h] = csub(u, t);
            s = cadd(s, a[h]);
        }
        v[off] = s;
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            float2 m = x0, y = make_float2(0.f, 0.f);
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const float c = (float)w.re[q * (h + 1) % R], sn = -(float)w.im[q * (h + 1) % R];
                m.x = fmaf(c, a[h].x, m.x);
                m.y = fmaf(c, a[h].y, m.y);
                y.x = fmaf(sn, b[h].x, y.x);
                y.y = fmaf(sn, b[h].y, y.y);
            }
            v[off + q * step] = make_float2(m.x + y.y, m.y - y.x);
            v[off + (R - q) * step] = make_float2(m.x - y.y, m.y + y.x);
        }
    }
}

// One pass over blocks of B values: butterfly j < S = B / (R1 R2) of a block.
template <int R1, int R2>
SKL_DEV void dif_pass(float2* z, int L, int B)
{
    constexpr int R = R1 * R2;
    const int S = B / R, nb = L / R;
    const unsigned magic = S > 1 ? (unsigned)(((1ull << 32) + S - 1) / S) : 0u;   // i / S, exact for i < 2^16
    for (int i = threadIdx.x; i < nb; i += kDifThreads) {
        const int blk = S > 1 ? (int)__umulhi((unsigned)i, magic) : i;
        const int j = i - blk * S;
        float2* x = z + blk * B + j;
        float2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = x[q * S];
#pragma unroll
        for (int q2 = 0; q2 < R2; ++q2) dft_at<R1, R>(v, q2, R2);   // v[t1 R2 + q2]
        if constexpr (R2 > 1) {
#pragma unroll
            for (int t1 = 1; t1 < R1; ++t1)
#pragma unroll
                for (int q2 = 1; q2 < R2; ++q2) v[t1 * R2 + q2] = cmul(v[t1 * R2 + q2], small_root<float, R>(t1 * q2));
#pragma unroll
            for (int t1 = 0; t1 < R1; ++t1) dft_at<R2, R>(v, t1 * R2, 1);
        }
        if (S > 1) {
            // times exp(-2 pi i j t / B), t = t1 + R1 t2: powers of two values of their own
            const float2 w1 = twiddle<float>(j, B);
            const float2 w2 = R2 > 1 ? twiddle<float>(R1 * j, B) : w1;
            float2 u2 = make_float2(1.f, 0.f);
#pragma unroll
            for (int t2 = 0; t2 < R2; ++t2) {
                float2 u = u2;
#pragma unroll
                for (int t1 = 0; t1 < R1; ++t1) {
                    if (t1 > 0) u = t2 == 0 && t1 == 1 ? w1 : cmul(u, w1);
                    if (t1 > 0 || t2 > 0) v[t1 * R2 + t2] = cmul(v[t1 * R2 + t2], u);
                }
                if (t2 + 1 < R2) u2 = t2 == 0 ? w2 : cmul(u2, w2);
            }
        }
#pragma unroll
        for (int q = 0; q < R; ++q) x[q * S] = v[q];
    }
    __syncthreads();
}

SKL_DEV void dif_run(const DifPlan& P, float2* z)
{
    int B = P.L;
    for (int s = 0; s < P.np; ++s) {
        const int r1 = P.r1[s], r2 = P.r2[s];
        switch (8 * r1 + r2) {
        case 8 * 7 + 3: dif_pass<7, 3>(z, P.L, B); break;
        case 8 * 7 + 2: dif_pass<7, 2>(z, P.L, B); break;
        case 8 * 5 + 5: dif_pass<5, 5>(z, P.L, B); break;
        case 8 * 5 + 4: dif_pass<5, 4>(z, P.L, B); break;
        case 8 * 5 + 3: dif_pass<5, 3>(z, P.L, B); break;
        case 8 * 5 + 2: dif_pass<5, 2>(z, P.L, B); break;
        case 8 * 4 + 4: dif_pass<4, 4>(z, P.L, B); break;
        case 8 * 4 + 3: dif_pass<4, 3>(z, P.L, B); break;
        case 8 * 4 + 2: dif_pass<4, 2>(z, P.L, B); break;
        case 8 * 3 + 3: dif_pass<3, 3>(z, P.L, B); break;
        case 8 * 3 + 2: dif_pass<3, 2>(z, P.L, B); break;
        case 8 * 7 + 1: dif_pass<7, 1>(z, P.L, B); break;
        case 8 * 5 + 1: dif_pass<5, 1>(z, P.L, B); break;
        case 8 * 4 + 1: dif_pass<4, 1>(z, P.L, B); break;
        case 8 * 3 + 1: dif_pass<3, 1>(z, P.L, B); break;
        default: dif_pass<2, 1>(z, P.L, B); break;
        }
        B /= r1 * r2;
    }
}

// Place of frequency k.
SKL_DEV int dif_place(const DifPlan& P, int k)
{
    int pos = 0;
    for (int h = 0; h < P.nd; ++h) {
        const int q = (int)__umulhi((unsigned)k, P.dm[h]);
        pos += (k - q * P.dr[h]) * P.ds[h];
        k = q;
    }
    return pos;
}

// part[k], k <= L / 2: the places of frequencies k and L - k (upper half);
// place[i], i < N: where H[i] ends, as an index of floats.
__global__ void k_dif_tables(DifPlan P, unsigned* __restrict__ part, unsigned* __restrict__ place)
{
    pdl_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x, L = P.L;
    if (k >= L) return;
    const int p = dif_place(P, k);
    if (k <= L / 2) part[k] = (unsigned)p | ((unsigned)dif_place(P, k ? L - k : 0) << 16);
    place[k] = 2 * p;
    place[k ? 2 * L - k : L] = 2 * p + 1;
}
__global__ void k_dif_entries(const int* __restrict__ bptr, const unsigned* __restrict__ bent, int m,
                              const unsigned* __restrict__ place, unsigned* __restrict__ out)
{
    pdl_wait();
    const int total = bptr[m];
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < total; q += gridDim.x * blockDim.x) {
        const unsigned e = bent[q];
        out[q] = place[e & 0x7fffffffu] | (e & 0x80000000u);
    }
}

// (float)a by its bits (round to nearest even); zeros, infinities, NaN and what
// is not normal in FP32 by the conversion.
SKL_DEV float round_f32(double a)
{
    const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
    const unsigned ex = (hi >> 20) & 0x7ffu;
    if (ex - 897u >= 253u) return (float)a;
    unsigned f = ((ex - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
    f += ((lo & 0x1fffffffu) + (f & 1u)) > 0x10000000u ? 1u : 0u;
    return __uint_as_float(f | (hi & 0x80000000u));
}

__global__ void __launch_bounds__(kDifThreads, 1)
k_dht_hash_smem(const double* __restrict__ A, int64_t lda, int n, int d, const double* __restrict__ D, DifPlan P,
                double scale, const int* __restrict__ bptr, const unsigned* __restrict__ ent, int m, double alpha_v,
                float* __restrict__ SA, int64_t ld, double* __restrict__ Yout, int64_t ldy,
                const unsigned* __restrict__ part)
{
    pdl_wait();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* z = reinterpret_cast<float2*>(smem_raw);
    const float* H = reinterpret_cast<const float*>(z);
    const int L = P.L, N = 2 * L;
    unsigned* sgn = reinterpret_cast<unsigned*>(z + L);   // bit i: D[i] < 0
    for (int w = threadIdx.x; w < (N + 31) / 32 * 32; w += kDifThreads) {
        const unsigned bits = __ballot_sync(0xffffffffu, w < n && D[w] < 0);
        if ((threadIdx.x & 31) == 0) sgn[w / 32] = bits;
    }
    __syncthreads();
    const float sc = (float)scale, av = (float)alpha_v;
    for (int j = blockIdx.x; j < d; j += gridDim.x) {
        const double* a = A + (int64_t)j * lda;
        if (j + (int)gridDim.x < d) {
            const char* nx = reinterpret_cast<const char*>(a + (int64_t)gridDim.x * lda);
            for (int64_t o = (int64_t)threadIdx.x * 128; o < (int64_t)n * 8; o += kDifThreads * 128)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + o));
        }
        // x[2t] + i x[2t+1] with D's signs, scaled; pairs of loads where they align
        const bool vec = ((reinterpret_cast<uintptr_t>(a) & 15) == 0);
        auto put = [&](int t, double x0, double x1) {
            const unsigned w = sgn[t >> 4] >> (2 * (t & 15));
            z[t] = make_float2(__uint_as_float(__float_as_uint(round_f32(x0)) ^ (w << 31)) * sc,
                               __uint_as_float(__float_as_uint(round_f32(x1)) ^ ((w >> 1) << 31)) * sc);
        };
        const int full = vec ? n / 2 : 0;
        constexpr int U = 8;
        int t = threadIdx.x;
        for (; t + (U - 1) * kDifThreads < full; t += U * kDifThreads) {
            double2 v[U];
#pragma unroll
            for (int q = 0; q < U; ++q) v[q] = reinterpret_cast<const double2*>(a)[t + q * kDifThreads];
#pragma unroll
            for (int q = 0; q < U; ++q) put(t + q * kDifThreads, v[q].x, v[q].y);
        }
#pragma unroll 4
        for (; t < L; t += kDifThreads)
            put(t, 2 * t < n ? a[2 * t] : 0.0, 2 * t + 1 < n ? a[2 * t + 1] : 0.0);
        __syncthreads();
        dif_run(P, z);
        // the pair of places (p, p2) holds Z[k], Z[L-k]: H[k], H[N-k] to p, H[L-k],
        // H[L+k] to p2 (exp(-2 pi i (L-k) / N) = -conj of k's)
#pragma unroll 4
        for (int k = threadIdx.x; k <= L / 2; k += kDifThreads) {
            int p, p2;
            if (SA) {
                const unsigned e = part[k];
                p = e & 0xffffu;
                p2 = e >> 16;
            } else {
                p = dif_place(P, k);
                p2 = dif_place(P, k ? L - k : 0);
            }
            const float2 zk = z[p], zc = z[p2];
            const float2 w = twiddle<float>(k, N);
            float2 h, g;
            dht_pair<float>(zk, zc, w, h.x, h.y);
            if (k == 0) h.y = zk.x - zk.y;
            dht_pair<float>(zc, zk, make_float2(-w.x, w.y), g.x, g.y);
            if (p2 != p) z[p2] = g;
            z[p] = h;
        }
        __syncthreads();
        if (Yout) {
            double* y = Yout + (int64_t)j * ldy;
            for (int k = threadIdx.x; k < L; k += kDifThreads) {
                const float2 h = z[dif_place(P, k)];   // H[k], H[N-k] (H[L] for k = 0)
                y[k] = (double)h.x;
                y[k ? N - k : L] = (double)h.y;
            }
        }
        if (SA) {
            // buckets h and h + 512: each sum in its order, eight entries' loads at a time
            auto step = [&](int q, int q1, const unsigned (&e)[4], float& acc) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float hv = H[e[c] & 0x7fffffffu];
                    if (q + c < q1) acc += (e[c] & 0x80000000u) ? -av * hv : av * hv;
                }
            };
            for (int h = threadIdx.x; h < m; h += 2 * kDifThreads) {
                const int h2 = h + kDifThreads;
                const bool two = h2 < m;
                int q = bptr[h], r = two ? bptr[h2] : 0;
                const int q1 = bptr[h + 1], r1 = two ? bptr[h2 + 1] : 0;
                float a0 = 0.f, a1 = 0.f;
                while (q < q1 || r < r1) {
                    unsigned e[4], f[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        e[c] = q + c < q1 ? ent[q + c] : 0u;
                        f[c] = r + c < r1 ? ent[r + c] : 0u;
                    }
                    step(q, q1, e, a0);
                    step(r, r1, f, a1);
                    q += 4;
                    r += 4;
                }
                SA[h + (int64_t)j * ld] = a0;
                if (two) SA[h2 + (int64_t)j * ld] = a1;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------ host side --
static bool factor_plan(int64_t L, FftPlan& P)
{
    P.L = (int)L;
    P.nr = 0;
    int64_t r = L;
    const int pref[] = {4, 2, 3, 5, 7};
    for (int f : {7, 5, 3}) {
        while (r % f == 0) {
            if (P.nr >= kFftMaxRadices) return false;
            P.radix[P.nr++] = f;
            r /= f;
        }
    }
    while (r % 4 == 0) {
        if (P.nr >= kFftMaxRadices) return false;
        P.radix[P.nr++] = 4;
        r /= 4;
    }
    while (r % 2 == 0) {
        if (P.nr >= kFftMaxRadices) return false;
        P.radix[P.nr++] = 2;
        r /= 2;
    }
    (void)pref;
    return r == 1;
}

static bool smooth(int64_t x)
{
    for (int f : {2, 3, 5, 7})
        while (x % f == 0) x /= f;
    return x == 1;
}

// Transform length: N = n when n is even and n/2 factors into 2,3,5,7;
// otherwise (or with wisdom) the next such even length >= n.  Zero padding
// keeps the transform orthonormal (the reference pads in its wisdom mode,
// src/fast_unitary_transform.cpp:63-64,98-99).
int64_t dht_length(int64_t n, int wisdom)
{
    int64_t N = n + (n & 1);
    if (!wisdom && smooth(N / 2)) return N;
    while (!smooth(N / 2)) N += 2;
    return N;
}

// Opt-in shared memory per block (the same on every GB300), read once; the
// initialisation is thread-safe for concurrent solves.
static size_t smem_optin_bytes()
{
    static const size_t v = [] {
        int dev = 0, o = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&o, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        return (size_t)o;
    }();
    return v;
}

// Passes of one or two radices, R1 R2 <= 25: the largest left with the largest that
// fits; multiples of 4 first, odd ones (and a lone 2) last.
static DifPlan dif_plan(const FftPlan& P)
{
    int cnt[8] = {};
    for (int s = 0; s < P.nr; ++s) ++cnt[P.radix[s]];
    cnt[4] += cnt[2] / 2;
    cnt[2] %= 2;
    DifPlan Q{};
    Q.L = P.L;
    auto push = [&](int a, int b) {
        Q.r1[Q.np] = a;
        Q.r2[Q.np++] = b;
    };
    for (int f : {7, 5, 4, 3, 2})
        while (cnt[f] > 0) {
            --cnt[f];
            int g = 1;
            for (int c : {5, 4, 3, 2})
                if (c <= f && cnt[c] > 0 && f * c <= 25) {
                    g = c;
                    --cnt[c];
                    break;
                }
            push(f, g);
        }
    // stable: multiples of 4, then the others, each by falling size
    for (int i = 1; i < Q.np; ++i)
        for (int j = i; j > 0; --j) {
            auto key = [&](int q) { const int R = Q.r1[q] * Q.r2[q]; return (R % 4 == 0 ? 1000 : 0) + R; };
            if (key(j - 1) >= key(j)) break;
            std::swap(Q.r1[j - 1], Q.r1[j]);
            std::swap(Q.r2[j - 1], Q.r2[j]);
        }
    int S = Q.L;
    for (int s = 0; s < Q.np; ++s)
        for (int r : {Q.r1[s], Q.r2[s]}) {
            if (r == 1) continue;
            S /= r;
            Q.dr[Q.nd] = r;
            Q.ds[Q.nd] = S;
            Q.dm[Q.nd++] = (unsigned)(((1ull << 32) + r - 1) / r);
        }
    return Q;
}

template <typename T>
static void launch_dht(const double* A, int64_t lda, int64_t n, int64_t d, const double* D,
                       int64_t N, const int* bptr, const unsigned* bent, int k, int64_t m, T* SA,
                       int64_t ld, double* Yout, int64_t ldy, void* gscratch_buf,
                       size_t gscratch_bytes, cudaStream_t st)
{
    using C = typename Cplx<T>::type;
    FftPlan P;
    if (N & 1) fail(SKL_ERR_INVALID, "DHT length must be even");
    if (!factor_plan(N / 2, P)) fail(SKL_ERR_INVALID, "DHT length must factor into 2,3,5,7");
    const double scale = 1.0 / std::sqrt((double)N);
    const double alpha_v = (1.0 / std::sqrt((double)k)) * (1.0 / std::sqrt((double)k));
    unsigned grid = (unsigned)std::min<int64_t>(d, 152);
    if constexpr (std::is_same<T, float>::value) {
        // in shared memory where the column, the signs and (in the scratch) a sketch's
        // tables fit
        const size_t need = (size_t)P.L * sizeof(C) + (size_t)((N + 31) / 32) * 4;
        const size_t tables = SA ? ((size_t)P.L + N + (size_t)N * k) * 4 : 0;
        const DifPlan Q = dif_plan(P);
        if (P.L <= kFftSmemMaxL && need + 1024 <= smem_optin_bytes() && tables <= gscratch_bytes) {
            unsigned* part = (unsigned*)gscratch_buf;
            unsigned* place = part + P.L;
            unsigned* ent = place + N;
            if (SA) {
                launch_k(k_dif_tables, (unsigned)((P.L + 255) / 256), 256, 0, st, Q, part, place);
                launch_k(k_dif_entries, (unsigned)std::min<int64_t>((N * k + 255) / 256, 1216), 256, 0, st, bptr, bent,
                         (int)m, (const unsigned*)place, ent);
                SKL_LAUNCHED();
                SKL_LAUNCHED();
            }
            allow_max_dynamic_smem((const void*)k_dht_hash_smem);
            launch_k(k_dht_hash_smem, grid, kDifThreads, need, st, A, lda, (int)n, (int)d, D, Q, scale, bptr,
                     (const unsigned*)ent, (int)m, alpha_v, SA, ld, Yout, ldy, (const unsigned*)part);
            SKL_LAUNCHED();
            return;
        }
    }
    const size_t per = 2 * (size_t)P.L * sizeof(C);
    grid = (unsigned)std::min<int64_t>(grid, (int64_t)(gscratch_bytes / per));
    if (grid == 0) fail(SKL_ERR_ALLOC, "DHT scratch too small");
    launch_k(k_dht_hash<T>, grid, kFftThreads, 0, st, A, lda, (int)n, (int)d, D, P, scale, bptr, bent,
             (int)m, alpha_v, SA, ld, Yout, ldy, (C*)gscratch_buf);
    SKL_LAUNCHED();
}

void dht_load_kernels()
{
    cudaFuncAttributes fa;
    SKL_CUDA(cudaFuncGetAttributes(&fa, k_dht_hash_smem));
    SKL_CUDA(cudaFuncGetAttributes(&fa, k_dht_hash<float>));
    SKL_CUDA(cudaFuncGetAttributes(&fa, k_dht_hash<double>));
}

size_t dht_scratch_bytes(int64_t N, int precision)
{
    const size_t csz = precision == SKL_PREC_FP64 ? sizeof(double2) : sizeof(float2);
    return (size_t)152 * 2 * (size_t)(N / 2) * csz;
}

template <typename T>
void dht_hash(const double* A, int64_t lda, int64_t n, int64_t d, const double* D, int64_t N,
              const int* bptr, const unsigned* bent, int k, int64_t m, T* SA, int64_t ld,
              double* Yout, int64_t ldy, void* scratch, size_t scratch_bytes, cudaStream_t st)
{
    launch_dht<T>(A, lda, n, d, D, N, bptr, bent, k, m, SA, ld, Yout, ldy, scratch, scratch_bytes, st);
}

template void dht_hash<float>(const double*, int64_t, int64_t, int64_t, const double*, int64_t,
                              const int*, const unsigned*, int, int64_t, float*, int64_t, double*,
                              int64_t, void*, size_t, cudaStream_t);
template void dht_hash<double>(const double*, int64_t, int64_t, int64_t, const double*, int64_t,
                               const int*, const unsigned*, int, int64_t, double*, int64_t,
                               double*, int64_t, void*, size_t, cudaStream_t);

// Sb: the same transform of b (one column, FP64 arithmetic) and bucket gather.
void dht_hash_rhs(const double* b, int64_t n, const double* D, int64_t N, const int* bptr,
                  const unsigned* bent, int k, int64_t m, double* Sb, void* scratch,
                  size_t scratch_bytes, cudaStream_t st)
{
    FftPlan P;
    if (N & 1) fail(SKL_ERR_INVALID, "DHT length must be even");
    if (!factor_plan(N / 2, P)) fail(SKL_ERR_INVALID, "DHT length must factor into 2,3,5,7");
    if (scratch_bytes < 2 * (size_t)P.L * sizeof(double2)) fail(SKL_ERR_ALLOC, "DHT scratch too small");
    const double scale = 1.0 / std::sqrt((double)N);
    const double alpha_v = (1.0 / std::sqrt((double)k)) * (1.0 / std::sqrt((double)k));
    double2* x = (double2*)scratch;
    double2* y = x + P.L;
    constexpr int kT = 64;   // small blocks: a pass has a few thousand butterflies
    auto blocks = [](int64_t c) { return (unsigned)((c + kT - 1) / kT); };
    launch_k(k_dht_load, blocks(P.L), kT, 0, st, b, (int)n, D, scale, P.L, x);
    SKL_LAUNCHED();
    int p = 1;
    for (int s = 0; s < P.nr; ++s) {
        const int R = P.radix[s];
        auto* f = R == 2 ? k_dht_pass<2> : R == 3 ? k_dht_pass<3> : R == 4 ? k_dht_pass<4> : R == 5 ? k_dht_pass<5>
                                                                                                  : k_dht_pass<7>;
        launch_k(f, blocks(P.L / R), kT, 0, st, (const double2*)x, y, P.L, p);
        SKL_LAUNCHED();
        std::swap(x, y);
        p *= R;
    }
    launch_k(k_dht_unpack, blocks(P.L), kT, 0, st, (const double2*)x, P.L, (double*)y);
    launch_k(k_dht_gather, blocks(m), kT, 0, st, (const double*)y, bptr, bent, (int)m, alpha_v, Sb);
    SKL_LAUNCHED();
    SKL_LAUNCHED();
}

// kFroParts partial sums of squares of a dense column-major matrix, in FP64: its
// entries may be as small or large as FP64 holds squares of.
__global__ void __launch_bounds__(256)
k_fro_partial(const double* __restrict__ A, int64_t lda, int64_t n, int64_t d, double* __restrict__ out)
{
    pdl_wait();
    __shared__ double red[8];
    double acc = 0.0;
    for (int64_t j = blockIdx.x; j < d; j += gridDim.x)
#pragma unroll 4
        for (int64_t i = threadIdx.x; i < n; i += 256) {
            const double v = A[i + j * lda];
            acc = fma(v, v, acc);
        }
    acc = block_sum(acc, red);
    if (threadIdx.x == 0) out[blockIdx.x] = acc;
}

void fro_partials(const double* A, int64_t lda, int64_t n, int64_t d, double* out, cudaStream_t st)
{
    launch_k(k_fro_partial, kFroParts, 256, 0, st, A, lda, n, d, out);
    SKL_LAUNCHED();
}

// kStatusRange where a column that is not zero has a sum of squares outside
// [2^-120, 2^126].
__global__ void __launch_bounds__(256)
k_column_range(const float* __restrict__ X, int64_t ld, int m, unsigned* __restrict__ status)
{
    pdl_wait();
    __shared__ float red[8];
    const float* x = X + blockIdx.x * ld;
    float s = 0.f;
    bool any = false;
    for (int i = threadIdx.x; i < m; i += 256) {
        s = fmaf(x[i], x[i], s);
        any |= x[i] != 0.f;
    }
    s = block_sum(s, red);
    any = __syncthreads_or(any);
    if (threadIdx.x == 0 && any && !(s >= 0x1p-120f && s <= 0x1p126f)) atomicOr(status, kStatusRange);
}

void check_column_range(const float* X, int64_t ld, int64_t m, int64_t d, unsigned* status, cudaStream_t st)
{
    launch_k(k_column_range, (unsigned)d, 256, 0, st, X, ld, (int)m, status);
    SKL_LAUNCHED();
}

}  // namespace skl
