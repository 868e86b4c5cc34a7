// k_lsqr_persist.cu -- the whole LSQR iteration in one persistent kernel.
//
// The iteration of k_lsqr.cu (src/IterSolver.cpp:160-284) is five kernels of
// 5-15 us that each do a few microseconds of work on problems up to a few
// thousand columns: 30-40 us per iteration went into ramp-up, tails, the
// launches between them and a host round trip per four iterations (20,000 x
// 1,000: 36 us per iteration, here 19; 31,013 x 1,507: 40 -> 21; 2,000 x 60: 30 ->
// 13; 1e6 x 1e4, which streams 0.6 GB: 288 -> 196).  Here the CTAs stay resident and
// the phases are separated by grid barriers:
//   A  z = M v        rows of the triangle, v in shared memory
//   B  u = A z - (alpha / beta) u,  partial ||u||^2      z in shared memory
//   C  t = A^T u      column chunks
//   D  v = M^T t / beta - (beta / alpha) v,  partial ||v||^2   t in shared memory
// u and v stay unnormalised and every scale (1 / alpha, 1 / beta) is applied by
// the phase after the one that would have waited for the norm, so an iteration
// has four barriers; each CTA reduces the norms' partials itself, in the same
// order, and runs the scalar recurrences redundantly.  Small problems run as
// one 16-CTA cluster (hardware barrier, no co-residency to ask for, so several
// of them share the GPU), larger ones as a grid of one CTA per SM, whose CTAs first
// make sure that all of them run (meet_all).
//
// Work split: phases A and D deal the triangle's rows (columns) to the CTAs in
// snake order, so that every CTA has long and short ones, and cut each into S
// segments, one warp per segment; the segments' sums meet in shared memory and
// one thread per row finishes it.  Phase C cuts columns into chunks of at most
// kChunkSteps steps, so that a power-law column does not hang on one warp; the
// last chunk of a column to finish adds the column's chunks up in order.
// Every sum has a fixed order: results are bitwise reproducible.
// FP64 is slow enough (see Sum) that the scalar recurrences of one lane take 2-5
// us: a warp of their own runs them beside phases A (alpha) and C (beta), and
// another one updates y and w of the previous iteration beside phase C.
// On small problems an iteration is latency, ~1.5 us per barrier (a release add and
// an acquire poll by one thread; fences of its own around them cost 0.3 us more)
// and ~2.5 to 4 us per phase.  What a phase reads that the previous one does not
// write (first row and chunk, old u and v, column numbers) is on its way before
// the staged vector arrives; with the short barriers, 22.6 -> 19.1 us per iteration at
// 20,000 x 1,000.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "skl_internal.hpp"
#include "launch.cuh"
#include "common.cuh"
#include "lsqr_types.cuh"
#include "tc_ptx.cuh"

namespace skl {

namespace {

// Threads per CTA: 512 (two CTAs of different solves fit an SM, barriers and block
// sums are cheaper), 1,024 for problems that stream from HBM.
constexpr int kSmallCta = 512, kBigCta = 1024;
constexpr int kCluster = 16;              // CTAs of the single-cluster variant
constexpr int kIterPerGraph = 4;          // iterations per graph of phase kernels
constexpr int kTU = 8;                    // entries per lane per step (columns)
// Steps per column chunk (1e6 x 1e4, power-law columns, LSQR of 118 iterations: 24.8 ms
// with 2, 25.3 with 4, 27.8 with 8, 29.3 with 16).
constexpr int kChunkSteps = 2;
constexpr unsigned kBarLimit = 1u << 23;  // polls before a grid barrier gives up
constexpr int kItersPerLaunch = 256;
constexpr int kNormParts = 152;

// Scalars of the iteration: one copy per CTA in the persistent kernel, two
// slots in memory otherwise (a phase kernel reads one and writes the other).
struct PScal {
    double alpha, beta, rhobar, phibar, nrm_a, nrm_ar;
    double ia, ib, coef_n, coef_t;         // 1/alpha, 1/beta, alpha/beta, beta/alpha
    double cs, sn, irho, t1, t2;
    double y_t1, y_t2, y_ia;               // the outstanding update of y and w
    double bs;                             // the right-hand side's scale, a power of two
    long long it;
    int done, flag;
    int pend;              // a finished iteration's alpha scalars are outstanding
    int ypend;             // its update of y and w is outstanding
};

struct PState {
    PScal sc[2];
    double tol;
    long long max_it;
    unsigned bar;          // grid barrier arrivals of this launch
    unsigned meet;         // its CTAs that have started; kMeetOff: called off
    int timeout;
};
constexpr unsigned kMeetOff = 1u << 31;
constexpr long long kMeetNs = 20000000;   // a launch waits this long for its CTAs

template <bool MIXED>
struct PArgs {
    using V = ValT<MIXED>;
    using MT = MatT<MIXED>;
    int n, r, d, L_n, L_t, S_seg;
    const int* rp; const int* ci; const V* cv;      // CSR
    const int* cp; const int* ri; const V* rv;      // CSC
    const int* cols; const double* opscale;
    const int4* chunks;       // per chunk: CSC range, column slot, chunks of the column
    const int* coff;          // first chunk of column slot i; coff[r] = all
    unsigned* ccnt;           // finished chunks of a column with several
    const MT* Mr; const MT* Mc; int64_t ldm;
    const double* b;
    const double* bpart;      // kNormParts partial sums of ||b||^2
    V* us; V* vs; V* z; V* t; V* tpart;
    double* vh;               // v in FP64; vs holds its pairs (FP64 path: vh itself)
    double* w; double* y;
    double* pa; double* pb;   // partials of ||v||^2, ||u||^2
    PState* S;
};

// loads of what other CTAs wrote in this launch: from L2
SKL_DEV float2 ld_cg(const float2* p) { return __ldcg(p); }
SKL_DEV double ld_cg(const double* p) { return __ldcg(p); }

template <bool CLUSTER>
SKL_DEV bool bar_all(PState* S, unsigned& gen)
{
    if constexpr (CLUSTER) {
        __syncthreads();
        cluster_sync();
        return true;
    } else {
        __shared__ int s_ok;
        __syncthreads();
        if (threadIdx.x == 0) {
            gen += gridDim.x;
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&S->bar) : "memory");
            unsigned v = 0, k = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&S->bar) : "memory");
            } while (v < gen && ++k < kBarLimit);
            s_ok = v >= gen;
        }
        __syncthreads();
        return s_ok != 0;
    }
}

SKL_DEV long long now_ns()
{
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Whether all CTAs of the grid run at once, the same answer in each.  With one that
// does not start within kMeetNs (another stream's kernel holds an SM) the launch is
// called off and the CTAs leave, the late ones too, so that the solve can go on in
// kernels that share the GPU.  A cooperative launch would wait for that kernel's
// end, which may itself wait for what the caller does after the solve.
SKL_DEV bool meet_all(PState* S)
{
    __shared__ int s_all;
    if (threadIdx.x == 0) {
        const unsigned G = gridDim.x;
        const long long t0 = now_ns();
        unsigned v = atomicAdd(&S->meet, 1u) + 1;
        for (unsigned k = 0; !(v & kMeetOff) && v < G; ++k) {
            if (now_ns() - t0 > kMeetNs || k >= kBarLimit) {
                // called off unless the last one has arrived meanwhile
                const unsigned was = atomicCAS(&S->meet, v, v | kMeetOff);
                v = was == v ? v | kMeetOff : was;
            } else {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&S->meet) : "memory");
            }
        }
        s_all = !(v & kMeetOff);
    }
    __syncthreads();
    return s_all != 0;
}

// Sum of ||u||^2.  GB300 issues two FP64 FMAs per SM and cycle, so one FP64
// instruction of a warp holds the pipe for 16 cycles whatever its active lanes: an
// epilogue of ten of them in each of 32 warps is 2.7 us.  The mixed path's u of a
// sparse problem is a float pair, and its squares are summed in pairs up to the warp,
// FP64 from there (the warps' 2^-48 average out over a few thousand of them).  What
// has one value per row of the triangle or of a tile (v, the dense u and their
// norms, y, w) is FP64 altogether: one or two warps of a CTA hold it.
template <bool MIXED>
struct Sum {
    ff a{0.f, 0.f};
    SKL_DEV void add_sq(ff x) { ff_fma(a, x, x); }
    SKL_DEV double warp() const { return ff_to_double(warp_sum_ff(a)); }
};
template <>
struct Sum<false> {
    double a = 0.0;
    SKL_DEV void add_sq(double x) { a = fma(x, x, a); }
    SKL_DEV double warp() const { return warp_sum(a); }
};

// The first nw warps' sums added up in thread 0; red is free again after the next
// barrier
SKL_DEV double sum_warps(double w, int nw, double* red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0 && warp < nw) red[warp] = w;
    __syncthreads();
    double t = 0.0;
    if (warp == 0) t = warp_sum(lane < nw ? red[lane] : 0.0);
    return t;
}

// Fixed-order sum of the CTAs' partials (one warp; every lane gets it).
SKL_DEV double sum_partials(const double* p, int np)
{
    double s = 0.0;
    for (int i = threadIdx.x & 31; i < np; i += 32) s += __ldcg(p + i);
    return warp_sum(s);
}

SKL_DEV float2 acc_store(const Acc<true>& a) { return make_float2(a.a.hi, a.a.lo); }
SKL_DEV double acc_store(const Acc<false>& a) { return a.a; }
SKL_DEV void acc_load(Acc<true>& a, float2 v) { a.a = ff{v.x, v.y}; }
SKL_DEV void acc_load(Acc<false>& a, double v) { a.a = v; }

// s = sqrt(x), r = 1 / s (0 for x = 0), each to about an ulp: the reciprocal root
// first, the root from it with one Newton correction.  Shorter than sqrt and a
// division after it, and several of them can overlap (an FP64 instruction's
// latency is what one lane waits for).
SKL_DEV void sqrt_rcp(double x, double& s, double& r)
{
    if (x > 1e-280 && x < 1e280) {
        r = rsqrt(x);
        s = x * r;
        s = fma(fma(-s, s, x), 0.5 * r, s);
    } else {
        s = sqrt(x);
        r = s > 0.0 ? 1.0 / s : 0.0;
    }
}

// s * dot - c * old, with s and c split once per phase by one thread: the FP64
// conversions of a whole CTA's warps took ~3,000 cycles of phase B
struct ScaleF {
    ff s, c;
    SKL_DEV ScaleF(double s64, double c64) : s(ff_from_double(s64)), c(ff_from_double(-c64)) {}
    SKL_DEV explicit ScaleF(float4 v) : s{v.x, v.y}, c{v.z, v.w} {}
    SKL_DEV float4 pack() const { return make_float4(s.hi, s.lo, c.hi, c.lo); }
    SKL_DEV ff operator()(const Acc<true>& dot, float2 old) const
    {
        ff v{0.f, 0.f};
        ff_fma(v, s, dot.a);
        ff_fma(v, c, ff{old.x, old.y});
        return v;
    }
};
struct ScaleD {
    double s, c;
    SKL_DEV ScaleD(double s64, double c64) : s(s64), c(c64) {}
    SKL_DEV double operator()(const Acc<false>& dot, double old) const { return dot.a * s - c * old; }
};
template <bool MIXED> using Scale = typename std::conditional<MIXED, ScaleF, ScaleD>::type;
SKL_DEV float2 to_v(ff x) { return make_float2(x.hi, x.lo); }
SKL_DEV double to_v(double x) { return x; }

template <bool MIXED>
SKL_DEV Acc<MIXED> warp_reduce(Acc<MIXED> a)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a.add(a.shfl_xor(o));
    return a;
}

// Partial dot of x[lo..hi) (contiguous, x 4-element aligned at index 0) with
// the staged vector sv, by `nl` lanes (lane index l): four elements per load.
template <bool MIXED>
SKL_DEV Acc<MIXED> dot_seg(const MatT<MIXED>* __restrict__ x, const ValT<MIXED>* sv, int lo, int hi, int l, int nl)
{
    Acc<MIXED> a0, a1;
    const int c1 = hi >> 2;                  // whole chunks end here
    int c = (lo >> 2) + l;
    // the first chunk may start before lo, the last may be ragged
    auto edge = [&](int cc) {
        for (int k = 4 * cc; k < 4 * cc + 4; ++k)
            if (k >= lo && k < hi) a0.fma_f(x[k], sv[k]);
    };
    if (l == 0 && (lo & 3)) {
        edge(c);
        c += nl;
    }
    if constexpr (MIXED) {
        const float4* x4 = reinterpret_cast<const float4*>(x);
        const float4* s4 = reinterpret_cast<const float4*>(sv);   // two entries each
        for (; c + 3 * nl < c1; c += 4 * nl) {
            float4 m[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) m[q] = __ldg(x4 + c + q * nl);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 u = s4[2 * (c + q * nl)], w = s4[2 * (c + q * nl) + 1];
                a0.fma_f(m[q].x, make_float2(u.x, u.y));
                a1.fma_f(m[q].y, make_float2(u.z, u.w));
                a0.fma_f(m[q].z, make_float2(w.x, w.y));
                a1.fma_f(m[q].w, make_float2(w.z, w.w));
            }
        }
        for (; c < c1; c += nl) {
            const float4 m = __ldg(x4 + c);
            const float4 u = s4[2 * c], w = s4[2 * c + 1];
            a0.fma_f(m.x, make_float2(u.x, u.y));
            a1.fma_f(m.y, make_float2(u.z, u.w));
            a0.fma_f(m.z, make_float2(w.x, w.y));
            a1.fma_f(m.w, make_float2(w.z, w.w));
        }
    } else {
        const double2* x2 = reinterpret_cast<const double2*>(x);
        for (; c < c1; c += nl) {
            const double2 m0 = __ldg(x2 + 2 * c), m1 = __ldg(x2 + 2 * c + 1);
            a0.fma_f(m0.x, sv[4 * c]);
            a1.fma_f(m0.y, sv[4 * c + 1]);
            a0.fma_f(m1.x, sv[4 * c + 2]);
            a1.fma_f(m1.y, sv[4 * c + 3]);
        }
    }
    if (c == c1 && 4 * c1 < hi) edge(c1);
    a0.add(a1);
    return a0;
}

constexpr int kMaxUnits = 512;            // row segments of a CTA

// What a CTA needs in every phase.
template <bool MIXED, int NT>
struct Cta {
    using V = ValT<MIXED>;
    static constexpr int kPT = NT, kPW = NT / 32;
    static constexpr int kSWarp = kPW - 1;   // the scalars' warp in phases A and C
    static constexpr int kYWarp = kPW - 2;   // the warp of y and w in phase C
    const PArgs<MIXED>& g;
    PScal& sc;              // shared memory
    V* sv;                  // staged vector, max(r, d) entries
    V* s_unit;              // kMaxUnits segment sums
    double* red;
    float4* scale;          // the phase's scales
    int tid, lane, warp, G, bid, nloc;

    // set by one thread beside the staging of the phase's vector, read after its barrier
    SKL_DEV void put_scale(double s, double c) const
    {
        if constexpr (MIXED) *scale = ScaleF(s, c).pack();
    }
    SKL_DEV Scale<MIXED> get_scale(double s, double c) const
    {
        if constexpr (MIXED) return ScaleF(*scale);
        else return ScaleD(s, c);
    }

    // Rows of the triangle this CTA owns, longest first: local row k is the q-th
    // longest, q = k G + bid (k even) or (k + 1) G - 1 - bid (k odd).
    SKL_DEV int tri_row(int k, bool rows) const
    {
        const int q = (k & 1) ? (k + 1) * G - 1 - bid : k * G + bid;
        return q >= g.r ? -1 : rows ? q : g.r - 1 - q;
    }
    // Dots of the owned rows (columns) with the staged vector: segment sums to
    // s_unit by the first nw warps.
    SKL_DEV void tri_units(const MatT<MIXED>* M, bool rows, int nw) const
    {
        for (int u = warp; u < nloc * g.S_seg; u += nw) {
            const int k = u / g.S_seg, s = u - k * g.S_seg;
            const int i = tri_row(k, rows);
            if (i < 0) continue;
            const int lo = rows ? i : 0, hi = rows ? g.r : i + 1, base = lo & ~3;
            const int len = ((hi - lo) / g.S_seg + 4) & ~3;
            const int a0 = max(lo, base + s * len);
            const int a1 = s == g.S_seg - 1 ? hi : min(hi, base + (s + 1) * len);
            Acc<MIXED> a;
            if (a0 < a1) a = dot_seg<MIXED>(M + (int64_t)i * g.ldm, sv, a0, a1, lane, 32);
            a = warp_reduce<MIXED>(a);
            if (lane == 0) s_unit[u] = acc_store(a);
        }
    }
    SKL_DEV Acc<MIXED> tri_sum(int k) const
    {
        Acc<MIXED> a;
        acc_load(a, s_unit[k * g.S_seg]);
        for (int s = 1; s < g.S_seg; ++s) {
            Acc<MIXED> o;
            acc_load(o, s_unit[k * g.S_seg + s]);
            a.add(o);
        }
        return a;
    }

    // beta_1 (one warp).  Mixed: the pairs hold b times a power of two that brings
    // ||b|| to [1, 2), so that neither they nor A^T b leave the float range; y is
    // scaled back at the end (k_lsqr_y).
    SKL_DEV void init_beta() const
    {
        const double beta = sqrt(sum_partials(g.bpart, kNormParts));
        if (lane == 0) {
            const long long e = (__double_as_longlong(beta) >> 52) & 0x7ff;   // 1 .. 1534 for a sum that is finite
            sc.bs = MIXED && beta > 0.0 && e < 0x7ff ? __longlong_as_double((2046 - e) << 52) : 1.0;
            sc.beta = beta * sc.bs;
            sc.ib = beta > 0.0 ? 1.0 / sc.beta : 0.0;
            sc.coef_t = 0.0;
        }
    }
    // u = b, once sc.bs is known to the CTA
    SKL_DEV void init_u() const
    {
        for (int i = bid * kPT + tid; i < g.n; i += G * kPT) g.us[i] = store_val<MIXED>(g.b[i] * sc.bs);
    }
    // alpha_1 (one warp); w = v, y = 0 by the warp that updates them later
    SKL_DEV void init_alpha() const
    {
        const double alpha = sqrt(sum_partials(g.pa, G));
        if (lane == 0) {
            sc.alpha = alpha;
            sc.ia = alpha > 0.0 ? 1.0 / alpha : 0.0;
            sc.coef_n = alpha * sc.ib;
            sc.rhobar = alpha;
            sc.phibar = sc.beta;
            sc.nrm_a = sc.nrm_ar = 0.0;
            sc.it = 0;
            // the reference's loop ends at once on alpha beta = 0 (IterSolver.cpp:200)
            sc.done = alpha * sc.beta == 0.0 ? 1 : 0;
            sc.flag = sc.done ? 0 : 1;
            sc.pend = sc.ypend = 0;
        }
    }
    SKL_DEV void init_yw() const
    {
        for (int i = bid * 32 + lane; i < g.r; i += G * 32) {
            g.w[i] = __ldcg(g.vh + i) * sc.ia;
            g.y[i] = 0.0;
        }
    }
    // y += t1 w, w = v + t2 w of this CTA's entries (one warp)
    SKL_DEV void update_yw() const
    {
        const double t1 = sc.y_t1, t2 = sc.y_t2, ia = sc.y_ia;
        for (int i = bid * 32 + lane; i < g.r; i += G * 32) {
            const double v = ia != 0.0 ? __ldcg(g.vh + i) * ia : 0.0;
            const double wi = g.w[i];
            g.y[i] += t1 * wi;
            g.w[i] = t2 * wi + v;
        }
    }

    // ---- A: z = M v (unscaled); alpha, stop test (last warp).  Returns with
    // sc.done decided; z is written unless it is set or `last`.
    SKL_DEV void phase_a(bool last) const
    {
        const int i0 = tid < nloc ? tri_row(tid, true) : -1;
        const int c0 = i0 >= 0 ? __ldg(g.cols + i0) : 0;
        for (int i = tid; i < g.r; i += kPT) sv[i] = ld_cg(g.vs + i);
        __syncthreads();
        if (warp < kSWarp) {
            tri_units(g.Mr, true, kSWarp);
        } else if (sc.pend) {
            const double a2 = sum_partials(g.pa, G);
            if (lane == 0) {
                // the reference skips the A^T u step when beta == 0 (IterSolver.cpp:242)
                double alpha = sc.alpha;
                if (sc.beta > 0.0) {
                    sqrt_rcp(a2, alpha, sc.ia);
                    sc.alpha = alpha;
                }
                sc.coef_n = alpha * sc.ib;
                sc.t2 = -sc.sn * alpha * sc.irho;
                sc.rhobar = -sc.cs * alpha;
                sc.it += 1;
                sc.nrm_ar = sc.phibar * alpha * fabs(sc.cs);
                if (sc.nrm_ar < g.S->tol * sc.nrm_a * sc.phibar) {
                    sc.done = 1;
                    sc.flag = 0;
                } else if (sc.it >= g.S->max_it) {
                    sc.done = 1;
                    sc.flag = 1;
                }
                sc.y_t1 = sc.t1;
                sc.y_t2 = sc.t2;
                sc.y_ia = sc.beta > 0.0 ? sc.ia : 0.0;
                sc.pend = 0;
                sc.ypend = 1;
            }
        }
        __syncthreads();
        if (last || sc.done) return;
        for (int k = tid; k < nloc; k += kPT) {
            const int i = tri_row(k, true);
            if (i < 0) continue;
            const Acc<MIXED> a = tri_sum(k);
            const int c = k == tid ? c0 : __ldg(g.cols + i);
            g.z[c] = g.opscale ? store_val<MIXED>(a.value() * g.opscale[c]) : acc_store(a);
        }
    }

    // ---- B: u = A z / alpha - (alpha / beta) u; partial ||u||^2
    // row pointers of this lane's first row: the same in every iteration
    SKL_DEV int2 first_row() const
    {
        const int per = 32 / g.L_n, i = (bid * kPW + warp) * per + lane / g.L_n;
        return i < g.n ? make_int2(__ldg(g.rp + i), __ldg(g.rp + i + 1)) : make_int2(0, 0);
    }
    SKL_DEV void phase_b(int2 row0) const
    {
        const int L = g.L_n, l = lane & (L - 1), per = 32 / L, rstep = G * kPW * per;
        if (tid == kPT - 1) put_scale(sc.ia, sc.coef_n);
        Sum<MIXED> ss;
        // the next row's entries and old u are loaded before this row's products
        int cc[4], nc[4];
        V aa[4], na[4], uo{}, nuo{};
        const int n_long = 4 * L + min(8 * L, 64);
        bool any_long = false;
        auto load_entries = [&](int i, int p0, int p1, int (&c)[4], V (&a)[4], V& u) {
            if (i < g.n && l == 0) u = ld_cg(g.us + i);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const bool ok = p0 + k * L < p1;
                c[k] = ok ? __ldg(g.ci + p0 + k * L) : 0;
                if (ok) a[k] = __ldg(g.cv + p0 + k * L);
                else a[k] = V{};
            }
        };
        int base = (bid * kPW + warp) * per;
        auto load_row = [&](int i, int& p0, int& p1, int (&c)[4], V (&a)[4], V& u) {
            p0 = p1 = 0;
            if (i < g.n) {
                p0 = __ldg(g.rp + i) + l;
                p1 = __ldg(g.rp + i + 1);
            }
            load_entries(i, p0, p1, c, a, u);
        };
        int i = base + lane / L, p0 = row0.x + l, p1 = row0.y, np0, np1;
        load_entries(i, p0, p1, cc, aa, uo);
        for (int j = tid; j < g.d; j += kPT) sv[j] = ld_cg(g.z + j);
        __syncthreads();
        const Scale<MIXED> sc2 = get_scale(sc.ia, sc.coef_n);
        for (; base < g.n; base += rstep) {
            load_row(i + rstep, np0, np1, nc, na, nuo);
            Acc<MIXED> acc, acc2;
#pragma unroll
            for (int k = 0; k < 4; k += 2) {
                acc.fma_mv(aa[k], sv[cc[k]]);
                acc2.fma_mv(aa[k + 1], sv[cc[k + 1]]);
            }
            const bool lng = p1 - (p0 - l) > n_long;
            any_long |= lng;
            if (!lng)
                for (int p = p0 + 4 * L; p < p1; p += 2 * L) {   // rows longer than 4 L
                    const int c0 = __ldg(g.ci + p);
                    acc.fma_mv(__ldg(g.cv + p), sv[c0]);
                    if (p + L < p1) {
                        const int c1 = __ldg(g.ci + p + L);
                        acc2.fma_mv(__ldg(g.cv + p + L), sv[c1]);
                    }
                }
            acc.add(acc2);
            for (int o = L / 2; o > 0; o >>= 1) acc.add(acc.shfl_xor(o));
            if (i < g.n && l == 0 && !lng) {
                const auto nv = sc2(acc, uo);
                g.us[i] = to_v(nv);
                ss.add_sq(nv);
            }
            i += rstep;
            p0 = np0;
            p1 = np1;
            uo = nuo;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                cc[k] = nc[k];
                aa[k] = na[k];
            }
        }
        // the long rows that this warp passed over, a row at a time: as two entries a
        // lane and step above, their steps wait for one another (20,000 x 1,000 with
        // 100 full rows: 115 us per iteration, 26 so); a loop of its own, since inside
        // the other one its registers would spill
        if (__any_sync(0xffffffffu, any_long))
            for (base = (bid * kPW + warp) * per; base < g.n; base += rstep) {
                i = base + lane / L;
                p0 = i < g.n ? __ldg(g.rp + i) : 0;
                p1 = i < g.n ? __ldg(g.rp + i + 1) : 0;
                unsigned todo = __ballot_sync(0xffffffffu, p1 - p0 > n_long && l == 0);
                while (todo) {
                    const int src = __ffs(todo) - 1, row = base + src / L;
                    todo &= todo - 1;
                    const int q1 = __shfl_sync(0xffffffffu, p1, src);
                    Acc<MIXED> acc, acc2;
                    for (int p = __shfl_sync(0xffffffffu, p0, src) + lane; p < q1; p += 128) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const bool ok = p + 32 * k < q1;
                            cc[k] = ok ? __ldg(g.ci + p + 32 * k) : 0;
                            if (ok) aa[k] = __ldg(g.cv + p + 32 * k);
                            else aa[k] = V{};
                        }
#pragma unroll
                        for (int k = 0; k < 4; k += 2) {
                            acc.fma_mv(aa[k], sv[cc[k]]);
                            acc2.fma_mv(aa[k + 1], sv[cc[k + 1]]);
                        }
                    }
                    acc.add(acc2);
                    acc = warp_reduce<MIXED>(acc);
                    if (lane == 0) {
                        const auto nv = sc2(acc, ld_cg(g.us + row));
                        g.us[row] = to_v(nv);
                        ss.add_sq(nv);
                    }
                }
            }
        const double tot = sum_warps(ss.warp(), kPW, red);
        if (tid == 0) g.pb[bid] = tot;
    }

    // beta and the Givens rotation (one warp, beside the chunks of phase C)
    SKL_DEV void beta_scalars() const
    {
        const double b2 = sum_partials(g.pb, G);
        if (lane == 0) {
            double beta, ib, rho, irho;
            sqrt_rcp(b2, beta, ib);
            sqrt_rcp(fma(sc.rhobar, sc.rhobar, b2), rho, irho);
            sc.beta = beta;
            sc.ib = ib;
            sc.coef_t = beta * sc.ia;
            sc.irho = irho;
            sc.cs = sc.rhobar * irho;
            sc.sn = beta * irho;
            sc.t1 = sc.cs * sc.phibar * irho;
            if (beta > 0.0) sc.nrm_a = sqrt(sc.nrm_a * sc.nrm_a + sc.alpha * sc.alpha + b2);
            sc.phibar = sc.sn * sc.phibar;
            sc.pend = 1;
            sc.ypend = 0;
        }
    }

    // ---- C: t(i) = A(:, c)^T u by chunks, on the first nw warps of each CTA
    // (ch0: this lane's first chunk, the same in every iteration)
    SKL_DEV int4 first_chunk(int nw) const
    {
        const int q = (bid * nw + warp) * (32 / g.L_t) + lane / g.L_t;
        return warp < nw && q < __ldg(g.coff + g.r) ? __ldg(g.chunks + q) : make_int4(0, 0, 0, 0);
    }
    SKL_DEV void chunks(int nw, const int4 ch0) const
    {
        if (warp >= nw) return;
        const int Lt = g.L_t, lt = lane & (Lt - 1), pert = 32 / Lt;
        const int total = __ldg(g.coff + g.r), first = (bid * nw + warp) * pert;
        for (int q0 = first; q0 < total; q0 += G * nw * pert) {
            const int q = q0 + lane / Lt;
            Acc<MIXED> acc, acc2;
            int4 ch = ch0;
            if (q < total) {
                if (q0 != first) ch = __ldg(g.chunks + q);
                for (int p = ch.x + lt; p < ch.y; p += kTU * Lt) {
                    int rr[kTU];
                    V aa[kTU], uu[kTU];
#pragma unroll
                    for (int k = 0; k < kTU; ++k) {
                        const bool ok = p + k * Lt < ch.y;
                        rr[k] = ok ? __ldg(g.ri + p + k * Lt) : -1;
                        if (ok) aa[k] = __ldg(g.rv + p + k * Lt);
                        else aa[k] = V{};
                    }
#pragma unroll
                    for (int k = 0; k < kTU; ++k) {
                        if (rr[k] >= 0) uu[k] = g.us[rr[k]];   // plain: the barrier's acquire dropped stale L1 lines
                        else uu[k] = V{};
                    }
#pragma unroll
                    for (int k = 0; k < kTU; k += 2) {
                        acc.fma_mv(aa[k], uu[k]);
                        acc2.fma_mv(aa[k + 1], uu[k + 1]);
                    }
                }
            }
            acc.add(acc2);
            for (int o = Lt / 2; o > 0; o >>= 1) acc.add(acc.shfl_xor(o));
            if (q < total && lt == 0) {
                bool fin = true;
                if (ch.w > 1) {
                    g.tpart[q] = acc_store(acc);
                    unsigned before;
                    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;"
                                 : "=r"(before)
                                 : "l"(g.ccnt + ch.z)
                                 : "memory");
                    fin = before == (unsigned)ch.w - 1;
                    if (fin) {
                        g.ccnt[ch.z] = 0;
                        const V* part = g.tpart + __ldg(g.coff + ch.z);
                        acc = Acc<MIXED>();
                        for (int k0 = 0; k0 < ch.w; k0 += 8) {
                            V x[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                if (k0 + k < ch.w) x[k] = ld_cg(part + k0 + k);
                                else x[k] = V{};
                            }
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                Acc<MIXED> o;
                                acc_load(o, x[k]);
                                acc.add(o);
                            }
                        }
                    }
                }
                if (fin) g.t[ch.z] = g.opscale ? store_val<MIXED>(acc.value() * g.opscale[g.cols[ch.z]]) : acc_store(acc);
            }
        }
    }
    SKL_DEV void phase_c(const int4 ch0) const
    {
        const int yp = sc.ypend;
        __syncthreads();   // beta_scalars clears the flag
        if (warp == kSWarp) beta_scalars();
        else if (warp == kYWarp && yp) update_yw();
        chunks(kYWarp, ch0);
    }

    // ---- D: v = M^T t / beta - (beta / alpha) v; partial ||v||^2
    SKL_DEV void phase_d() const
    {
        for (int i = tid; i < g.r; i += kPT) sv[i] = ld_cg(g.t + i);
        tri_finish();
    }
    SKL_DEV void tri_finish() const
    {
        const bool has_old = (__double_as_longlong(sc.coef_t) << 1) != 0;   // coef_t != 0
        // this thread's first entry of v, on its way beside the products
        const int j0 = tid < nloc ? tri_row(tid, false) : -1;
        double old0 = 0.0;
        if (j0 >= 0 && has_old) old0 = g.vh[j0];
        __syncthreads();
        tri_units(g.Mc, false, kPW);
        __syncthreads();
        const double ib = sc.ib, coef = sc.coef_t;
        double ss = 0.0;
        for (int k = tid; k < nloc; k += kPT) {
            const int j = tri_row(k, false);
            if (j < 0) continue;
            double old = old0;
            if (k != tid) old = has_old ? g.vh[j] : 0.0;
            const double nv = fma(-coef, old, tri_sum(k).value() * ib);
            if (ib > 0.0) {   // v stays when beta = 0 (IterSolver.cpp:242)
                g.vh[j] = nv;
                if constexpr (MIXED) g.vs[j] = store_val<true>(nv);
            }
            ss = fma(nv, nv, ss);
        }
        // only the warps that own rows hold a sum
        const int nw = min(kPW, (nloc + 31) / 32);
        if (warp < nw) ss = warp_sum(ss);
        if (nw > 1) ss = sum_warps(ss, nw, red);
        if (tid == 0) g.pa[bid] = ss;
    }
};

#define SKL_CTA(MIXED, NT)                                                                                   \
    extern __shared__ __align__(16) unsigned char smem_raw[];                                            \
    __shared__ PScal sc;                                                                                 \
    __shared__ ValT<MIXED> s_unit[kMaxUnits];                                                            \
    __shared__ double red[NT / 32];                                                                      \
    __shared__ __align__(16) float4 s_phase_scale;                                                       \
    using C = Cta<MIXED, NT>;                                                                            \
    const C c{g, sc, reinterpret_cast<ValT<MIXED>*>(smem_raw), s_unit, red, &s_phase_scale, (int)threadIdx.x,   \
                       (int)threadIdx.x & 31, (int)threadIdx.x >> 5, (int)gridDim.x, (int)blockIdx.x,    \
                       (g.r + (int)gridDim.x - 1) / (int)gridDim.x}

// The persistent iteration: up to `budget` iterations from the state in slot 0
// (start != 0: from b), back to slot 0.
template <bool MIXED, int NT, bool CLUSTER>
__global__ void __launch_bounds__(NT, 1024 / NT) k_lsqr_persist(const PArgs<MIXED> g, int start, int budget)
{
    pdl_wait();
    SKL_CTA(MIXED, NT);
    PState* S = g.S;
    if constexpr (!CLUSTER)
        if (!meet_all(S)) return;
    unsigned gen = 0;
    auto give_up = [&] {
        if (c.tid == 0) S->timeout = 1;
    };
    const int4 ch0 = c.first_chunk(C::kYWarp);
    const int2 row0 = c.first_row();
    if (start) {
        if (c.warp == C::kSWarp) c.init_beta();
        __syncthreads();
        c.init_u();
        if (!bar_all<CLUSTER>(S, gen)) return give_up();
        c.chunks(C::kYWarp, ch0);
        if (!bar_all<CLUSTER>(S, gen)) return give_up();
        c.phase_d();
        if (!bar_all<CLUSTER>(S, gen)) return give_up();
        if (c.warp == C::kYWarp) c.init_alpha();
        __syncthreads();
        if (c.warp == C::kYWarp) c.init_yw();
    } else {
        if (c.tid == 0) sc = S->sc[0];
    }
    __syncthreads();
    while (!sc.done) {
        c.phase_a(budget <= 0);
        if (sc.done || budget <= 0) break;
        --budget;
        if (!bar_all<CLUSTER>(S, gen)) return give_up();
        c.phase_b(row0);
        if (!bar_all<CLUSTER>(S, gen)) return give_up();
        c.phase_c(ch0);
        if (!bar_all<CLUSTER>(S, gen)) return give_up();
        c.phase_d();
        if (!bar_all<CLUSTER>(S, gen)) return give_up();
    }
    if (sc.ypend && c.warp == C::kYWarp) c.update_yw();
    __syncthreads();
    if (c.bid == 0 && c.tid == 0) {
        sc.ypend = 0;
        S->sc[0] = sc;
    }
}

// The same phases as kernels of their own: the same grid, work split and sums,
// so the same bits.  Several solves at once (the batched entry point) run these:
// a persistent kernel holds its stream's hardware queue, and the streams behind
// it, for the whole iteration.  Also the profiled runs, which time the products.
// PH 0..2: the start (u; t; v), 3: w and y, 4..7: A..D.
template <bool MIXED, int NT, int PH>
__global__ void __launch_bounds__(NT, 1024 / NT) k_lsqr_phase(const PArgs<MIXED> g)
{
    pdl_wait();
    SKL_CTA(MIXED, NT);
    // slots: no phase writes the one that its own CTAs read.  0 reads 0 and writes 1,
    // 1 and 2 read 1, 3 reads 1 and writes 0; A reads 0 and writes 1, B reads 1, C
    // reads 1 and writes 0, D reads 0
    constexpr int in = (PH == 0 || PH == 4 || PH == 7) ? 0 : 1;
    if (c.tid == 0) sc = g.S->sc[in];
    __syncthreads();
    if (PH >= 4 && sc.done) {
        // A found the end and told slot 1, D and the next A read slot 0; where the
        // start found it (alpha beta = 0), slot 0 knows and B and C read slot 1
        if ((PH == 4 || PH == 6) && c.bid == 0 && c.tid == 0) g.S->sc[PH == 4 ? 1 : 0] = sc;
        return;
    }
    if constexpr (PH == 0) {
        if (c.warp == C::kSWarp) c.init_beta();
        __syncthreads();
        if (c.bid == 0 && c.tid == 0) g.S->sc[1] = sc;
        c.init_u();
    }
    if constexpr (PH == 1) c.chunks(C::kYWarp, c.first_chunk(C::kYWarp));
    if constexpr (PH == 2 || PH == 7) c.phase_d();
    if constexpr (PH == 3) {
        if (c.warp == C::kYWarp) c.init_alpha();
        __syncthreads();
        if (c.warp == C::kYWarp) c.init_yw();
        if (c.bid == 0 && c.tid == 0) g.S->sc[0] = sc;
    }
    if constexpr (PH == 4) {
        c.phase_a(false);
        if (sc.done && sc.ypend && c.warp == C::kYWarp) c.update_yw();
        __syncthreads();
        if (c.bid == 0 && c.tid == 0) g.S->sc[1] = sc;
    }
    if constexpr (PH == 5) c.phase_b(c.first_row());
    if constexpr (PH == 6) {
        c.phase_c(c.first_chunk(C::kYWarp));
        __syncthreads();
        if (c.bid == 0 && c.tid == 0) g.S->sc[0] = sc;
    }
}

// ---- dense problems -------------------------------------------------------------
// The dense products are bound by A: 1.28 GB at 40,000 x 4,000, read once for A z
// and again for A^T u.  A row of u needs the whole row's dot first, but only that
// row: here a CTA holds a few whole rows (a tile) in shared memory, forms their
// u, and adds u times the tile to its share of A^T u, so that an iteration reads A
// once (40,000 x 4,000: 463 us per iteration with the two products as kernels of
// their own at 0.95 of HBM, 360 here; the pass is bound by the float-float
// arithmetic, ~26 FP32 instructions per entry, and by the sums over the CTA between
// two of its barriers).  u and its norm are FP64, formed by one warp between the
// barriers, and A^T u is summed four rows at a time: 340 us with pairs and one chain,
// which left x 25 % further off.  Tried: packed f32x2 arithmetic (487 us: it
// issues at a quarter of the scalar rate), a tile ring read twice from shared
// memory with the sums on a warp of their own (440 us), two CTAs of 256 threads per
// SM (380 us).
//
// Storage (k_split_tiles): rows in pairs, columns in K chunks of CW <= 512 (one
// column per thread); an entry is {hi0, hi1, lo0, lo1} of the pair (one 16-byte
// read), a chunk is one contiguous bulk copy and a tile RB row pairs.  Threads 0..T-1 keep a ring of chunks in flight
// (cp.async.bulk, one mbarrier per slot) across tiles, phases and barriers.
//
// A tile is in registers before its products start, so its slots are refilled at
// once and the copies run beside the arithmetic, the barriers and the other
// phases.  The old u is loaded a tile ahead: it waits ~2 us behind the copies in
// flight.
// Phases per iteration: A (M v), BC (the pass over A), R (the CTAs' shares of
// A^T u added up, in order; beta, y and w beside it), D (M^T t).
constexpr int kDT = 512;
constexpr int kDenseMaxD = 8 * kDT;

struct DArgs {
    const float4* A;          // tiles
    double* uh;               // u
    float2* part;             // [G][K * CW] shares of A^T u
    float2* tn;               // A^T u, natural column order
    int CW, ntiles, nslots;
    int sv_bytes;             // staged-vector bytes before the ring
    long long* prof;          // 4 summed phase times (ns) of CTA 0, or null
};

// acc += a x without renormalising acc (the error terms gather in acc.lo, which a
// few terms leave 2^-22 of acc.hi at most); ff_norm after a handful of terms.
SKL_DEV void ff_fma_lazy(ff& acc, float ah, float al, ff x)
{
    const float p = __fmul_rn(ah, x.hi);
    const float pe = __fmaf_rn(ah, x.hi, -p);
    const float pl = __fmaf_rn(ah, x.lo, __fmaf_rn(al, x.hi, pe));
    float s, e;
    two_sum(acc.hi, p, s, e);
    acc.hi = s;
    acc.lo = __fadd_rn(acc.lo, __fadd_rn(e, pl));
}
// a x, unnormalised
SKL_DEV ff ff_mul_lazy(float ah, float al, ff x)
{
    const float p = __fmul_rn(ah, x.hi);
    return {p, __fmaf_rn(ah, x.lo, __fmaf_rn(al, x.hi, __fmaf_rn(ah, x.hi, -p)))};
}
SKL_DEV void ff_norm(ff& a)
{
    const float h = __fadd_rn(a.hi, a.lo);
    a.lo = __fsub_rn(a.lo, __fsub_rn(h, a.hi));
    a.hi = h;
}

// Sum over the warp of N values per lane (N a power of two): lane l ends with value
// l / (32 / N).  Halving exchanges, then a plain butterfly: fixed order.
template <int N>
SKL_DEV ff warp_sum_n(ff (&v)[N], int lane)
{
    int off = 16;
#pragma unroll
    for (int n = N; n > 1; n >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const ff send = up ? v[i] : v[i + n / 2];
            const ff keep = up ? v[i + n / 2] : v[i];
            v[i] = keep;
            ff_add(v[i], ff_shfl_xor(send, off));
        }
    }
#pragma unroll
    for (int o = 32 / N / 2; o > 0; o >>= 1) ff_add(v[0], ff_shfl_xor(v[0], o));
    return v[0];
}

template <int K, int RB>
__global__ void __launch_bounds__(kDT, 1)
k_lsqr_dense(const PArgs<true> g, const DArgs a, int start, int budget)
{
    pdl_wait();
    SKL_CTA(true, kDT);
    constexpr int T = K * RB;            // chunks of a tile
    constexpr int NV = 2 * RB;           // rows of a tile
    constexpr int kMaxSlots = 64;
    constexpr int kW = kDT / 32;
    __shared__ __align__(8) uint64_t bars[kMaxSlots];
    __shared__ float2 s_part[kW][NV];
    __shared__ __align__(16) float4 s_u[RB];
    __shared__ float2 s_red[C::kYWarp][32];
    PState* S = g.S;
    if (!meet_all(S)) return;
    const int tid = c.tid, lane = c.lane, warp = c.warp;
    const int CW = a.CW, NS = a.nslots;
    const unsigned chunk_bytes = (unsigned)CW * 16;
    unsigned char* ring = smem_raw + a.sv_bytes;
    float2* zs = c.sv;                    // the pass's z, by thread
    const int mine = (a.ntiles - c.bid + c.G - 1) / c.G;   // this CTA's tiles
    const bool col_ok = tid < CW;
    const int col = min(tid, CW - 1);     // a thread past the last column reads it with z = 0
    unsigned gen = 0;
    if (tid < NS) tc::mbar_init(smem_u32(bars + tid), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    // Chunk sequence of this CTA: tile by tile, over and over (A does not change
    // between iterations), round the ring's slots.  All positions advance by
    // T per tile and wrap by a compare.
    const int per_pass = mine * T;
    auto issue = [&](int q, int slot) {
        const unsigned bar = smem_u32(bars + slot);
        tc::mbar_expect_tx(bar, chunk_bytes);
        const float4* src = a.A + ((int64_t)(c.bid + (q / T) * c.G) * T + q % T) * CW;
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_u32(ring) + (unsigned)slot * chunk_bytes),
                     "l"(src), "r"(chunk_bytes), "r"(bar)
                     : "memory");
    };
    auto arrived = [&](int slot, unsigned parity) {
        for (unsigned i = 0; i < tc::kWaitLimit; ++i)
            if (tc::mbar_try(smem_u32(bars + slot), parity)) return true;
        return false;
    };
    int slot0 = 0;                        // slot and parity of the next tile's first chunk
    unsigned par0 = 0;
    int next_q = mine > 0 ? (NS + tid) % per_pass : 0;   // thread t < T: its next chunk to ask for
    if (mine > 0)
        for (int q = tid; q < NS; q += kDT) issue(q % per_pass, q);
    auto slot_of = [&](int q, unsigned& parity) {
        const int sl = slot0 + q;
        parity = sl >= NS ? par0 ^ 1u : par0;
        return sl >= NS ? sl - NS : sl;
    };
    // the copies in flight land before the CTA exits
    auto leave = [&] {
        if (mine > 0 && tid < NS) {
            unsigned parity;
            const int sl = slot_of(tid, parity);
            arrived(sl, parity);
        }
        __syncthreads();
    };
    auto give_up = [&] {
        if (tid == 0) S->timeout = 1;
        leave();
    };
    // the pass over A: u = ia A z - coef u, this CTA's share of A^T u; false on a
    // copy that did not arrive
    auto pass = [&]() -> bool {
        // z of the thread's columns: its own shared-memory entries (registers are
        // short with 64 of them holding the tile)
        ff t[K];
        const bool use_z = (__double_as_longlong(sc.ia) << 1) != 0;   // sc.ia != 0
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int j = k * CW + tid;
            float2 zz = make_float2(0.f, 0.f);
            if (col_ok && j < g.d && use_z) zz = ld_cg(g.z + j);
            zs[k * kDT + tid] = zz;
            t[k] = ff{0.f, 0.f};
        }
        double ss = 0.0;
        // warp 0 finishes the tile's rows: lane l row l % NV, and lanes below NV write u
        const bool fin = tid < NV;
        double un = 0.0;                     // the next tile's old u
        if (fin && c.bid * NV + tid < g.n) un = a.uh[c.bid * NV + tid];
        for (int it = 0; it < mine; ++it) {
            // each warp waits for the tile's chunks with one lane per chunk
            bool ok = true;
            if (lane < T) {
                unsigned parity;
                const int sl = slot_of(lane, parity);
                ok = arrived(sl, parity);
            }
            __syncwarp();
            float4 x[T];
#pragma unroll
            for (int q = 0; q < T; ++q) {
                unsigned parity;
                x[q] = reinterpret_cast<const float4*>(ring + (unsigned)slot_of(q, parity) * chunk_bytes)[col];
            }
            if (__syncthreads_or(!ok)) return false;
            if (tid < T) {
                unsigned parity;
                const int sl = slot_of(tid, parity);
                issue(next_q, sl);
                next_q += T;
                if (next_q >= per_pass) next_q -= per_pass;
            }
            slot0 += T;
            if (slot0 >= NS) {
                slot0 -= NS;
                par0 ^= 1u;
            }
            const int row = (c.bid + it * c.G) * NV + tid;
            const double uc = -sc.coef_n * un;   // off the chain below
            un = 0.0;
            if (fin && it + 1 < mine && row + c.G * NV < g.n) un = a.uh[row + c.G * NV];
            ff v[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) v[q] = ff{0.f, 0.f};
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const float2 zz = zs[k * kDT + tid];
                const ff z{zz.x, zz.y};
#pragma unroll
                for (int rb = 0; rb < RB; ++rb) {
                    ff_fma_lazy(v[2 * rb], x[rb * K + k].x, x[rb * K + k].z, z);
                    ff_fma_lazy(v[2 * rb + 1], x[rb * K + k].y, x[rb * K + k].w, z);
                }
            }
#pragma unroll
            for (int q = 0; q < NV; ++q) ff_norm(v[q]);
            const ff s = warp_sum_n<NV>(v, lane);
            if (lane % (32 / NV) == 0) s_part[warp][lane / (32 / NV)] = make_float2(s.hi, s.lo);
            __syncthreads();
            if (warp == 0) {
                // 32 / NV lanes share a row's warps
                constexpr int kPer = kW * NV / 32;
                ff r[kPer];
#pragma unroll
                for (int w = 0; w < kPer; ++w) {
                    const float2 p = s_part[(lane / NV) * kPer + w][lane % NV];
                    r[w] = ff{p.x, p.y};
                }
#pragma unroll
                for (int h = kPer / 2; h > 0; h >>= 1)
#pragma unroll
                    for (int w = 0; w < h; ++w) ff_add(r[w], r[w + h]);
#pragma unroll
                for (int o = 16; o >= NV; o >>= 1) ff_add(r[0], ff_shfl_xor(r[0], o));
                if (fin) {
                    const double nv = fma((double)r[0].lo, sc.ia, fma((double)r[0].hi, sc.ia, uc));
                    const float2 nf = store_val<true>(nv);
                    float* su = reinterpret_cast<float*>(&s_u[lane >> 1]);
                    su[lane & 1] = nf.x;
                    su[2 + (lane & 1)] = nf.y;
                    if (row < g.n) {
                        a.uh[row] = nv;
                        ss = fma(nv, nv, ss);
                    }
                }
            }
            __syncthreads();
            // A^T u: up to four rows' products first, then one normalised addition to the
            // running sum, whose rounding errors the long chain would gather
            constexpr int GR = RB == 8 ? 1 : 2;
#pragma unroll
            for (int r0 = 0; r0 < RB; r0 += GR) {
                float4 u[GR];
#pragma unroll
                for (int q = 0; q < GR; ++q) u[q] = s_u[r0 + q];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    ff w;
#pragma unroll
                    for (int q = 0; q < GR; ++q) {
                        const float4 xx = x[(r0 + q) * K + k];
                        if (q == 0) w = ff_mul_lazy(xx.x, xx.z, ff{u[q].x, u[q].z});
                        else ff_fma_lazy(w, xx.x, xx.z, ff{u[q].x, u[q].z});
                        ff_fma_lazy(w, xx.y, xx.w, ff{u[q].y, u[q].w});
                    }
                    ff_add(t[k], w);
                }
            }
        }
        if (col_ok)
#pragma unroll
            for (int k = 0; k < K; ++k) a.part[(int64_t)c.bid * K * CW + k * CW + tid] = make_float2(t[k].hi, t[k].lo);
        if (warp == 0) {
            ss = warp_sum(ss);
            if (lane == 0) g.pb[c.bid] = ss;
        }
        return true;
    };
    // t = the shares' sum: this CTA's columns, by the first kYWarp warps
    auto reduce = [&] {
        const int per = (g.d + c.G - 1) / c.G, c0 = c.bid * per, c1 = min(g.d, c0 + per);
        for (int b0 = c0; b0 < c1; b0 += 32) {
            const int col = b0 + lane;
            if (warp < C::kYWarp) {
                // four shares at a time, in pairs: short chains round less
                ff r{0.f, 0.f};
                if (col < c1)
                    for (int q = warp; q < c.G; q += 4 * C::kYWarp) {
                        ff p[4];
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            const int qq = q + h * C::kYWarp;
                            const float2 v = qq < c.G ? ld_cg(a.part + (int64_t)qq * K * CW + col) : make_float2(0.f, 0.f);
                            p[h] = ff{v.x, v.y};
                        }
                        ff_add(p[0], p[1]);
                        ff_add(p[2], p[3]);
                        ff_add(p[0], p[2]);
                        ff_add(r, p[0]);
                    }
                s_red[warp][lane] = make_float2(r.hi, r.lo);
            }
            __syncthreads();
            if (warp == 0 && col < c1) {
                static_assert(C::kYWarp % 2 == 0, "sums in pairs");
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < C::kYWarp; w += 2) {
                    const float2 p = s_red[w][lane], q = s_red[w + 1][lane];
                    ff r{p.x, p.y};
                    ff_add(r, q.x, q.y);
                    s += ff_to_double(r);
                }
                a.tn[col] = store_val<true>(s);
            }
            __syncthreads();
        }
    };
    auto phase_d = [&] {
        for (int i = tid; i < g.r; i += kDT) c.sv[i] = ld_cg(a.tn + __ldg(g.cols + i));
        c.tri_finish();
    };
    long long tp = 0;
    auto lap = [&](int k) {
        if (a.prof && c.bid == 0 && tid == 0) {
            const long long t = now_ns();
            if (k >= 0) a.prof[k] += t - tp;
            tp = t;
        }
    };
    if (start) {
        // u = b through the pass itself: u = 0 - (-1) u
        if (warp == C::kSWarp) c.init_beta();
        __syncthreads();
        for (int i = c.bid * kDT + tid; i < g.n; i += c.G * kDT) a.uh[i] = g.b[i] * sc.bs;
        if (tid == 0) {
            sc.ia = 0.0;
            sc.coef_n = -1.0;
        }
        if (!bar_all<false>(S, gen)) return give_up();
        if (!pass()) return give_up();
        if (!bar_all<false>(S, gen)) return give_up();
        reduce();
        if (!bar_all<false>(S, gen)) return give_up();
        phase_d();
        if (!bar_all<false>(S, gen)) return give_up();
        if (warp == C::kYWarp) c.init_alpha();
        __syncthreads();
        if (warp == C::kYWarp) c.init_yw();
    } else {
        if (tid == 0) sc = S->sc[0];
    }
    __syncthreads();
    while (!sc.done) {
        lap(-1);
        c.phase_a(budget <= 0);
        if (sc.done || budget <= 0) break;
        --budget;
        if (!bar_all<false>(S, gen)) return give_up();
        lap(0);
        if (!pass()) return give_up();
        if (!bar_all<false>(S, gen)) return give_up();
        lap(1);
        const int yp = sc.ypend;
        __syncthreads();   // beta_scalars clears the flag
        if (warp == C::kSWarp) c.beta_scalars();
        else if (warp == C::kYWarp && yp) c.update_yw();
        reduce();
        if (!bar_all<false>(S, gen)) return give_up();
        lap(2);
        phase_d();
        if (!bar_all<false>(S, gen)) return give_up();
        lap(3);
    }
    if (sc.ypend && warp == C::kYWarp) c.update_yw();
    __syncthreads();
    if (c.bid == 0 && tid == 0) {
        sc.ypend = 0;
        S->sc[0] = sc;
    }
    leave();
}

// A (FP64, column-major) to the tile storage, with the range check of the mixed
// path and ||A||_F^2 partials.  FP64 arithmetic on every element would hold the
// FP64 pipe for ~2 ms at 40,000 x 4,000: hi and lo are cut from the bits, and the
// squares are summed in float pairs, in three sums, so that none of the admitted
// values' squares leaves the float range.
constexpr int kSplitRows = 64, kSplitCols = 32;

// hi = x rounded to 24 bits, lo = the rest rounded to 24: as ff_from_double for
// magnitudes in [2^-100, 2^100] and 0, except that ties round away
SKL_DEV ff ff_from_bits(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned hiw = (unsigned)(b >> 32);
    const int e = (int)((hiw >> 20) & 0x7ff) - 1023;
    if (e < -101 || e > 100) return ff_from_double(x);
    const unsigned sign = hiw & 0x80000000u;
    const unsigned low = (unsigned)b & 0x1fffffffu;                       // the 29 bits below FP32
    const unsigned top = ((hiw & 0xfffffu) << 3) | ((unsigned)b >> 29);   // 23 bits
    const unsigned up = low >> 28;
    const float h = __uint_as_float(sign | (((unsigned)(e + 127) << 23) + top + up));
    const int rest = (int)low - (int)(up << 29);                          // in units of 2^(e - 52)
    const float l = (float)rest * __uint_as_float(sign | ((unsigned)(e - 52 + 127 + 30) << 23)) * 0x1p-30f;
    return ff{h, l};
}

__global__ void __launch_bounds__(256)
k_split_tiles(const double* __restrict__ A, int64_t lda, int n, int d, int K, int CW, int64_t blocks,
              float4* __restrict__ out, double* __restrict__ fro, unsigned* __restrict__ status)
{
    pdl_wait();
    __shared__ float2 tile[kSplitCols][kSplitRows + 1];
    __shared__ ff red[8];
    ff ss{0.f, 0.f}, big{0.f, 0.f}, small{0.f, 0.f};   // of x, of x 2^-60, of x 2^60
    bool bad = false;
    const int64_t rtiles = (blocks * 2 + kSplitRows - 1) / kSplitRows;
    const int ctiles = (K * CW + kSplitCols - 1) / kSplitCols;
    for (int64_t w = blockIdx.x; w < rtiles * ctiles; w += gridDim.x) {
        const int64_t r0 = (w % rtiles) * kSplitRows;
        const int c0 = (int)(w / rtiles) * kSplitCols;
        double x[kSplitRows * kSplitCols / 256];
#pragma unroll
        for (int q = 0; q < kSplitRows * kSplitCols / 256; ++q) {
            const int e = threadIdx.x + q * 256, i = e % kSplitRows, j = e / kSplitRows;
            x[q] = (r0 + i < n && c0 + j < d) ? A[(r0 + i) + (int64_t)(c0 + j) * lda] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < kSplitRows * kSplitCols / 256; ++q) {
            const int e = threadIdx.x + q * 256, i = e % kSplitRows, j = e / kSplitRows;
            const unsigned long long m = (unsigned long long)__double_as_longlong(x[q]) & 0x7fffffffffffffffull;
            // |x| > 2^100 or 0 < |x| < 2^-100 (a NaN is neither)
            bad |= (m > 0x4630000000000000ull && m <= 0x7ff0000000000000ull) || (m != 0 && m < 0x39b0000000000000ull);
            const ff f = ff_from_bits(x[q]);
            const float mag = fabsf(f.hi);
            if (mag <= 0x1p40f && mag >= 0x1p-40f) {
                ff_fma(ss, f, f);
            } else if (mag > 1.f) {
                const ff g{f.hi * 0x1p-60f, f.lo * 0x1p-60f};
                ff_fma(big, g, g);
            } else if (mag > 0.f) {
                const ff g{f.hi * 0x1p60f, f.lo * 0x1p60f};
                ff_fma(small, g, g);
            }
            tile[j][i] = make_float2(f.hi, f.lo);
        }
        __syncthreads();
        for (int e = threadIdx.x; e < kSplitRows / 2 * kSplitCols; e += 256) {
            const int j = e % kSplitCols, p = e / kSplitCols;   // row pair p
            const int col = c0 + j;
            const int64_t blk = r0 / 2 + p;
            if (col < K * CW && blk < blocks) {
                const float2 e = tile[j][2 * p], o = tile[j][2 * p + 1];
                out[(blk * K + col / CW) * CW + col % CW] = make_float4(e.x, o.x, e.y, o.y);
            }
        }
        __syncthreads();
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(status, kStatusRange);
    const double t = ff_to_double(block_sum_ff(ss, red)) + ff_to_double(block_sum_ff(big, red)) * 0x1p120 +
                     ff_to_double(block_sum_ff(small, red)) * 0x1p-120;
    if (threadIdx.x == 0) fro[blockIdx.x] = t;
}

// ---- start and end -------------------------------------------------------------
// kNormParts partial sums of ||b||^2, FP64 as b is: squares of pairs leave the
// float range where ||b|| is below 1e-19 or above 1e19.  3 us of a solve.
__global__ void __launch_bounds__(256) k_lsqr_norm(const double* __restrict__ b, int64_t n, double* __restrict__ part)
{
    pdl_wait();
    __shared__ double red[8];
    double s = 0.0;
    for (int64_t i = blockIdx.x * 256 + threadIdx.x; i < n; i += kNormParts * 256) s = fma(b[i], b[i], s);
    s = block_sum(s, red);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// y for the caller: the scale of b taken out
__global__ void k_lsqr_y(const double* __restrict__ y, int r, const PState* __restrict__ S, double* __restrict__ out)
{
    pdl_wait();
    const double inv = 1.0 / S->sc[0].bs;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r; i += gridDim.x * blockDim.x) out[i] = y[i] * inv;
}

void norm_launch(const double* b, int64_t n, double* part, cudaStream_t st)
{
    launch_k(k_lsqr_norm, kNormParts, 256, 0, st, b, n, part);
    SKL_LAUNCHED();
}
void y_launch(const double* y, int64_t r, const PState* S, double* out, cudaStream_t st)
{
    launch_k(k_lsqr_y, (unsigned)std::min<int64_t>((r + 255) / 256, 152), 256, 0, st, y, (int)r, S, out);
    SKL_LAUNCHED();
}

// ---- column chunks -------------------------------------------------------------
__global__ void k_chunk_count(const int* __restrict__ cp, const int* __restrict__ cols, int r, int len,
                              int* __restrict__ cnt)
{
    pdl_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r; i += gridDim.x * blockDim.x) {
        const int c = cols[i];
        cnt[i] = max(1, (cp[c + 1] - cp[c] + len - 1) / len);   // an empty column is a chunk too
    }
}

__global__ void k_chunk_fill(const int* __restrict__ cp, const int* __restrict__ cols, int r, int len,
                             const int* __restrict__ coff, int4* __restrict__ chunks, unsigned* __restrict__ ccnt)
{
    pdl_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r; i += gridDim.x * blockDim.x) {
        const int c = cols[i], p1 = cp[c + 1], q0 = coff[i], nq = coff[i + 1] - q0;
        int p = cp[c];
        for (int q = 0; q < nq; ++q, p += len) chunks[q0 + q] = make_int4(p, min(p1, p + len), i, nq);
        ccnt[i] = 0;
    }
}

int sm_count_p()
{
    static const int v = [] {
        int dev = 0, s = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&s, cudaDevAttrMultiProcessorCount, dev);
        return s > 0 ? s : 148;
    }();
    return v;
}

// lanes per row: each lane handles about four nonzeros
int lanes_row(double avg) { return avg >= 96 ? 32 : avg >= 40 ? 16 : avg >= 16 ? 8 : 4; }
// lanes per column: about eight per step
int lanes_col(double avg) { return avg >= 128 ? 32 : avg >= 64 ? 16 : avg >= 24 ? 8 : 4; }

struct PBufs {
    PState* S;
    void *us, *vs, *z, *t, *tpart;
    double *vh, *w, *y, *pa, *pb, *bpart;
    int4* chunks; int* coff; int* scan; int* cnt; unsigned* ccnt;
    size_t bytes;
};

int64_t max_chunks(const LsqrProblem& P, int len) { return P.r + P.nnz / len + 1; }

PBufs pcarve(const LsqrProblem& P, void* work)
{
    PBufs B;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        void* p = (char*)work + off;
        off += (bytes + 255) & ~(size_t)255;
        return p;
    };
    const size_t vs = P.precision == SKL_PREC_MIXED ? sizeof(float2) : sizeof(double);
    const int64_t nch = max_chunks(P, 4 * kTU * kChunkSteps);   // the shortest chunks
    B.S = (PState*)take(sizeof(PState));
    B.us = take(P.n * vs);
    B.vs = take(P.r * vs);
    B.z = take(P.d * vs);
    B.t = take(P.r * vs);
    B.tpart = take(nch * vs);
    B.vh = P.precision == SKL_PREC_MIXED ? (double*)take(P.r * sizeof(double)) : (double*)B.vs;
    B.w = (double*)take(P.r * sizeof(double));
    B.y = (double*)take(P.r * sizeof(double));
    B.pa = (double*)take(1024 * sizeof(double));
    B.pb = (double*)take(1024 * sizeof(double));
    B.bpart = (double*)take(kNormParts * sizeof(double));
    B.chunks = (int4*)take(nch * sizeof(int4));
    B.ccnt = (unsigned*)take(P.r * sizeof(unsigned));
    B.coff = (int*)take((P.r + 1) * sizeof(int));
    B.cnt = (int*)take(P.r * sizeof(int));
    B.scan = (int*)take(scan_scratch_ints(P.r) * sizeof(int));
    B.bytes = off;
    return B;
}

// Bytes one iteration reads: both copies of A and both triangles.
double iter_bytes(const LsqrProblem& P)
{
    const double vb = P.precision == SKL_PREC_MIXED ? 4.0 : 8.0;
    return 24.0 * (double)P.nnz + 16.0 * (double)P.n + vb * (double)P.r * (double)P.r;
}

size_t vec_smem(const LsqrProblem& P)
{
    const size_t vs = P.precision == SKL_PREC_MIXED ? sizeof(float2) : sizeof(double);
    return (size_t)((std::max(P.r, P.d) + 4) & ~(int64_t)3) * vs;
}

// CTAs: one per ~100 KB an iteration reads (a barrier costs more with more of
// them, a CTA streams ~50 KB per us), at least one cluster, at most one per SM;
// with more than ~400 KB per SM the loads in flight matter and the CTAs get 1,024
// threads (120,000 x 5,000: 136 -> 107 us per iteration; 31,013 x 1,507, 130 KB
// per SM: 28 us with 512, 31 with 1,024).
struct Grid {
    int ctas, threads;
};
Grid grid_of(const LsqrProblem& P)
{
    const double bytes = iter_bytes(P);
    return {(int)std::max<double>(kCluster, std::min<double>(sm_count_p(), std::ceil(bytes / 100e3))),
            bytes / sm_count_p() > 400e3 ? kBigCta : kSmallCta};
}

template <bool MIXED, int NT, int PH>
void launch_phase(const PArgs<MIXED>& g, int G, size_t smem, cudaStream_t st)
{
    if (smem > 32 * 1024) allow_max_dynamic_smem((const void*)k_lsqr_phase<MIXED, NT, PH>);
    launch_k(k_lsqr_phase<MIXED, NT, PH>, (unsigned)G, NT, smem, st, g);
    SKL_LAUNCHED();
}

double time_limit_s()
{
    static const double v = [] {
        const char* e = getenv("SKILLS_LSQR_TIMEOUT_S");
        return e ? atof(e) : 60.0;
    }();
    return v;
}

struct Clock {
    std::chrono::steady_clock::time_point t0 = std::chrono::steady_clock::now();
    void check() const
    {
        if (std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() > time_limit_s())
            fail(SKL_ERR_TIMEOUT, "LSQR exceeded its time limit (SKILLS_LSQR_TIMEOUT_S)");
    }
};

// Phase kernels: a graph of kIterPerGraph iterations, replayed until the state
// says done; the next replay is queued before the last one's state is read, so
// the GPU does not wait for the host.  start: from b, else from slot 0's state.
// profile: events around the products.
template <bool MIXED, int NT>
const PState* run_phases(const PArgs<MIXED>& g, int G, size_t smem, void* host_pinned, cudaStream_t st,
                         cudaStream_t cap, bool start, int profile, LsqrResult& res)
{
    if (start) {
        launch_phase<MIXED, NT, 0>(g, G, smem, st);
        launch_phase<MIXED, NT, 1>(g, G, smem, st);
        launch_phase<MIXED, NT, 2>(g, G, smem, st);
        launch_phase<MIXED, NT, 3>(g, G, smem, st);
    }
    struct Owned {
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        cudaEvent_t ev[2] = {nullptr, nullptr};
        std::vector<cudaEvent_t> pev;
        ~Owned()
        {
            for (cudaEvent_t e : ev)
                if (e) cudaEventDestroy(e);
            for (cudaEvent_t e : pev)
                if (e) cudaEventDestroy(e);
            if (exec) cudaGraphExecDestroy(exec);
            if (graph) cudaGraphDestroy(graph);
        }
    } o;
    for (auto& e : o.ev) SKL_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    o.pev.assign(profile ? 8 * kIterPerGraph : 0, nullptr);
    for (auto& e : o.pev) SKL_CUDA(cudaEventCreate(&e));
    // capture on the library's stream (the caller's may be the legacy default
    // stream, which cannot be captured); replay on the caller's
    SKL_CUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
    for (int q = 0; q < kIterPerGraph; ++q) {
        auto mark = [&](int k) {
            if (profile) SKL_CUDA(cudaEventRecordWithFlags(o.pev[8 * q + k], cap, cudaEventRecordExternal));
        };
        mark(4);
        launch_phase<MIXED, NT, 4>(g, G, smem, cap);
        mark(5);
        mark(0);
        launch_phase<MIXED, NT, 5>(g, G, smem, cap);
        mark(1);
        mark(2);
        launch_phase<MIXED, NT, 6>(g, G, smem, cap);
        mark(3);
        mark(6);
        launch_phase<MIXED, NT, 7>(g, G, smem, cap);
        mark(7);
    }
    SKL_CUDA(cudaStreamEndCapture(cap, &o.graph));
    SKL_CUDA(cudaGraphInstantiate(&o.exec, o.graph, 0));
    const Clock clock;
    long long it_prev = 0;
    auto replay = [&](int k) {
        SKL_CUDA(cudaGraphLaunch(o.exec, st));
        for (int q = 0; q < 4 * kIterPerGraph; ++q) SKL_LAUNCHED();
        SKL_CUDA(cudaMemcpyAsync((char*)host_pinned + k * 1024, g.S, sizeof(PState), cudaMemcpyDeviceToHost, st));
        SKL_CUDA(cudaEventRecord(o.ev[k], st));
    };
    static_assert(sizeof(PState) <= 1024, "two states in the pinned scratch");
    if (!profile) replay(0);
    for (int k = 0;; k ^= 1) {
        // a profiled replay is read before the next one overwrites its events
        replay(profile ? k : k ^ 1);
        SKL_CUDA(cudaEventSynchronize(o.ev[k]));
        const PState* hs = (const PState*)((char*)host_pinned + k * 1024);
        if (profile) {
            const long long ran = hs->sc[0].it + hs->sc[0].pend - it_prev;
            it_prev += ran;
            for (long long q = 0; q < ran && q < kIterPerGraph; ++q)
                for (int kk = 0; kk < 4; ++kk) {
                    float ms = 0.f;
                    SKL_CUDA(cudaEventElapsedTime(&ms, o.pev[8 * q + 2 * kk], o.pev[8 * q + 2 * kk + 1]));
                    res.prof_ms[kk] += ms;
                    res.prof_launches[kk] += 1;
                }
        }
        if (hs->sc[0].done) {
            // the replay still queued returns at once, but it uses the graph
            if (!profile) SKL_CUDA(cudaEventSynchronize(o.ev[k ^ 1]));
            return hs;
        }
        clock.check();
    }
}

// The launches of a persistent kernel fn(args, more, start, budget) until the
// state says done, or one is called off (meet_all): false, with the state of the
// launches before it.
bool run_resident(const void* fn, bool cluster, int G, int threads, size_t smem, PState* S, void* host_pinned,
                  cudaStream_t st, void* arg0, void* arg1)
{
    if (cluster) SKL_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)G);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    if (cluster) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kCluster;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
    }
    const PState* hs = (const PState*)host_pinned;
    const Clock clock;
    for (int start = 1;; start = 0) {
        int budget = kItersPerLaunch;
        void* with1[] = {arg0, arg1, (void*)&start, (void*)&budget};
        void* without[] = {arg0, (void*)&start, (void*)&budget};
        SKL_CUDA(cudaLaunchKernelExC(&cfg, fn, arg1 ? with1 : without));
        SKL_LAUNCHED();
        SKL_CUDA(cudaMemcpyAsync(host_pinned, S, sizeof(PState), cudaMemcpyDeviceToHost, st));
        SKL_CUDA(cudaStreamSynchronize(st));
        if (hs->timeout) fail(SKL_ERR_TIMEOUT, "a bounded wait gave up (LSQR's grid barrier or its copies)");
        if (hs->meet & kMeetOff) return false;
        if (hs->sc[0].done) return true;
        clock.check();
        static_assert(offsetof(PState, meet) == offsetof(PState, bar) + sizeof(unsigned), "reset together");
        SKL_CUDA(cudaMemsetAsync(&S->bar, 0, 2 * sizeof(unsigned), st));
    }
}

// The phase kernels loaded before a persistent launch can be called off: loading one
// (CUDA does so at its first use) may itself wait for the kernel that holds the SM.
template <bool MIXED, int NT, int... PH>
void load_phases(std::integer_sequence<int, PH...>)
{
    cudaFuncAttributes fa;
    (SKL_CUDA(cudaFuncGetAttributes(&fa, k_lsqr_phase<MIXED, NT, PH>)), ...);
}

template <bool MIXED, int NT>
bool run_persistent(const PArgs<MIXED>& g, int G, size_t smem, void* host_pinned, cudaStream_t st)
{
    const void* fn = G <= kCluster ? (const void*)k_lsqr_persist<MIXED, NT, true>
                                   : (const void*)k_lsqr_persist<MIXED, NT, false>;
    allow_max_dynamic_smem(fn);
    if (G > kCluster) {
        static std::once_flag once;
        std::call_once(once, [] { load_phases<MIXED, NT>(std::make_integer_sequence<int, 8>{}); });
    }
    PArgs<MIXED> a = g;
    return run_resident(fn, G <= kCluster, G, NT, smem, g.S, host_pinned, st, (void*)&a, nullptr);
}

// The kernels' arguments, and the column chunks that they name.
template <bool MIXED, int NT>
PArgs<MIXED> persist_args(const LsqrProblem& P, const PBufs& B, const double* b, cudaStream_t st)
{
    using V = ValT<MIXED>;
    using MT = MatT<MIXED>;
    PArgs<MIXED> g{};
    g.n = (int)P.n;
    g.r = (int)P.r;
    g.d = (int)P.d;
    g.L_n = P.lanes_n ? P.lanes_n : lanes_row(P.n ? (double)P.nnz / P.n : 0.0);
    g.L_t = P.lanes_t ? P.lanes_t : lanes_col(P.d ? (double)P.nnz / P.d : 0.0);
    g.rp = P.rp;
    g.ci = P.ci;
    g.cv = (const V*)P.cx;
    g.cp = P.cp;
    g.ri = P.ri;
    g.rv = (const V*)P.rx;
    g.cols = P.cols;
    g.opscale = P.opscale;
    g.chunks = B.chunks;
    g.coff = B.coff;
    g.ccnt = B.ccnt;
    g.Mr = (const MT*)P.Mrow;
    g.Mc = (const MT*)P.M;
    g.ldm = P.ldm;
    g.b = b;
    g.us = (V*)B.us;
    g.vs = (V*)B.vs;
    g.z = (V*)B.z;
    g.t = (V*)B.t;
    g.tpart = (V*)B.tpart;
    g.vh = B.vh;
    g.w = B.w;
    g.y = B.y;
    g.pa = B.pa;
    g.pb = B.pb;
    g.bpart = B.bpart;
    g.S = B.S;
    const int G = grid_of(P).ctas;
    // segments per row of the triangle: one round of the 15 (31) warps where the
    // CTA has fewer rows than that, else about four per warp, which evens out
    // the rows' lengths
    const int nloc = (int)((P.r + G - 1) / G), nw = NT / 32 - 1;
    g.S_seg = std::max(1, std::min(8, nloc <= nw ? nw / nloc : 4 * nw / nloc));
    // chunks of the columns
    const int len = g.L_t * kTU * kChunkSteps;
    const unsigned gr = (unsigned)std::max<int64_t>(1, std::min<int64_t>((P.r + 255) / 256, 152));
    launch_k(k_chunk_count, gr, 256, 0, st, P.cp, P.cols, (int)P.r, len, B.cnt);
    SKL_LAUNCHED();
    scan_exclusive(B.cnt, P.r, B.coff, B.scan, st);
    launch_k(k_chunk_fill, gr, 256, 0, st, P.cp, P.cols, (int)P.r, len, B.coff, B.chunks, B.ccnt);
    SKL_LAUNCHED();
    SKL_CUDA(cudaMemsetAsync(B.z, 0, P.d * sizeof(V), st));
    return g;
}

template <bool MIXED, int NT>
LsqrResult persist_impl(const LsqrProblem& P, const double* b, double tol, int64_t max_it, double* y_out, void* work,
                        void* host_pinned, cudaStream_t st, int profile, cudaStream_t capture_stream)
{
    PBufs B = pcarve(P, work);
    const PArgs<MIXED> g = persist_args<MIXED, NT>(P, B, b, st);
    const int G = grid_of(P).ctas;
    PState init{};
    init.tol = tol;
    init.max_it = max_it;
    SKL_CUDA(cudaMemcpyAsync(B.S, &init, sizeof(PState), cudaMemcpyHostToDevice, st));
    norm_launch(b, P.n, B.bpart, st);
    trace_phase(st, "lsqr: init");
    const size_t smem = vec_smem(P);
    LsqrResult res;
    const PState* hs = (const PState*)host_pinned;
    const bool phases = profile || P.shared_gpu;
    if (phases || !run_persistent<MIXED, NT>(g, G, smem, host_pinned, st)) {
        // the state is the start's unless a launch before the one called off ended
        const bool start = phases || hs->sc[0].it == 0;
        hs = run_phases<MIXED, NT>(g, G, smem, host_pinned, st, capture_stream ? capture_stream : st, start, profile, res);
    }
    trace_phase(st, "lsqr: done");
    res.flag = hs->sc[0].flag;
    res.it = hs->sc[0].it;
    y_launch(B.y, P.r, B.S, y_out, st);
    return res;
}

// Lanes per row and column by time: phases B and C at each choice, median of three
// after a warm-up.  The persistent kernel runs the same phases on the same grid.
template <bool MIXED, int NT>
void persist_tune(LsqrProblem& P, void* work, cudaStream_t st)
{
    const PBufs B = pcarve(P, work);
    struct Events {
        cudaEvent_t e[2] = {nullptr, nullptr};
        ~Events()
        {
            for (cudaEvent_t v : e)
                if (v) cudaEventDestroy(v);
        }
    } ev;
    for (auto& e : ev.e) SKL_CUDA(cudaEventCreate(&e));
    PState init{};
    for (PScal& sc : init.sc) sc.alpha = sc.beta = sc.rhobar = sc.phibar = sc.ia = sc.ib = sc.bs = 1.0;
    SKL_CUDA(cudaMemcpyAsync(B.S, &init, sizeof(PState), cudaMemcpyHostToDevice, st));
    SKL_CUDA(cudaMemsetAsync(B.us, 0, P.n * sizeof(ValT<MIXED>), st));
    const int G = grid_of(P).ctas;
    const size_t smem = vec_smem(P);
    auto time_of = [&](auto&& launch) {
        launch();
        float t[3];
        for (float& v : t) {
            SKL_CUDA(cudaEventRecord(ev.e[0], st));
            launch();
            SKL_CUDA(cudaEventRecord(ev.e[1], st));
            SKL_CUDA(cudaEventSynchronize(ev.e[1]));
            SKL_CUDA(cudaEventElapsedTime(&v, ev.e[0], ev.e[1]));
        }
        std::sort(t, t + 3);
        return t[1];
    };
    float best_n = 1e30f, best_t = 1e30f;
    int ln = 0, lt = 0;
    for (int L : {4, 8, 16, 32}) {
        P.lanes_n = P.lanes_t = L;
        const PArgs<MIXED> g = persist_args<MIXED, NT>(P, B, nullptr, st);
        const float tn = time_of([&] { launch_phase<MIXED, NT, 5>(g, G, smem, st); });
        if (tn < best_n) best_n = tn, ln = L;
        const float tt = time_of([&] { launch_phase<MIXED, NT, 6>(g, G, smem, st); });
        if (tt < best_t) best_t = tt, lt = L;
    }
    P.lanes_n = ln;
    P.lanes_t = lt;
}

// ---- dense host side -------------------------------------------------------------
// Row pairs of a tile: at most 16 entries per thread (64 registers).
constexpr int tile_rb(int K) { return K == 1 ? 8 : K <= 4 ? 4 : 2; }

struct DenseShape {
    int K, CW, RB, ntiles;
    int64_t blocks;
    size_t bytes() const { return (size_t)blocks * K * CW * 16; }
};
DenseShape dense_shape(int64_t n, int64_t d)
{
    DenseShape s;
    s.K = (int)((d + kDT - 1) / kDT);
    s.CW = (int)((d + s.K - 1) / s.K);
    s.RB = tile_rb(s.K);
    s.ntiles = (int)((n + 2 * s.RB - 1) / (2 * s.RB));
    s.blocks = (int64_t)s.ntiles * s.RB;
    return s;
}

// One CTA per tile, at most one per SM: a tile takes ~3.5 us whatever its columns, more
// than the grid barrier gains from fewer CTAs (one per 100 KB, 9 for 1,588 x 71: 3.3 ms
// per solve against 1.7; 5,003 x 301 the same 2.5 ms with 120 CTAs as with 152).
int dense_ctas(const LsqrProblem& P)
{
    return std::max(1, std::min(sm_count_p(), dense_shape(P.n, P.d).ntiles));
}

struct DBufs {
    PState* S;
    float2 *vs, *z, *part, *tn;
    double *uh, *vh, *w, *y, *pa, *pb, *bpart;
    long long* prof;
    size_t bytes;
};
DBufs dcarve(const LsqrProblem& P, void* work)
{
    DBufs B;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        void* p = (char*)work + off;
        off += (bytes + 255) & ~(size_t)255;
        return p;
    };
    const DenseShape s = dense_shape(P.n, P.d);
    B.S = (PState*)take(sizeof(PState));
    B.uh = (double*)take(P.n * sizeof(double));
    B.vh = (double*)take(P.r * sizeof(double));
    B.vs = (float2*)take(P.r * sizeof(float2));
    B.z = (float2*)take(P.d * sizeof(float2));
    B.part = (float2*)take((size_t)sm_count_p() * s.K * s.CW * sizeof(float2));
    B.tn = (float2*)take(P.d * sizeof(float2));
    B.pa = (double*)take(1024 * sizeof(double));
    B.pb = (double*)take(1024 * sizeof(double));
    B.w = (double*)take(P.r * sizeof(double));
    B.y = (double*)take(P.r * sizeof(double));
    B.bpart = (double*)take(kNormParts * sizeof(double));
    B.prof = (long long*)take(4 * sizeof(long long));
    B.bytes = off;
    return B;
}

const void* dense_kernel(int K)
{
    static const void* const f[8] = {
        (const void*)k_lsqr_dense<1, tile_rb(1)>, (const void*)k_lsqr_dense<2, tile_rb(2)>,
        (const void*)k_lsqr_dense<3, tile_rb(3)>, (const void*)k_lsqr_dense<4, tile_rb(4)>,
        (const void*)k_lsqr_dense<5, tile_rb(5)>, (const void*)k_lsqr_dense<6, tile_rb(6)>,
        (const void*)k_lsqr_dense<7, tile_rb(7)>, (const void*)k_lsqr_dense<8, tile_rb(8)>};
    return f[K - 1];
}

LsqrResult dense_impl(const LsqrProblem& P, const double* b, double tol, int64_t max_it, double* y_out, void* work,
                      void* host_pinned, cudaStream_t st, int profile)
{
    const DenseShape s = dense_shape(P.n, P.d);
    DBufs B = dcarve(P, work);
    PArgs<true> g{};
    g.n = (int)P.n;
    g.r = (int)P.r;
    g.d = (int)P.d;
    g.cols = P.cols;
    g.Mr = (const float*)P.Mrow;
    g.Mc = (const float*)P.M;
    g.ldm = P.ldm;
    g.b = b;
    g.vs = B.vs;
    g.vh = B.vh;
    g.z = B.z;
    g.w = B.w;
    g.y = B.y;
    g.pa = B.pa;
    g.pb = B.pb;
    g.bpart = B.bpart;
    g.S = B.S;
    const int G = dense_ctas(P);
    const int nloc = (int)((P.r + G - 1) / G), nw = kDT / 32 - 1;
    g.S_seg = std::max(1, std::min(8, nloc <= nw ? nw / nloc : 4 * nw / nloc));
    DArgs a{};
    a.A = (const float4*)P.At;
    a.uh = B.uh;
    a.part = B.part;
    a.tn = B.tn;
    a.CW = s.CW;
    a.ntiles = s.ntiles;
    a.sv_bytes = (int)((std::max(vec_smem(P), (size_t)s.K * kDT * sizeof(float2)) + 127) & ~(size_t)127);
    const void* fn = dense_kernel(s.K);
    static std::once_flag once;
    std::call_once(once, [] { lsqr_load_dense_kernels(); });   // as load_phases
    allow_max_dynamic_smem(fn);
    cudaFuncAttributes fa;
    SKL_CUDA(cudaFuncGetAttributes(&fa, fn));
    const int room = fa.maxDynamicSharedSizeBytes - a.sv_bytes;
    a.nslots = std::min(64, room / (s.CW * 16));
    if (a.nslots < s.K * s.RB) fail(SKL_ERR_INVALID, "dense LSQR: the tile ring does not fit");
    a.prof = profile ? B.prof : nullptr;
    SKL_CUDA(cudaMemsetAsync(B.z, 0, P.d * sizeof(float2), st));
    if (profile) SKL_CUDA(cudaMemsetAsync(B.prof, 0, 4 * sizeof(long long), st));
    PState init{};
    init.tol = tol;
    init.max_it = max_it;
    SKL_CUDA(cudaMemcpyAsync(B.S, &init, sizeof(PState), cudaMemcpyHostToDevice, st));
    norm_launch(b, P.n, B.bpart, st);
    trace_phase(st, "lsqr: init");
    LsqrResult res;
    if (!run_resident(fn, false, G, kDT, (size_t)a.sv_bytes + (size_t)a.nslots * s.CW * 16, B.S, host_pinned, st,
                      (void*)&g, (void*)&a)) {
        res.called_off = true;
        return res;
    }
    const PState* hs = (const PState*)host_pinned;
    trace_phase(st, "lsqr: done");
    res.flag = hs->sc[0].flag;
    res.it = hs->sc[0].it;
    if (profile) {
        // M v, the pass over A (both products), M^T t with the shares' sum
        long long ns[4];
        SKL_CUDA(cudaMemcpyAsync(host_pinned, B.prof, sizeof ns, cudaMemcpyDeviceToHost, st));
        SKL_CUDA(cudaStreamSynchronize(st));
        std::memcpy(ns, host_pinned, sizeof ns);
        const double ms[4] = {ns[1] * 1e-6, 0.0, ns[0] * 1e-6, (ns[2] + ns[3]) * 1e-6};
        for (int q = 0; q < 4; ++q) {
            res.prof_ms[q] = ms[q];
            res.prof_launches[q] = q == 1 ? 0 : res.it;
        }
    }
    y_launch(B.y, P.r, B.S, y_out, st);
    return res;
}

}  // namespace

// SKILLS_LSQR_PERSIST=0: the kernels of k_lsqr.cu for every problem, none of which
// waits for the whole GPU.
static bool persist_enabled()
{
    static const bool v = [] {
        const char* e = getenv("SKILLS_LSQR_PERSIST");
        return !(e && e[0] == '0');
    }();
    return v;
}

bool lsqr_dense_tiled(int64_t d, int precision)
{
    return persist_enabled() && precision == SKL_PREC_MIXED && d >= 1 && d <= kDenseMaxD;
}
size_t lsqr_dense_tile_bytes(int64_t n, int64_t d) { return dense_shape(n, d).bytes(); }

void split_dense_tiles(const double* A, int64_t lda, int64_t n, int64_t d, void* out, double* fro, unsigned* status,
                       cudaStream_t st)
{
    const DenseShape s = dense_shape(n, d);
    launch_k(k_split_tiles, kFroParts, 256, 0, st, A, lda, (int)n, (int)d, s.K, s.CW, s.blocks, (float4*)out, fro,
             status);
    SKL_LAUNCHED();
}

bool lsqr_persist_fits(const LsqrProblem& P)
{
    if (P.At) return true;
    if (!persist_enabled()) return false;
    const int G = grid_of(P).ctas;
    return !P.Ad && P.r > 0 && (P.r + G - 1) / G <= kMaxUnits && vec_smem(P) <= 200 * 1024;
}

size_t lsqr_persist_workspace_bytes(const LsqrProblem& P)
{
    return P.At ? dcarve(P, nullptr).bytes : pcarve(P, nullptr).bytes;
}

LsqrResult lsqr_persist_run(const LsqrProblem& P, const double* b, double tol, int64_t max_it, double* y, void* work,
                            void* host_pinned, cudaStream_t st, int profile, cudaStream_t capture_stream)
{
    if (P.At) return dense_impl(P, b, tol, max_it, y, work, host_pinned, st, profile);
    const bool big = grid_of(P).threads == kBigCta;
    auto* fn = P.precision == SKL_PREC_MIXED
                   ? (big ? persist_impl<true, kBigCta> : persist_impl<true, kSmallCta>)
                   : (big ? persist_impl<false, kBigCta> : persist_impl<false, kSmallCta>);
    return fn(P, b, tol, max_it, y, work, host_pinned, st, profile, capture_stream);
}

void lsqr_persist_tune(LsqrProblem& P, void* work, cudaStream_t st)
{
    const bool big = grid_of(P).threads == kBigCta;
    auto* fn = P.precision == SKL_PREC_MIXED ? (big ? persist_tune<true, kBigCta> : persist_tune<true, kSmallCta>)
                                             : (big ? persist_tune<false, kBigCta> : persist_tune<false, kSmallCta>);
    fn(P, work, st);
}

}  // namespace skl
