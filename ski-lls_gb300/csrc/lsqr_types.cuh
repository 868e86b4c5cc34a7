// lsqr_types.cuh -- storage and accumulation types of LSQR's products: float
// pairs with float-float accumulators on the mixed path, FP64 otherwise.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace skl {

template <bool MIXED>
struct VecT {
    using type = double;
};
template <>
struct VecT<true> {
    using type = float2;
};

template <bool MIXED>
SKL_DEV typename VecT<MIXED>::type store_val(double x)
{
    if constexpr (MIXED) {
        ff f = ff_from_double(x);
        return make_float2(f.hi, f.lo);
    } else {
        return x;
    }
}

template <bool MIXED>
struct Acc {
    ff a{0.f, 0.f};
    SKL_DEV void fma_mv(float2 m, float2 x) { ff_fma(a, ff{m.x, m.y}, ff{x.x, x.y}); }
    SKL_DEV void fma_f(float m, float2 x) { ff_fma_f(a, m, ff{x.x, x.y}); }
    SKL_DEV void add(const Acc& o) { ff_add(a, o.a); }
    SKL_DEV Acc shfl_xor(int o) const { Acc r; r.a = ff_shfl_xor(a, o); return r; }
    SKL_DEV double value() const { return ff_to_double(a); }
};
template <>
struct Acc<false> {
    double a = 0.0;
    SKL_DEV void fma_mv(double m, double x) { a = fma(m, x, a); }
    SKL_DEV void fma_f(double m, double x) { a = fma(m, x, a); }
    SKL_DEV void add(const Acc& o) { a += o.a; }
    SKL_DEV Acc shfl_xor(int o) const { Acc r; r.a = __shfl_xor_sync(0xffffffffu, a, o); return r; }
    SKL_DEV double value() const { return a; }
};

template <bool MIXED>
using MatT = typename std::conditional<MIXED, float, double>::type;
template <bool MIXED>
using ValT = typename VecT<MIXED>::type;   // stored A values: float2 (hi,lo) or double

}  // namespace skl
