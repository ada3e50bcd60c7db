// The arithmetic of the triangular solves in each precision: int32 fixed point
// with int64 accumulation, FP64, FP32.
#pragma once
#include <type_traits>

#include "../sagb_internal.hpp"
#include "common.cuh"

namespace sagb {

constexpr size_t kSmemMax = 227 * 1024;

template <int VT>
using vt_t = typename std::conditional<VT == VT_I32, int, typename std::conditional<VT == VT_F64, double, float>::type>::type;
template <int VT>
using acc_t = typename std::conditional<VT == VT_I32, long long, vt_t<VT>>::type;

// t - v*o in the accumulator type of each precision
template <int VT, bool EXACT>
__device__ __forceinline__ acc_t<VT> acc_sub(acc_t<VT> t, vt_t<VT> v, vt_t<VT> o) {
    if constexpr (VT == VT_I32) return wsub(t, (long long)v * (long long)o);
    else if constexpr (EXACT && VT == VT_F64) return __dsub_rn(t, __dmul_rn(v, o));
    else if constexpr (EXACT) return __fsub_rn(t, __fmul_rn(v, o));
    else return t - v * o;
}
template <int VT>
__device__ __forceinline__ acc_t<VT> acc_init(vt_t<VT> in, int bit) {
    if constexpr (VT == VT_I32) return wshl((long long)in, bit);
    else return in;
}
template <int VT>
__device__ __forceinline__ acc_t<VT> acc_reduce(acc_t<VT> t, int G) {
    for (int o = G / 2; o > 0; o >>= 1) {
        if constexpr (VT == VT_I32) t = wadd(t, shfl_xor(t, o));
        else t += shfl_xor(t, o);
    }
    return t;
}
// out_i from the accumulated row: (t >> bit) * dinv >> dbit, or t * dinv
template <int VT>
__device__ __forceinline__ vt_t<VT> acc_finish(acc_t<VT> t, vt_t<VT> d, int bit, int dbit, bool &ovf) {
    if constexpr (VT == VT_I32) {
        const long long s = wmul(t >> bit, (long long)d) >> dbit;
        ovf |= !fits32(s);
        return lo32(s);
    } else if constexpr (VT == VT_F64) {
        return __dmul_rn(t, d);
    } else {
        return __fmul_rn(t, d);
    }
}

}  // namespace sagb
