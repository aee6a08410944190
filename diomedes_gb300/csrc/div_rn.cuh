// div_rn.cuh -- several quotients by one divisor, each bit-identical to the
// IEEE round-to-nearest division a / b.
//
// solve6's unpivoted LDL^T divides 20 times by 5 distinct pivots.  For each
// pivot b the correctly rounded reciprocal y = RN(1/b) is formed once
// (__frcp_rn); each quotient then takes Markstein's final correction step
// (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Develop. 34(1), 1990):
//     q0 = RN(a y),   s = b q0 - a (exact: one FMA),   q = RN(q0 - s y),
// which gives q = RN(a / b) when y = RN(1/b) and no intermediate leaves the
// normal range.  Quotients are used only for b in [2^-24, 2^40] and |a| in
// [2^-84, 2^100] or a = 0: then q0 lies in [2^-125, 2^125] (normal) and the
// last bit of b q0 above 2^-132, so s is exact and q0 needs no test; a zero a
// gives q0 = a y = a's zero, s = +0 and q = a's zero (the negated remainder
// keeps a -0 numerator's sign).  Every other case (zero, negative or extreme
// pivots, tiny, huge, infinite or NaN numerators) takes the IEEE division
// itself.  Within the range the computation scales exactly with the exponents
// of a and b, so it is checked against the IEEE division for every pair of
// significands a, b in [1, 2) (tests/test_gpu_division.py) and on random
// full-range pairs.
//
// The range is tested once for all quotients by a pivot, not per quotient:
// the per-quotient test and branch (about ten instructions) cost more than
// the three of the quotient itself and kept a column's chains from
// overlapping.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace dio {

// A divisor and (float) its correctly rounded reciprocal.
template <class R>
struct Pivot {
    R b;
    __device__ __forceinline__ explicit Pivot(R b_) : b(b_) {}
    __device__ __forceinline__ bool ok() const { return true; }
};
template <>
struct Pivot<float> {
    float b, y;
    __device__ __forceinline__ explicit Pivot(float b_) : b(b_) {
#ifdef __CUDA_ARCH__
        y = __frcp_rn(b_);
#endif
    }
    __device__ __forceinline__ bool ok() const { return b >= 0x1p-24f && b <= 0x1p40f; }  // false for NaN
};

// Forms quotients a / p.b and collects their numerators' magnitudes;
// in_range() then says whether the correction step was valid for all of
// them (with the pivots' ok()).  Other types: plain division.
template <class R>
struct Quotients {
    __device__ __forceinline__ R div(const Pivot<R>& p, R a) { return a / p.b; }
    __device__ __forceinline__ bool in_range() const { return true; }
};
template <>
struct Quotients<float> {
    // 2 bits(a) - 1 drops the sign and puts a zero above every magnitude, so
    // the minimum sees nonzero numerators only
    uint32_t lo = 0xFFFFFFFFu;
    float hi = 0.f;
    __device__ __forceinline__ float div(const Pivot<float>& p, float a) {
        const float q0 = __fmul_rn(a, p.y);
        const float s = __fmaf_rn(p.b, q0, -a);
        lo = min(lo, 2u * __float_as_uint(a) - 1u);
        hi = fmaxf(hi, fabsf(a));
        return __fmaf_rn(-s, p.y, q0);
    }
    // every |a| in [2^-84, 2^100] or zero (a NaN numerator gives NaN either way)
    __device__ __forceinline__ bool in_range() const { return lo >= 2u * 0x15800000u - 1u && hi <= 0x1p100f; }
};

// The quotients v[0..N) / p.b in place.
template <int N, class R>
__device__ __forceinline__ void divide_all(const Pivot<R>& p, R (&v)[N]) {
    Quotients<R> qs;
    R q[N];
#pragma unroll
    for (int k = 0; k < N; ++k) q[k] = qs.div(p, v[k]);
    if (!(qs.in_range() && p.ok())) {
#pragma unroll
        for (int k = 0; k < N; ++k) q[k] = v[k] / p.b;
    }
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = q[k];
}

// One quotient at a time.
template <class R>
struct Divisor {
    Pivot<R> p;
    __device__ __forceinline__ explicit Divisor(R b) : p(b) {}
    __device__ __forceinline__ R div(R a) const {
        R v[1] = {a};
        divide_all(p, v);
        return v[0];
    }
};

}  // namespace dio
