// div_rn.cuh -- several quotients by one divisor, each bit-identical to the
// IEEE round-to-nearest division a / b.
//
// solve6's unpivoted LDL^T divides 21 times by 6 distinct pivots.  For each
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
// keeps a -0 numerator's sign).  Tiny numerators are scaled up, divided so and
// brought down again (quotient_tiny); every other case (zero, negative or
// extreme pivots, huge, infinite or NaN numerators) takes the IEEE division
// itself.  Within the range the computation scales exactly with the exponents
// of a and b, so it is checked against the IEEE division for every pair of
// significands a, b in [1, 2) (tests/test_gpu_division.py) and on random
// full-range pairs.
//
// The range is tested once for a whole system (or, in divide_all, for all
// quotients by a pivot), not per quotient: the per-quotient test and branch
// (about ten instructions) cost more than the three of the quotient itself and
// kept a column's chains from overlapping.  What fails the test is formed again
// by quotient_tiny, or by the division.
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

// RN(a / p.b) for a pivot in range and any |a| up to 2^100: what fails the test
// for a tiny numerator is formed again with.  Bodies at rest along the axes have
// products of rounding errors for off-diagonal entries, below 2^-84 and down to
// subnormal ones.
// A numerator below 2^-40 is taken times 2^72 (exact: a subnormal's least bit
// comes to 2^-77), and q = RN(2^72 a / b) brought down: exactly where 2^-72 q is
// normal, else rounded to the subnormals' step 2^-149 (2^-77 of q).  That second
// rounding goes the way of a single one unless q lies exactly between two steps;
// then the sign of the remainder b q - 2^72 a (exact: one FMA) tells on which
// side of q the quotient is, and a zero one leaves the tie to even.  Without a
// branch, so that a column's quotients overlap.
__device__ __forceinline__ float quotient_tiny(const Pivot<float>& p, float a) {
    const bool tiny = fabsf(a) < 0x1p-40f;
    const float n = __fmul_rn(a, tiny ? 0x1p72f : 1.f);
    const float q0 = __fmul_rn(n, p.y);
    const float q = __fmaf_rn(-__fmaf_rn(p.b, q0, -n), p.y, q0), mq = fabsf(q);
    float t = __fsub_rn(__fadd_rn(mq, 0x1p-54f), 0x1p-54f);  // to a multiple of 2^-77, ties to even
    const float rest = __fmaf_rn(p.b, mq, -fabsf(n));        // above 0: the quotient lies below q
    const bool tie = fabsf(__fsub_rn(mq, t)) == 0x1p-78f && rest != 0.f;
    t = tie ? __fadd_rn(mq, rest > 0.f ? -0x1p-78f : 0x1p-78f) : t;
    return __fmul_rn(tiny && mq < 0x1p-54f ? copysignf(t, a) : q, tiny ? 0x1p-72f : 1.f);
}

// The quotients v[k] / p[k] in place (divide_all: by one pivot).
template <int N, class R, class P>
__device__ __forceinline__ void divide_by(const P& pivot, R (&v)[N]) {
    Quotients<R> qs;
    R q[N];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        q[k] = qs.div(pivot(k), v[k]);
        ok = ok && pivot(k).ok();
    }
    if (!(ok && qs.in_range())) {
        bool plain = true;
        if constexpr (sizeof(R) == 4) {
            plain = !(ok && qs.hi <= 0x1p100f);
            if (!plain) {
#pragma unroll
                for (int k = 0; k < N; ++k) q[k] = quotient_tiny(pivot(k), v[k]);
            }
        }
        if (plain) {
#pragma unroll
            for (int k = 0; k < N; ++k) q[k] = v[k] / pivot(k).b;
        }
    }
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = q[k];
}
template <int N, class R>
__device__ __forceinline__ void divide_all(const Pivot<R>& p, R (&v)[N]) {
    divide_by(
        [&](int) -> const Pivot<R>& { return p; }, v);
}
template <int N, class R>
__device__ __forceinline__ void divide_each(const Pivot<R> (&p)[N], R (&v)[N]) {
    divide_by(
        [&](int k) -> const Pivot<R>& { return p[k]; }, v);
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
