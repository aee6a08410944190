// cvt64.cuh -- conversions between FP64 poses and FP32 arithmetic (the split
// precision), bit-identical to the hardware's conversions.
//
// FP64 instructions, conversions among them, issue once in 64 cycles on an
// SM sub-partition of this part (measured, one warp: 64 cycles a DADD or
// DMUL, 64 to 98 a conversion either way), so a split-precision primal was
// bound by them.  Conversions of values in FP32's normal range and of zeros
// are formed with integer instructions (the bits of the value moved between
// the formats; to FP32 rounded to nearest, ties to even); every other value
// (subnormal, overflowing, infinite, NaN) takes the conversion instruction.
#pragma once

#include "dio_math.cuh"

namespace dio {

__device__ __forceinline__ double widen(float x) {
    const uint32_t b = __float_as_uint(x), m = b & 0x7FFFFFFFu;
    if (m - 0x00800000u < 0x7F000000u || m == 0u) {  // normal, or zero
        const uint32_t hi = m ? (m >> 3) + 0x38000000u : 0u;
        return __hiloint2double((int)(hi | (b & 0x80000000u)), (int)(b << 29));
    }
    return (double)x;
}
__device__ __forceinline__ double widen(double x) { return x; }

__device__ __forceinline__ float to_float(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x), m = hi & 0x7FFFFFFFu;
    const bool zero = (m | lo) == 0u;
    // exponents -126 .. 126: rounding up stays finite
    if (m - 0x38100000u < 0x0FD00000u || zero) {
        const uint32_t t = __funnelshift_l(lo, hi, 3);  // exponent's low bits and the leading 23 of the fraction
        const uint32_t up = ((lo & 0x1FFFFFFFu) + 0x0FFFFFFFu + (t & 1u)) >> 29;
        const uint32_t f = ((t & 0x7FFFFFFFu) ^ 0x40000000u) + up;
        return __uint_as_float((zero ? 0u : f) | (hi & 0x80000000u));
    }
    return (float)x;
}
template <class R, class P>
__device__ __forceinline__ R narrow(P x) {
    if constexpr (sizeof(R) < sizeof(P))
        return to_float(x);
    else
        return x;
}
template <class R, class P>
__device__ __forceinline__ V3<R> narrow3(V3<P> a) { return {narrow<R>(a.x), narrow<R>(a.y), narrow<R>(a.z)}; }
template <class R, class P>
__device__ __forceinline__ Q4<R> narrowq(Q4<P> q) {
    return {narrow<R>(q.x), narrow<R>(q.y), narrow<R>(q.z), narrow<R>(q.w)};
}
template <class P, class R>
__device__ __forceinline__ V3<P> widen3(V3<R> a) {
    if constexpr (sizeof(R) < sizeof(P))
        return {widen(a.x), widen(a.y), widen(a.z)};
    else
        return a;
}

// quat_step of the split mode: the increment (d, 0) * q / 2 is formed in R
// from the rounded quaternion and added to the P quaternion; 1/|q| is seeded
// in R (correctly rounded sqrt and division) and refined by one Newton step
// in P (relative error ~1e-14; the quaternion is renormalised every step),
// or taken in P when |u|^2 lies outside [1e-30, 1e30].
// qr: q rounded to R.
template <class P, class R>
__device__ __forceinline__ Q4<P> quat_step_split(Q4<P> q, Q4<R> qr, V3<R> d) {
    Q4<R> s = qmul(Q4<R>{d.x, d.y, d.z, R(0)}, qr);
    s = {s.x * R(0.5), s.y * R(0.5), s.z * R(0.5), s.w * R(0.5)};
    const Q4<P> u{q.x + widen(s.x), q.y + widen(s.y), q.z + widen(s.z), q.w + widen(s.w)};
    const P n = u.x * u.x + u.y * u.y + u.z * u.z + u.w * u.w;
    // an R seed only where n and its root stay well inside R's range; a
    // quaternion blown up by a huge increment (|u|^2 beyond R) is normalised
    // in P (an R seed would overflow to a zero quaternion, then NaN)
    P r;
    // n in [2^-98, 2^99) -- inside that range -- is told from its exponent,
    // where halving it is a subtraction from the exponent
    const uint32_t hi = (uint32_t)__double2hiint(n);
    if (hi - 0x39D00000u < 0x46200000u - 0x39D00000u) {
        const P half = __hiloint2double((int)(hi - 0x00100000u), __double2loint(n));
        r = widen(R(1) / dsqrt(narrow<R>(n)));
        r = r * (P(1.5) - half * r * r);
    } else if (n > P(1.0e-30) && n < P(1.0e30)) {
        r = widen(R(1) / dsqrt(narrow<R>(n)));
        r = r * (P(1.5) - P(0.5) * n * r * r);
    } else {
        r = P(1) / dsqrt(n);
    }
    return {u.x * r, u.y * r, u.z * r, u.w * r};
}

}  // namespace dio
