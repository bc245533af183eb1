// Device functions of the box-constrained solvers: predicates of bounds and iterates, the MPRGP step bound.
#pragma once
#include "device_util.cuh"

namespace ugpu {

// the predicates of MPRGP / VariableBoundSolverInterface with their comparisons on the integer
// pipes (device_util.cuh: exact for non-NaN bounds and iterates)
__device__ __forceinline__ double proj(double l, double u, double x) {
    const long long xk = dkey(x);
    return (dkey(l) >= xk) ? l : ((dkey(u) <= xk) ? u : x);
}
__device__ __forceinline__ double phi(double l, double u, double x, double g) { return (dlt(l, x) && dlt(x, u)) ? g : 0.0; }
// (|l - x| < 1e-14) ? min(0, g) : ((|u - x| < 1e-14) ? max(0, g) : 0)
__device__ __forceinline__ double chopped(double l, double u, double x, double g) {
    if (dabs_lt(l - x, 1e-14)) return dmin0(g);
    return dabs_lt(u - x, 1e-14) ? dmax0(g) : 0.0;
}

// the MPRGP step bound of one row as an order key (utopia_MPRGP.hpp:289-316, get_alpha_f:
// min((p > 0) ? (x - l) / p : 1e15, (p < 0) ? (x - u) / p : 1e15)), one division, the
// comparisons on the integer pipes
__device__ __forceinline__ unsigned long long qp_alpha_f_key(double x, double p, double l, double u) {
    const long long pk = dkey(p);
    if (pk == 0) return qp_key(1e15);
    const double h = (x - (pk > 0 ? l : u)) / p;
    const unsigned long long hk = qp_key(h), big = qp_key(1e15);
    return hk < big ? hk : big;
}
// A bracket [lo, hi] of qp_alpha_f_key's h = (x - l) / p (p > 0) or (x - u) / p (p < 0) from
// single-precision arithmetic alone, as order keys: the key of the double-precision h lies
// inside.  x, the bound b and p are truncated to binary32 (relative error < 2^-23 each); the
// difference x - b is used only where it does not cancel (|x| + |b| <= 8 |x - b|, so it is within
// 2^-20), and the quotient by the fast reciprocal (2 ulp) stays within 2^-19; the bracket widens it
// by 2^-16.  Rows with p = 0, and rows whose bound is at infinity on the side p moves towards
// (|b| >= 2^61, |p| < 2^10: h > 2^50 > 1e15), bound at the cap 1e15 and get no bracket
// (lo = hi = ~0); rows outside these cases (operands outside 2^-60 .. 2^60, cancellation) get
// lo = 0, hi = ~0: they are always evaluated exactly.
__device__ __forceinline__ void qp_alpha_f_bracket(double x, double p, double l, double u, unsigned long long &lo,
                                                   unsigned long long &hi) {
    const long long pk = dkey(p);
    if (pk == 0) {
        lo = hi = ~0ull;
        return;
    }
    const double b = pk > 0 ? l : u;
    const uint64_t bx = (uint64_t)__double_as_longlong(x), bb = (uint64_t)__double_as_longlong(b),
                   bp = (uint64_t)__double_as_longlong(p);
    const uint32_t ex = uint32_t(bx >> 52) & 0x7ffu, eb = uint32_t(bb >> 52) & 0x7ffu,
                   ep = uint32_t(bp >> 52) & 0x7ffu;
    lo = 0ull;  // by default: evaluated exactly
    hi = ~0ull;
    const bool x_ok = ex - 963u <= 120u || (bx << 1) == 0;  // 2^-60 <= |x| < 2^61, or zero
    const bool b_ok = eb - 963u <= 120u || (bb << 1) == 0;
    if (ep - 963u > 120u || !x_ok) return;
    if (!b_ok) {
        // b beyond 2^61 on the far side (b < 0 for p > 0, b > 0 for p < 0): h > 2^60 / 2^10
        const bool far = (pk > 0) == ((bb >> 63) != 0);
        if (eb >= 1084u && eb != 2047u && ep < 1033u && far) lo = hi = ~0ull;
        return;
    }
    auto trunc32 = [](uint64_t v, uint32_t e) {
        if ((v << 1) == 0) return __uint_as_float(uint32_t(v >> 32) & 0x80000000u);
        return __uint_as_float((uint32_t(v >> 32) & 0x80000000u) | ((e - 896u) << 23) |
                               uint32_t((v & 0xfffffffffffffull) >> 29));
    };
    const float xf = trunc32(bx, ex), bf = trunc32(bb, eb);
    const float af = xf - bf;
    if (!(fabsf(xf) + fabsf(bf) <= 8.0f * fabsf(af))) return;  // x - b cancels: evaluated exactly
    const float q = __fdividef(af, trunc32(bp, ep));
    const float q1 = q * (1.0f - 0x1p-16f), q2 = q * (1.0f + 0x1p-16f);
    lo = qp_key(f2d_bits(fminf(q1, q2)));
    hi = qp_key(f2d_bits(fmaxf(q1, q2)));
}
__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w < v ? w : v;
    }
    return v;
}
}  // namespace ugpu
