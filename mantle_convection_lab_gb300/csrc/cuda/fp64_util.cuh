// Arithmetic of the converged solvers that keeps work off the FP64 pipe (two
// lanes per clock and SM on GB300, FP32 128): conversions between FP32 and FP64,
// and the divergence of FP32 velocities in pairs of FP32 values.
#pragma once
#include "mclg_dev.cuh"

namespace mclg {

// F2F between FP32 and FP64 runs at the FP64 rate on GB300 (measured 595 G
// conversions/s, the rate of DFMA; FP32 FMA 33.4 T/s): exact widening and
// round-to-nearest narrowing by integer operations, with the instruction itself
// only for the values outside the formats' common normal range.
__device__ __forceinline__ double widen(float f)
{
	const unsigned u = __float_as_uint(f), ex = (u >> 23) & 0xffu;
	if (__builtin_expect(ex - 1u >= 254u && (u << 1) != 0u, 0))
		return (double)f;   // subnormal, infinite or NaN
	const unsigned hi = (u & 0x80000000u) | ((ex ? ((u & 0x7fffffffu) >> 3) + (896u << 20) : 0u));
	return __hiloint2double((int)hi, (int)(u << 29));
}
__device__ __forceinline__ double widen(double d) { return d; }

__device__ __forceinline__ float narrow(double d)
{
	const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
	const unsigned ex = (hi >> 20) & 0x7ffu;
	if (__builtin_expect(ex - 897u >= 253u, 0)) {   // outside 2^-126 <= |d| < 2^127
		if (ex == 0u)   // zero (a subnormal double rounds to it)
			return __uint_as_float(hi & 0x80000000u);
		return (float)d;
	}
	// the 29 bits that go away decide the rounding, to even on a tie; a carry
	// into the exponent is the correctly rounded next power of two
	const unsigned keep = ((hi & 0x7fffffffu) << 3 | lo >> 29) - (896u << 23);
	const unsigned rest = lo & 0x1fffffffu;
	const unsigned up = (rest > 0x10000000u || (rest == 0x10000000u && (keep & 1u))) ? 1u : 0u;
	return __uint_as_float((hi & 0x80000000u) | (keep + up));
}
template <class T> __device__ __forceinline__ T narrow_to(double d);
template <> __device__ __forceinline__ float narrow_to<float>(double d) { return narrow(d); }
template <> __device__ __forceinline__ double narrow_to<double>(double d) { return d; }

// a + b = s + e exactly (Knuth's TwoSum)
__device__ __forceinline__ void two_sum_f(float a, float b, float &s, float &e)
{
	s = __fadd_rn(a, b);
	const float bb = __fsub_rn(s, a);
	e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// (a + b) - (c + d) of four FP32 values as a pair of floats (see gt_elem)
__device__ __forceinline__ void diff4(float a, float b, float c, float d, float &s, float &l)
{
	float p, pe, q, qe, t;
	two_sum_f(a, b, p, pe);
	two_sum_f(c, d, q, qe);
	two_sum_f(p, -q, s, t);
	l = __fadd_rn(t, __fsub_rn(pe, qe));
}

// (G^T u)_e from the element's corner velocities (0 = (ex,ez), 1 = (ex,ez+1),
// 2 = (ex+1,ez+1), 3 = (ex+1,ez)): g0 [(u0+u1) - (u2+u3)] + g1 [(w0+w3) - (w1+w2)].
// In FP32 the sums run as float pairs on the FP32 pipe and the FP64 pipe only adds and
// scales the result: to 2^-52 of the largest product where the corners' values are of
// one size, to 2^-47 over 12 binades (400000 random elements each; summing the products
// in float pairs corner by corner gives 2^-52 and 2^-46.5, and 2^-43 where the element
// is not square).  For the uniform meshes' MINRES: the FP64 residual around it
// runs on the other overload.
__device__ __forceinline__ double gt_elem(float u0, float u1, float u2, float u3, float w0, float w1, float w2, float w3,
                                          double g0, double g1)
{
	float s, l, t, m;
	diff4(u0, u1, u2, u3, s, l);
	diff4(w0, w3, w1, w2, t, m);
	if (g0 == g1) {
		float a, e;
		two_sum_f(s, t, a, e);
		return g0 * (widen(a) + widen(__fadd_rn(e, __fadd_rn(l, m))));
	}
	return g0 * (widen(s) + widen(l)) + g1 * (widen(t) + widen(m));
}
__device__ __forceinline__ double gt_elem(double u0, double u1, double u2, double u3, double w0, double w1, double w2,
                                          double w3, double g0, double g1)
{
	return g0 * ((u0 + u1) - (u2 + u3)) + g1 * ((w0 + w3) - (w1 + w2));
}

}  // namespace mclg
