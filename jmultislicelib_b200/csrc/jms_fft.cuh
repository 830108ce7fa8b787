// jms_fft.cuh -- register/shared-memory FFT building blocks for sm_100a.
//
// The multislice step needs unnormalised 2-D C2C transforms of the wave
// (forward = exp(-i), inverse = exp(+i), no scaling), as the reference takes
// them from cuFFT (src/JFFTCUDAcore.cpp:299-336) and MKL
// (src/JFFTMKLcore.cpp:170-241).  Here every 1-D line transform of length
// N = A*B is done in two register stages with one shared-memory exchange:
//
//   stage 1: thread j (0 <= j < B) holds x[j + B*m], m < A; it runs an
//            A-point DFT in registers and multiplies by W_N^(j*k1);
//   exchange through shared memory;
//   stage 2: thread k1 (0 <= k1 < A) holds the B values of row k1 and runs a
//            B-point DFT; it ends up with X[k1 + A*k2], k2 < B.
//
// Both the loads before stage 1 (stride-B elements per thread, consecutive
// threads on consecutive elements) and the stores after stage 2 are
// coalesced, so a line never needs a staging pass through shared memory.
// A forward transform with (A,B) leaves data in exactly the layout an inverse
// transform with (B,A) expects, which lets one kernel run FT -> x P -> IFT
// (or IFT -> x t -> FT) on a line without touching global memory in between.
//
// In-register DFTs are mixed radix (2, 3, 4, 5) with compile-time twiddles:
// every index is a template constant (static_for), so the twiddles are literal
// constants computed in double by constexpr trigonometry and rounded once.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace jms {

// ---------------------------------------------------------------------------
// compile-time loops and trigonometry
// ---------------------------------------------------------------------------
template <int... Is, class F>
__device__ __forceinline__ void static_for_impl(std::integer_sequence<int, Is...>, F&& f)
{
	(f(std::integral_constant<int, Is>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f)
{
	static_for_impl(std::make_integer_sequence<int, N>{}, f);
}

constexpr double kPi = 3.14159265358979323846264338327950288;

// sin and cos of x for |x| <= pi/4 by Taylor series (exact to double rounding)
__host__ __device__ constexpr double cx_sin_small(double x)
{
	double t = x, s = x;
	for (int k = 1; k < 14; k++) { t *= -x * x / ((2.0 * k) * (2.0 * k + 1.0)); s += t; }
	return s;
}
__host__ __device__ constexpr double cx_cos_small(double x)
{
	double t = 1.0, s = 1.0;
	for (int k = 1; k < 14; k++) { t *= -x * x / ((2.0 * k - 1.0) * (2.0 * k)); s += t; }
	return s;
}
// cos / sin of 2*pi*num/den with exact octant reduction in integers
__host__ __device__ constexpr double cx_cos_turn(long num, long den)
{
	num %= den; if (num < 0) num += den;
	// angle = 2 pi num/den; work in units of den/8 (octants)
	long n8 = num * 8;
	long oct = n8 / den;                 // octant 0..7
	double frac = (double)(n8 - oct * den) / (double)den; // in [0,1) of an octant
	double x = frac * (kPi / 4.0);
	double c = 0, s = 0;
	switch (oct) {
	case 0: c = cx_cos_small(x); break;
	case 1: c = cx_sin_small(kPi / 4.0 - x); break;
	case 2: c = -cx_sin_small(x); break;
	case 3: c = -cx_cos_small(kPi / 4.0 - x); break;
	case 4: c = -cx_cos_small(x); break;
	case 5: c = -cx_sin_small(kPi / 4.0 - x); break;
	case 6: c = cx_sin_small(x); break;
	default: c = cx_cos_small(kPi / 4.0 - x); break;
	}
	(void)s;
	return c;
}
__host__ __device__ constexpr double cx_sin_turn(long num, long den)
{
	// sin(2 pi num/den) = cos(2 pi (num/den - 1/4)) = cos(2 pi (4 num - den) / (4 den))
	return cx_cos_turn(4 * num - den, 4 * den);
}

// ---------------------------------------------------------------------------
// complex helpers
// ---------------------------------------------------------------------------
// Complex add and subtract as one packed FP32x2 instruction each (sm_100:
// add.f32x2 / fma.f32x2, both lanes rounded to nearest like the scalar
// forms).  a - b is formed as fma(b, -1, a): b * -1 is exact, so the result is
// the correctly rounded difference.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
	return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) // a * conj(b)
{
	return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ float cnorm(float2 a) { return fmaf(a.x, a.x, a.y * a.y); }

// The same element of two waves: real parts and imaginary parts side by side,
// so that every complex operation on the two waves is a packed one with the
// rounding of the scalar form, a wave's result does not depend on which of
// the two places it takes, and factors common to both waves (twiddles, the
// propagator, the grating of one configuration) are loaded once.  Packed FP32
// runs at the scalar rate per value (measured 0.48 packed against 0.97 scalar
// operations per cycle and SM quarter), with broadcast and negated operands
// free: what it saves is issue slots.  In memory: re0, re1, im0, im1.
struct __align__(16) cpair {
	float2 re, im;
};
__device__ __forceinline__ float2 bcast(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ cpair cadd(cpair a, cpair b) { return {__fadd2_rn(a.re, b.re), __fadd2_rn(a.im, b.im)}; }
__device__ __forceinline__ cpair csub(cpair a, cpair b)
{
	return {__fadd2_rn(a.re, neg2(b.re)), __fadd2_rn(a.im, neg2(b.im))};
}
__device__ __forceinline__ cpair cmul(cpair a, float2 w)
{
	return {__ffma2_rn(a.re, bcast(w.x), __fmul2_rn(a.im, bcast(-w.y))),
		__ffma2_rn(a.re, bcast(w.y), __fmul2_rn(a.im, bcast(w.x)))};
}
__device__ __forceinline__ cpair cmulc(cpair a, float2 w) // a * conj(w)
{
	return {__ffma2_rn(a.re, bcast(w.x), __fmul2_rn(a.im, bcast(w.y))),
		__ffma2_rn(a.im, bcast(w.x), __fmul2_rn(a.re, bcast(-w.y)))};
}
// each wave times its own factor
__device__ __forceinline__ cpair cmul(cpair a, float2 w0, float2 w1)
{
	const float2 wr = make_float2(w0.x, w1.x), wi = make_float2(w0.y, w1.y);
	return {__ffma2_rn(a.re, wr, __fmul2_rn(a.im, neg2(wi))), __ffma2_rn(a.re, wi, __fmul2_rn(a.im, wr))};
}
__device__ __forceinline__ float2 cnorm(cpair a) { return __ffma2_rn(a.re, a.re, __fmul2_rn(a.im, a.im)); }

template <class V> __device__ __forceinline__ V czero();
template <> __device__ __forceinline__ float2 czero<float2>() { return make_float2(0.f, 0.f); }
template <> __device__ __forceinline__ cpair czero<cpair>() { return {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
// s a + b with a real s
__device__ __forceinline__ float2 cfma(float s, float2 a, float2 b) { return __ffma2_rn(bcast(s), a, b); }
__device__ __forceinline__ cpair cfma(float s, cpair a, cpair b)
{
	return {__ffma2_rn(bcast(s), a.re, b.re), __ffma2_rn(bcast(s), a.im, b.im)};
}
// b + s (-+i) a: -i for the forward, +i for the inverse transform
template <bool INV>
__device__ __forceinline__ float2 cfma_i(float s, float2 a, float2 b)
{
	return INV ? make_float2(fmaf(-s, a.y, b.x), fmaf(s, a.x, b.y)) : make_float2(fmaf(s, a.y, b.x), fmaf(-s, a.x, b.y));
}
template <bool INV>
__device__ __forceinline__ cpair cfma_i(float s, cpair a, cpair b)
{
	return INV ? cpair{__ffma2_rn(bcast(-s), a.im, b.re), __ffma2_rn(bcast(s), a.re, b.im)}
		: cpair{__ffma2_rn(bcast(s), a.im, b.re), __ffma2_rn(bcast(-s), a.re, b.im)};
}
// s a with a real s
__device__ __forceinline__ float2 cscale(float2 a, float s) { return __fmul2_rn(a, bcast(s)); }
__device__ __forceinline__ cpair cscale(cpair a, float s) { return {__fmul2_rn(a.re, bcast(s)), __fmul2_rn(a.im, bcast(s))}; }
// (im, -re) = -i a, and i a
__device__ __forceinline__ float2 cmul_mi(float2 a) { return make_float2(a.y, -a.x); }
__device__ __forceinline__ cpair cmul_mi(cpair a) { return {a.im, neg2(a.re)}; }
__device__ __forceinline__ float2 cmul_pi(float2 a) { return make_float2(-a.y, a.x); }
__device__ __forceinline__ cpair cmul_pi(cpair a) { return {neg2(a.im), a.re}; }
__device__ __forceinline__ float2 cneg(float2 a) { return neg2(a); }
__device__ __forceinline__ cpair cneg(cpair a) { return {neg2(a.re), neg2(a.im)}; }
__device__ __forceinline__ float2 cshfl_xor(float2 a, int lanes)
{
	return make_float2(__shfl_xor_sync(0xffffffffu, a.x, lanes), __shfl_xor_sync(0xffffffffu, a.y, lanes));
}
__device__ __forceinline__ cpair cshfl_xor(cpair a, int lanes) { return {cshfl_xor(a.re, lanes), cshfl_xor(a.im, lanes)}; }

// multiply by exp(sgn * 2 pi i E / R) with compile-time E, R; sgn = -1 for the
// forward transform, +1 for the inverse.  Trivial angles cost no multiply.
template <int E, int R, bool INV, class V>
__device__ __forceinline__ V twiddle_ct(V v)
{
	constexpr int e = ((E % R) + R) % R;
	if constexpr (e == 0) {
		return v;
	}
	else if constexpr (4 * e == R) { // angle -+pi/2: forward multiplies by -i
		return INV ? cmul_pi(v) : cmul_mi(v);
	}
	else if constexpr (2 * e == R) {
		return cneg(v);
	}
	else if constexpr (4 * e == 3 * R) {
		return INV ? cmul_mi(v) : cmul_pi(v);
	}
	else {
		constexpr float c = (float)cx_cos_turn(e, R);
		constexpr float s = INV ? (float)cx_sin_turn(e, R) : -(float)cx_sin_turn(e, R);
		return cmul(v, make_float2(c, s));
	}
}

__host__ __device__ constexpr int first_factor(int r)
{
	return (r % 4 == 0) ? 4 : (r % 2 == 0) ? 2 : (r % 3 == 0) ? 3 : (r % 5 == 0) ? 5 : r;
}

// In-register DFT of x[OFF + S*i], i < R (natural order in and out); V is
// float2 (one wave) or cpair (two waves).
template <int R, int S, int OFF, bool INV, class V, int LEN>
__device__ __forceinline__ void dft_reg(V (&x)[LEN])
{
	if constexpr (R == 1) {
		return;
	}
	else if constexpr (R == 2) {
		V a = x[OFF], b = x[OFF + S];
		x[OFF] = cadd(a, b);
		x[OFF + S] = csub(a, b);
	}
	else if constexpr (R == 3) {
		// X0 = a + t, X1,2 = (a - t / 2) -+ i sqrt(3)/2 (b - c), t = b + c
		constexpr float s3 = (float)cx_sin_turn(1, 3);
		const V a = x[OFF], t = cadd(x[OFF + S], x[OFF + 2 * S]), d = csub(x[OFF + S], x[OFF + 2 * S]);
		const V m = cfma(-0.5f, t, a);
		x[OFF] = cadd(a, t);
		x[OFF + S] = cfma_i<INV>(s3, d, m);
		x[OFF + 2 * S] = cfma_i<INV>(-s3, d, m);
	}
	else if constexpr (R == 4) {
		V a = x[OFF], b = x[OFF + S], c = x[OFF + 2 * S], d = x[OFF + 3 * S];
		V t0 = cadd(a, c), t1 = csub(a, c), t2 = cadd(b, d), t3 = twiddle_ct<1, 4, INV>(csub(b, d));
		x[OFF] = cadd(t0, t2);
		x[OFF + 2 * S] = csub(t0, t2);
		x[OFF + S] = cadd(t1, t3);
		x[OFF + 3 * S] = csub(t1, t3);
	}
	else if constexpr (R == 5) {
		// sums and differences of x1, x4 and x2, x3: the sums see cosines, the
		// differences sines (36 FP32 operations; the direct form takes 104)
		constexpr float c1 = (float)cx_cos_turn(1, 5), c2 = (float)cx_cos_turn(2, 5);
		constexpr float s1 = (float)cx_sin_turn(1, 5), s2 = (float)cx_sin_turn(2, 5);
		const V a = x[OFF];
		const V p = cadd(x[OFF + S], x[OFF + 4 * S]), q = cadd(x[OFF + 2 * S], x[OFF + 3 * S]);
		const V d = csub(x[OFF + S], x[OFF + 4 * S]), f = csub(x[OFF + 2 * S], x[OFF + 3 * S]);
		const V m1 = cfma(c2, q, cfma(c1, p, a)), m2 = cfma(c1, q, cfma(c2, p, a));
		const V u1 = cfma(s2, f, cscale(d, s1)), u2 = cfma(-s1, f, cscale(d, s2));
		x[OFF] = cadd(a, cadd(p, q));
		x[OFF + S] = cfma_i<INV>(1.f, u1, m1);
		x[OFF + 4 * S] = cfma_i<INV>(-1.f, u1, m1);
		x[OFF + 2 * S] = cfma_i<INV>(1.f, u2, m2);
		x[OFF + 3 * S] = cfma_i<INV>(-1.f, u2, m2);
	}
	else {
		// decimation in time: R = P * M; sub-DFTs on the P interleaved
		// sequences, twiddle W_R^(q k), then P-point DFTs across them.
		constexpr int P = first_factor(R);
		static_assert(P < R, "radices 2, 3, 4 and 5 only");
		constexpr int M = R / P;
		V t[R];
		// t[q*M + i] = x[OFF + S*(q + P*i)]
		static_for<P>([&](auto Q) {
			static_for<M>([&](auto I) { t[Q.value * M + I.value] = x[OFF + S * (Q.value + P * I.value)]; });
		});
		static_for<P>([&](auto Q) { dft_reg<M, 1, Q.value * M, INV>(t); });
		static_for<M>([&](auto K) {
			constexpr int k = K.value;
			V u[P];
			static_for<P>([&](auto Q) {
				constexpr int q = Q.value;
				u[q] = twiddle_ct<q * k, R, INV>(t[q * M + k]);
			});
			dft_reg<P, 1, 0, INV>(u);
			static_for<P>([&](auto Q) { x[OFF + S * (k + M * Q.value)] = u[Q.value]; });
		});
	}
}

} // namespace jms
