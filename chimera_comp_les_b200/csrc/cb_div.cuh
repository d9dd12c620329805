// Branch-free FP64 division and square root of the FP64 form.
//
// The FP64 form follows the reference's IEEE divisions (about 42 per cell of
// the MUSCL scheme, 190 of the WENO schemes).  CUDA's a / b carries a branch
// to a slow path, so the divisions of a face run one after another, each a
// chain of dependent FP64 operations; the stage kernel waits on those chains
// (FP64 pipe 34 % active).  Here a denominator's reciprocal is formed once and
// every quotient with it is corrected by its exact remainder (P. Markstein,
// IA-64 and Elementary Functions, 2000, ch. 8; Muller et al., Handbook of
// Floating-Point Arithmetic, 2018, sec. 4.7):
//   y0 ~ 1/b (rcp.approx, |1 - b y0| <= 2^-19.9 measured), e = 1 - b y0,
//   y = y0 + y0 (e + e^2)                    -- the cubic step, error 2^-53
//   q0 = a y,  r = a - b q0 (exact),  q = q0 + r y
// q is the IEEE quotient unless a / b lies within 2^-52 ulp of a rounding
// boundary (tests/test_gpu_quotients.py: random pairs, and pairs built from a
// boundary; a power of two over a mantissa of ones is such a pair), in 3 FP64
// operations per quotient after 3 for the reciprocal, with no branch, so the
// chains of a face's quotients overlap.  The square root is the same correction
// of a Goldschmidt iterate (IEEE unless within 2^-50 ulp of one).  Measured per
// time step, before and after, with bit-identical results: MUSCL + Rusanov 128^3
// 1.50 -> 1.36 ms, WENO3 blend 97x75x61 1.60 -> 1.00 ms, WENO5-JS + Roe 96^3
// 4.22 -> 2.86 ms, inviscid WENO5-JS + Rusanov 64^3 1.08 -> 0.63 ms; mixed form
// (the node reciprocal only) WENO5-JS + Roe 192^3 7.97 -> 7.85 ms.
//
// Range: that holds for denominators and radicands with |b| in 2^-960 .. 2^960
// (in_range) and finite numerators whose quotient does not overflow; below
// |a| = 2^-960 the remainder may underflow and q miss its last bit.  For other
// denominators the hardware approximations flush: a zero, infinite, subnormal or
// NaN b gives NaN, one above 2^1022 the finite value 0.  So the stage kernels do
// not rely on the result alone: every node's state is tested once, where it
// enters the ring (wide_state), and what a face can cancel (densities, c^2) or
// overflow is tested there; a tile march that met one out of bounds is done
// again with a / b and sqrt (FLUX_IEEE).  The bounds on the nodes leave room for
// everything the faces build from them: squared WENO smoothness measures stay
// below 2^960, their weights and sums above 2^-960.  The model's kernels test their
// results, where a NaN of a quotient shows, and the denominators' upper end, and
// form them again with a / b; the sensor takes quot.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

namespace cb {

__device__ __forceinline__ double rcp_approx(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
}
__device__ __forceinline__ double rsqrt_approx(double b) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
}

// FP32 (the mixed form): a / b as a times the hardware reciprocal.  For
// |b| < 2^126 it has the bits of the fast division the form is compiled with
// (-prec-div=false; none of 1.6e9 random pairs with exponents up to +-120
// differed, nor 1 / b, nor the square root), without that division's range
// scaling.  rcp_approx flushes: a larger b gives 0, a subnormal one infinity.  It
// serves the WENO weights, scaled so that no finite squared smoothness measure
// reaches 2^126, and the sum of two roots.  Densities and Roe's c^2 take 1 / b,
// and the roots sqrtf and rsqrtf: the full-range approximations (squared metrics
// are subnormal where a cell face is smaller than 1e-19).  Measured per step, with
// every quotient flushing: WENO5-JS + Roe 192^3 7.8 -> 5.9 ms, immersed sphere
// 96x96x128 1.91 -> 1.63 ms; the full-range ones take back 1.4 and 1.9 % (MUSCL
// 128^3 0.8 %).
__device__ __forceinline__ float rcp_approx(float b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  return y;
}

// Two FP32 values in one instruction (sm_100's packed FP32: the peak rate of
// the scalar one, 72 TFLOP/s measured for both, in half the issue slots, which
// is what the mixed stage kernel runs out of).  Each lane rounds as the scalar
// instruction does.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "mul.rn.f32x2 w, x, y;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "add.rn.f32x2 w, x, y;\n\tmov.b64 {%0, %1}, w;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float a, float2 b, float2 c) { return fma2(both(a), b, c); }
__device__ __forceinline__ float2 mul2(float a, float2 b) { return mul2(both(a), b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return fma2(both(-1.f), b, a); }
__device__ __forceinline__ float2 rcp2(float2 b) { return make_float2(rcp_approx(b.x), rcp_approx(b.y)); }

// A denominator: Den<R> d(b); d(a) = a / b.
template <typename R>
struct Den;
template <>
struct Den<float> {
  float y;
  __device__ __forceinline__ explicit Den(float b) : y(1.f / b) {}
  __device__ __forceinline__ Den(float, float y_) : y(y_) {}
  __device__ __forceinline__ Den doubled() const { return Den(0.f, 0.5f * y); }  // divides by 2 b
  // __fmul_rn: the quotient is rounded before it enters a sum
  __device__ __forceinline__ float operator()(float a) const { return __fmul_rn(a, y); }
};
template <>
struct Den<double> {
  double b, y;
  __device__ __forceinline__ explicit Den(double b_) : b(b_) {
    const double y0 = rcp_approx(b_), e = fma(-b_, y0, 1.0);
    y = fma(y0, fma(e, e, e), y0);
  }
  __device__ __forceinline__ Den doubled() const { return Den(2.0 * b, 0.5 * y); }  // divides by 2 b
  // a denominator whose reciprocal is known (rounded to nearest)
  __device__ __forceinline__ Den(double b_, double y_) : b(b_), y(y_) {}
  __device__ __forceinline__ double operator()(double a) const {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
  }
};

// A denominator that is well inside the range: FP32 by the flushing reciprocal.
template <typename R>
struct FlushDen : Den<R> {
  using Den<R>::Den;
};
template <>
struct FlushDen<float> {
  float y;
  __device__ __forceinline__ explicit FlushDen(float b) : y(rcp_approx(b)) {}
  __device__ __forceinline__ float operator()(float a) const { return __fmul_rn(a, y); }
};

// The same by a / b: for values out of the branch-free quotients' range.  Out of
// line, for code that hardly ever runs.
template <typename R>
static __device__ __noinline__ R plain_quot(R a, R b) { return a / b; }
template <typename R>
static __device__ __noinline__ R plain_root(R x) { return sqrt(x); }
template <typename R>
struct PlainDen {
  R b;
  __device__ __forceinline__ explicit PlainDen(R b_) : b(b_) {}
  __device__ __forceinline__ PlainDen doubled() const { return PlainDen(R(2.0) * b); }
  __device__ __forceinline__ R operator()(R a) const { return plain_quot(a, b); }
};
template <typename R, bool IEEE>
using DenOf = std::conditional_t<IEEE, PlainDen<R>, Den<R>>;
template <typename R, bool IEEE>
using FlushDenOf = std::conditional_t<IEEE, PlainDen<R>, FlushDen<R>>;

// a / 3 (FP64: with the reciprocal rounded to nearest)
template <typename R, bool IEEE>
__device__ __forceinline__ R third(R a) {
  if constexpr (sizeof(R) == 4) return a / R(3.0);
  else if constexpr (IEEE) return plain_quot(a, R(3.0));
  else return Den<double>(3.0, 1.0 / 3.0)(a);
}

__device__ __forceinline__ double root(double x) {
  const double z = rsqrt_approx(x);
  double g = x * z, h = 0.5 * z;
  const double r = fma(-g, h, 0.5), s = fma(r, 1.5 * r, r);
  g = fma(g, s, g);
  h = fma(h, s, h);
  return fma(fma(-g, g, x), h, g);
}
__device__ __forceinline__ float root(float x) { return sqrtf(x); }

template <bool IEEE>
__device__ __forceinline__ double by27(double a) {
  if constexpr (IEEE) return plain_quot(a, 27.0);
  else return Den<double>(27.0, 1.0 / 27.0)(a);
}
template <typename R, bool IEEE>
__device__ __forceinline__ R root_of(R x) {
  if constexpr (IEEE) return plain_root(x);
  else return root(x);
}

// false for an infinity or a NaN
__device__ __forceinline__ bool finite_hi(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) < 0x7ff00000u;
}

// the exponent bits of x above its sign-free high word: monotone in |x|
__device__ __forceinline__ unsigned mag_hi(double x) { return (unsigned)__double2hiint(x) << 1; }
__host__ __device__ constexpr unsigned mag_pow2(int e) { return (unsigned)(1023 + e) << 21; }  // mag_hi of 2^e
// |b| in 2^-960 .. 2^960
__device__ __forceinline__ bool in_range(double b) {
  return mag_hi(b) - mag_pow2(-960) < mag_pow2(960) - mag_pow2(-960);
}

// a / b as the branch-free quotient, redone by a / b where that leaves its range
// (an infinite or overflowing quotient included)
__device__ __forceinline__ double quot(double a, double b) {
  const double q = Den<double>(b)(a);
  return mag_hi(b) < mag_pow2(960) && finite_hi(q) ? q : a / b;
}

// Whether a node's conserved state v and pressure p lie outside |x| < 2^230,
// |rho| >= 2^-500 (also true for a NaN).  Inside, rho's quotients are in range
// and finite; differences of values square to at most 2^466 and, with the
// smoothness measures' coefficients, (eps + beta)^2 stays below 2^932.
__device__ __forceinline__ bool wide_state(const double *v, double p) {
  const unsigned r = mag_hi(v[0]);
  const unsigned a = max(max(r, mag_hi(v[1])), mag_hi(v[2])), b = max(max(mag_hi(v[3]), mag_hi(v[4])), mag_hi(p));
  return max(a, b) >= mag_pow2(230) || r < mag_pow2(-500);
}

}  // namespace cb
