// tri_common.cuh -- constants and small device helpers shared by the kernels.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace tri {

// Physical constants and tolerances of the reference (constants.h:38-50,
// 117-118).  SQRTG is the reference's literal, not sqrt(9.81).
constexpr double kGravity = 9.81;
constexpr double kSqrtG = 3.132091953;
constexpr double kMaxValue = 1e10;  // "dry" cell dt sentinel (MAX_VALUE)

template <typename T>
__host__ __device__ constexpr T eps12();
template <>
__host__ __device__ constexpr double eps12<double>() { return 1e-12; }
// The FP32 form keeps the FP64 absolute threshold (the reference's
// single-precision build flushes flux contributions below 1e-6, which deletes
// the mass of thin sheet flow) and adds a relative one, kNoise32, for
// contributions that are rounding noise of larger terms.
template <>
__host__ __device__ constexpr float eps12<float>() { return 1e-12f; }

// FP32 form: relative size below which a face contribution is rounding noise
// of the terms that formed it (about 17 float ulps).
constexpr double kNoise32 = 2e-6;

__device__ __forceinline__ double dev_sqrt(double x) { return sqrt(x); }
// FP32 form: the approximate hardware square root, one PTX instruction, so it
// is the same in every kernel the solver is inlined into.
__device__ __forceinline__ float dev_sqrt(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ double dev_cbrt(double x) { return cbrt(x); }
__device__ __forceinline__ float dev_cbrt(float x) { return cbrtf(x); }
__device__ __forceinline__ double dev_fabs(double x) { return fabs(x); }
__device__ __forceinline__ float dev_fabs(float x) { return fabsf(x); }
__device__ __forceinline__ double dev_fmax(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float dev_fmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double dev_fmin(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ float dev_fmin(float a, float b) { return fminf(a, b); }

__device__ __forceinline__ double dev_fma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float dev_fma(float a, float b, float c) { return fmaf(a, b, c); }

// IEEE quotient a / b, compiled out of line: for divisions on paths the
// solver rarely takes (entropy fix, dry-side tests, the fallback of
// div_shared), so their instruction sequences do not crowd the instruction
// cache of the step loop (ncu showed 17 % of warp cycles stalled on
// instruction fetch with them inline; out of line: FP64 flux launches 3-6 %
// shorter).  The same rounding as an inline '/'.  The FP32 form's quotient
// is short and stays inline (out of line measured 1 % slower there).
static __device__ __noinline__ double div_rare(double a, double b) { return a / b; }
__device__ __forceinline__ float div_rare(float a, float b) { return a / b; }

// a / b rounded to nearest from y = RN(1/b), the correctly rounded reciprocal
// (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990): q0 = RN(a*y) is within
// one ulp of a/b, the residual r = a - b*q0 is exact in one fused
// multiply-add, and RN(q0 + r*y) is the correctly rounded quotient.  The
// theorem needs a, b and a/b normal (no overflow or underflow).  Three
// operations instead of a full division when the divisor is reused.  For a
// dividend that is never a zero (and never subnormal): with q0 != 0, an exact
// quotient (r == 0) gives fma(0, y, q0) == q0.  The solver's uses: dt*p with
// |p| >= 1e-12 (smaller face contributions are flushed to +0 before, and dt*(+0)
// is the exact quotient +0 both ways: r = +0, fma(+0, y, +0) = +0), and h*dx/2
// (a depth far above the subnormal range, or a zero whose sign does not matter).
template <typename T>
__device__ __forceinline__ T div_nz(T a, T b, T y) {
  const T q0 = a * y;
  return dev_fma(dev_fma(-q0, b, a), y, q0);
}
template <>
__device__ __forceinline__ float div_nz<float>(float a, float, float y) {
  return a * y;
}

// a / b rounded to nearest for a divisor b shared by several quotients, from
// y = RN(1/b): Markstein's quotient where its conditions provably hold (|a| >=
// 2^-900 so the residual a - b*q0 is exact, and q0 = RN(a*y) between 2^-1000
// and 2^1000 so the quotient is normal), a plain division otherwise.  A zero
// dividend gives the signed zero of a/b.  Bit-identical to a / b for every
// finite a and finite non-zero b (a NaN dividend gives a NaN, not
// necessarily with the payload IEEE division would propagate); the solver
// divides by Roe-averaged celerities, sums of sqrt(h) and the friction term
// this way.  The conditions are tested as FP64 comparisons of magnitudes:
// the same tests on the exponent bits take integer instructions from the
// issue slots of an issue-limited kernel (Thacker 2048^2 FP64 flux launch
// 0.1270 ms with them, 0.1244 ms with comparisons); on the 32-bit high words,
// with the zero residual left to fma, they measured 17 % slower.
__device__ __forceinline__ double div_shared(double a, double b, double y) {
  const double q0 = a * y;
  const double fa = fabs(a), fq = fabs(q0);
  if (a != 0.0 && (fa < 0x1p-900 || fq < 0x1p-1000 || fq > 0x1p1000)) return div_rare(a, b);
  const double r = fma(-q0, b, a);
  return r == 0.0 ? q0 : fma(r, y, q0);
}
// FP32 form: one multiplication (within 1.5 ulp).
__device__ __forceinline__ float div_shared(float a, float, float y) { return a * y; }

// ---------------------------------------------------------------------------
// Straight-line square roots, reciprocals and quotients of the FP64 flux tile
// (no branch per operation).  They give the IEEE results for operands whose
// exponents keep every intermediate normal; the tile proves that for its
// cells with regular_cell() and is computed again with the guarded forms
// above where it does not hold.  Own design from published methods: a hardware
// seed (rsqrt / rcp approximation), one third-order Newton-Householder
// step, then Markstein's final corrections (exact FMA residual times the
// refined reciprocal; IBM J. Res. Dev. 34(1), 1990).  One seed serves both a
// square root and a reciprocal.  tri_selftest_division compares them with
// IEEE results bit for bit.  Why: a face is one long dependent FP64 chain, and
// a branch per square root and quotient (range test, slow path) keeps the
// compiler from interleaving its independent parts.  Flux launch of a Thacker
// bowl 2048^2 122.6 -> 101.4 us, of an all-wet 1531x2049 watershed 205 ->
// 166 us, of a 512^2 dam break (one tile per warp, pure latency) 40.9 ->
// 31.5 us.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rcp_seed(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
// x^-1/2 within about one ulp: with e = 1 - x*y0^2, y0*(1 + e/2 + 3e^2/8)
// leaves a relative error of 5e^3/16, below 2^-58 for a seed good to 2^-20.
// Rounded up: see recip_line.
__device__ __forceinline__ double rsqrt_line(double x) {
  const double y0 = rsqrt_seed(x);
  const double e = fma(-(x * y0), y0, 1.0);
  return __fma_ru(fma(e, 0.375, 0.5), y0 * e, y0);
}
// Square root from y, x^-1/2 within an ulp: the residual x - g*g is exact.
__device__ __forceinline__ double sqrt_line(double x, double y) {
  const double g = x * y;
  return fma(fma(-g, g, x), 0.5 * y, g);
}
// RN(1/b) from y, 1/b within two ulps.  A b whose mantissa is all ones has
// its reciprocal next to the midpoint of two doubles, where the last step is
// right only from above: the approximations it starts from are rounded up,
// and cells with such a depth are not regular (below).
__device__ __forceinline__ double recip_line(double b, double y) { return fma(y, fma(-b, y, 1.0), y); }
// RN(1/b) from a seed: y0*(1 + e + e^2) leaves a relative error of e^3.
__device__ __forceinline__ double recip_line(double b) {
  const double y0 = rcp_seed(b);
  const double e = fma(-b, y0, 1.0);
  return recip_line(b, __fma_ru(y0, fma(e, e, e), y0));
}
// RN(a/b) for b > 0 from y = RN(1/b).  The residual is taken negated, so that
// an exact quotient adds a zero of the sign that keeps a zero's own sign.
__device__ __forceinline__ double div_line(double a, double b, double y) {
  const double q0 = a * y;
  return fma(fma(q0, b, -a), -y, q0);
}

// True where the straight-line forms are exact on everything a face of this
// cell computes: h is 0 (of either sign, as rasters hold it) or within 2^-300 ..
// 2^100 and the discharges are at most 2^100 in magnitude, so velocities are at
// most 2^400 whatever depth they begin at, and no quotient passes 2^900.  A
// depth whose low word is all ones is left out (see recip_line; one depth in
// 2^32).  (Quotients of dividends below 2^-900 can then be off by 2^-700 at
// most, far below the 1e-12 flush of the contributions they enter.)  Ranges are
// tested on the high words, in integer slots; the zero in FP64, one instruction
// for two (flood of 96x150 1187 -> 1177 us a pass, rain 1531x2049 18.82 -> 18.72
// ms).
__device__ __forceinline__ bool regular_cell(double h, double qx, double qy) {
  constexpr uint32_t kLo = (1023u - 300u) << 20, kHi = (1023u + 100u) << 20;
  const uint32_t hh = (uint32_t)__double2hiint(h), hl = (uint32_t)__double2loint(h);
  const uint32_t ax = (uint32_t)__double2hiint(qx) & 0x7FFFFFFFu, ay = (uint32_t)__double2hiint(qy) & 0x7FFFFFFFu;
  const bool hok = (hh - kLo <= kHi - kLo && hl != 0xFFFFFFFFu) || h == 0.0;
  return hok && max(ax, ay) <= kHi;
}
__device__ __forceinline__ bool regular_cell(float, float, float) { return true; }

// Programmatic dependent launch: the step kernels are launched so that the
// next one may be scheduled while the previous one drains.  Each of them
// first waits until its predecessor has completed and its memory is visible
// (pdl_wait, before it reads or writes anything), so the order of their
// effects is exactly stream order; pdl_trigger lets the successor's launch
// begin once every block of this grid has reached it.  Both are no-ops for a
// kernel launched without the attribute.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Integer mix of a cell index and a step number (deterministic, so a batch
// member rounds exactly as its solo run).
__device__ __forceinline__ uint32_t cell_hash(uint32_t id, uint32_t step) {
  uint32_t x = id * 0x9E3779B1u ^ (step * 0x85EBCA77u + 0x27D4EB2Fu);
  x ^= x >> 15;
  x *= 0x2C1B3C6Du;
  x ^= x >> 12;
  x *= 0x297A2D39u;
  x ^= x >> 15;
  return x;
}

// a + b rounded stochastically between its two neighbouring floats
// (unbiased), computed in FP32: the rounding error of a + b is exact by
// Knuth's TwoSum, and the sum moves to the neighbour on the error's side with
// probability |error| / gap.  r uniform in [0, 2^32).  *exact_lo receives the
// error, so (double)RN(a + b) + error is the exact sum.
__device__ __forceinline__ float sr_add(float a, float b, uint32_t r, float* exact_lo) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  const float err = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  *exact_lo = err;
  if (err == 0.0f) return s;
  // the neighbour of s on the error's side, one step of its bits (s is not 0:
  // a sum that rounds to 0 is exact)
  const float t = __uint_as_float(__float_as_uint(s) + ((err > 0.0f) == (s > 0.0f) ? 1u : 0xFFFFFFFFu));
  const float u = (float)(r >> 8) * 0x1p-24f;
  return u * fabsf(t - s) < fabsf(err) ? t : s;
}

// Two products.  FP32: one instruction for both, each rounded (and flushed) as
// the single product is, since the FP32 flux kernel is bound by issue: rain on
// 4096^2 403.5 -> 378.4 us a launch, bowl 2048^2 65.2 -> 63.0.  Products only:
// of a paired product and a paired sum the assembler makes fused
// multiply-adds, which round otherwise.
__device__ __forceinline__ void mul2(float a0, float a1, float b0, float b1, float* r0, float* r1) {
  float x, y;
  asm("{\n.reg .b64 a, b, r;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\n"
      "mul.rn.ftz.f32x2 r, a, b;\nmov.b64 {%0, %1}, r;\n}"
      : "=f"(x), "=f"(y)
      : "f"(b0), "f"(b1), "f"(a0), "f"(a1));
  *r0 = x;
  *r1 = y;
}
__device__ __forceinline__ void mul2(double a0, double a1, double b0, double b1, double* r0, double* r1) {
  *r0 = a0 * b0;
  *r1 = a1 * b1;
}

// Reciprocal of a divisor shared by several quotients.  FP64: RN(1/b), as
// div_shared requires.  FP32 form: the hardware's approximate reciprocal
// (within 2 ulp), written as an intrinsic so it is the same instruction in
// every kernel the solver is inlined into (a compiler allowed to approximate
// divisions may rewrite them differently in different contexts, and a batch
// member must compute exactly what the same domain computes alone).
__device__ __forceinline__ double recip(double b) { return 1.0 / b; }
__device__ __forceinline__ float recip(float b) { return __fdividef(1.0f, b); }
// a / b where the FP32 form accepts the approximate quotient (same reason).
__device__ __forceinline__ double fdiv(double a, double b) { return a / b; }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }

// The CFL dt of a wet cell is RN(A / D) with A = RN(courant*dx) and the wave
// speed D = maxu + sqrt(g)*sqrt(h) (compute_dt_and_sqrt, kernels.h:167-193).
// RN(A / D) never increases with D, so the minimum over cells of the dt is
// RN(A / max D): the kernels reduce the largest D and divide once.  The slot
// holds kDtKeyInf - bits(D), an order-reversing key (bits of a non-negative
// double order like the double) under an unsigned atomic min; kDtKeyInf is
// the empty slot (no wet cell), and NaN speeds are left out (the reference's
// "a < m ? a : m" fold never selects a NaN dt).
constexpr unsigned long long kDtKeyInf = 0x7FF0000000000000ull;
__host__ __device__ inline unsigned long long speed_key(double d) {
  if (!(d >= 0.0)) return kDtKeyInf;
  unsigned long long b;
#ifdef __CUDA_ARCH__
  b = (unsigned long long)__double_as_longlong(d);
#else
  __builtin_memcpy(&b, &d, 8);
#endif
  return kDtKeyInf - (b > kDtKeyInf ? kDtKeyInf : b);
}
// dt of a slot: RN(A / D) for the largest speed, DBL_MAX for an empty slot.
__host__ __device__ inline double dt_of_key(unsigned long long key, double cfl_a) {
  if (key >= kDtKeyInf) return 1.7976931348623157e308;
  const unsigned long long b = kDtKeyInf - key;
  double d;
#ifdef __CUDA_ARCH__
  d = __longlong_as_double((long long)b);
#else
  __builtin_memcpy(&d, &b, 8);
#endif
  return cfl_a / d;
}


}  // namespace tri
