// tri_selftest.cu -- tri_selftest_division: checks on the device that the
// exact quotients from a correctly rounded reciprocal equal the IEEE quotient
// bit for bit: div_nz over operands shaped like the step's (dt*d/dx,
// h*dx/2/dt: magnitudes 1e-14 .. 1e7 over divisors 1e-3 .. 1e3) and
// div_shared over every finite dividend magnitude (subnormals included,
// zeros of both signs) and divisors of either sign from 1e-30 to 1e30.  Also
// the straight-line forms of the FP64 flux tile (tri_common.cuh) over the range
// of its faces, 2^-300 .. 2^300 (depths end at 2^100), a part of it at operands
// whose result lies next to the midpoint of two doubles or whose mantissa is all
// ones, and over that of its friction terms, 2^-700 .. 2^760.
#include <cuda_runtime.h>

#include "tri_common.cuh"
#include "tri_internal.h"

using namespace tri;

namespace {

__device__ __forceinline__ unsigned long long mix(unsigned long long x) {
  // splitmix64 finaliser
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

__device__ __forceinline__ double unit(unsigned long long r) { return (double)(r >> 11) * (1.0 / 9007199254740992.0); }

__device__ __forceinline__ bool differ(double a, double b) {
  return __double_as_longlong(a) != __double_as_longlong(b);
}

// Mismatches of the straight-line forms for one random x of 2^-300 .. 2^300.
__device__ int line_check(unsigned long long r1, unsigned long long r2) {
  const int e = (int)((r1 >> 52) % 600) - 300;
  const double m = __longlong_as_double((long long)((r1 & 0x000FFFFFFFFFFFFFull) | 0x3FF0000000000000ull));  // 1 .. 2
  double x = ldexp(m, e);
  switch (r2 & 7) {
    case 0: {  // sqrt(x) next to the midpoint above m
      const double s = ldexp(m, e / 2), u = ldexp(0x1p-53, e / 2);
      x = s * s + 2.0 * s * u;
      break;
    }
    case 1: {  // 1/x next to the midpoint above m
      const double y = 1.0 / m;
      x = ldexp(fma(-y * y, 0x1p-53, y), e);
      break;
    }
    case 2:  // mantissa of (nearly) all ones or (nearly) all zeros
      x = ldexp((r2 & 8) ? 2.0 - (double)((r2 >> 4) & 3) * 0x1p-52 - 0x1p-52 : 1.0 + (double)((r2 >> 4) & 3) * 0x1p-52, e);
      break;
    case 3: {  // sqrt(x) of (nearly) all ones
      const double t = ldexp(2.0 - (double)((r2 >> 4) & 1) * 0x1p-52 - 0x1p-52, e / 2);
      x = t * t;
      x = __longlong_as_double(__double_as_longlong(x) + (long long)((r2 >> 5) & 3) - 1);
      break;
    }
    default: break;
  }
  int bad = 0;
  const double y = rsqrt_line(x), s = sqrt_line(x, y), rx = 1.0 / x;
  bad += differ(s, sqrt(x));
  if (__double2loint(x) != -1) bad += differ(recip_line(x, y * y), rx);  // such depths are not regular
  bad += differ(recip_line(s, y), 1.0 / s);
  bad += differ(recip_line(x), rx);
  const double a = ldexp(1.0 + (double)(r2 >> 12) * 0x1p-52, (int)(r2 % 601) - 300) * ((r2 & 16) ? -1.0 : 1.0);
  bad += differ(div_line(a, x, rx), a / x);
  bad += div_line(0.0, x, rx) != 0.0;
  const int ew = (int)((r1 >> 8) % 1460) - 700;  // friction terms and their denominators
  const double w = ldexp(m, ew), rw = 1.0 / w;
  bad += differ(sqrt_line(w, rsqrt_line(w)), sqrt(w));
  bad += differ(recip_line(w), rw);
  const int lo = max(-300, ew - 960), hi = min(751, ew + 760);
  const double d = ldexp(1.0 + (double)(r2 >> 12) * 0x1p-52, lo + (int)((r2 >> 8) % (unsigned)(hi - lo + 1)));
  bad += differ(div_line(d, w, rw), d / w);
  return bad;
}

__global__ void k_div_check(long long n, unsigned long long seed, unsigned long long* bad) {
  unsigned long long local = 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long r1 = mix(seed ^ (2 * i)), r2 = mix(seed ^ (2 * i + 1));
    const double ea = -14.0 + 21.0 * unit(r1);  // |a| in 1e-14 .. 1e7
    const double eb = -3.0 + 6.0 * unit(r2);    // b in 1e-3 .. 1e3
    double a = exp10(ea) * ((r1 & 1) ? -1.0 : 1.0);
    const double b = exp10(eb);
    if ((r2 & 0xFF) == 0) a = 0.0;
    const double y = 1.0 / b;
    const double q = div_nz(a, b, y);
    const double ref = a / b;
    if (__double_as_longlong(q) != __double_as_longlong(ref)) local++;
    // div_shared over any finite dividend (subnormal to 1e300) and divisors
    // 1e-30 .. 1e30
    const unsigned long long r3 = mix(seed ^ (0x5DEECE66Dull + 2 * i)), r4 = mix(r3);
    double a2 = exp10(-320.0 + 620.0 * unit(r3)) * ((r3 & 1) ? -1.0 : 1.0);
    if ((r4 & 0x3F) == 0) a2 = (r4 & 0x40) ? -0.0 : 0.0;
    const double b2 = exp10(-30.0 + 60.0 * unit(r4)) * ((r4 & 0x80) ? -1.0 : 1.0);
    const double q2 = div_shared(a2, b2, 1.0 / b2);
    if (__double_as_longlong(q2) != __double_as_longlong(a2 / b2)) local++;
    local += (unsigned)line_check(mix(r3 ^ 0x2545F4914F6CDD1Dull), r4);
  }
  if (local) atomicAdd(bad, local);
}

}  // namespace

extern "C" int tri_selftest_division(int64_t n, uint64_t seed, int64_t* mismatches) {
  TRI_CHECK_ARG(mismatches && n >= 0, "bad argument");
  unsigned long long* dbad = nullptr;
  TRI_CUDA_TRY(cudaMalloc(&dbad, sizeof(unsigned long long)));
  cudaMemset(dbad, 0, sizeof(unsigned long long));
  k_div_check<<<148 * 8, 256>>>(n, seed, dbad);
  cudaError_t e = cudaGetLastError();
  unsigned long long h = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&h, dbad, sizeof(h), cudaMemcpyDeviceToHost);
  cudaFree(dbad);
  if (e != cudaSuccess) return set_error(TRI_E_CUDA, "division self-test: %s", cudaGetErrorString(e));
  *mismatches = (int64_t)h;
  return TRI_OK;
}
