// tri_face.cuh -- the per-face augmented Roe solver of TRITON, as a device
// function shared by every step kernel in this library.
//
// Reference: kernels_flux.h:84-273 (x faces, normal (1,0)) and :367-556
// (y faces, normal (0,1)).  "1" is the cell that owns the face, "2" the
// neighbour across it (east for x faces, NORTH for y faces: row-1).
//
// Bit-exactness contract: with T=double and the library's compile flags
// (--fmad=false, IEEE div/sqrt), every output equals the reference's bit for
// bit for finite states: each non-zero term keeps the reference's operand
// order and association.  Terms that are zero by construction are left out
// (products with the zero component of the face normal, contributions of a
// wave with zero speed, entropy-fix parts of waves without a fix): adding a
// zero never changes a non-zero sum, and a sum that is zero is flushed to +0
// before it is used, so only the sign of zeros inside the solver differs, and
// NaN propagation in a state that is already non-finite.
#pragma once

#include "tri_common.cuh"

namespace tri {

// Cell quantities every face of a cell uses, computed once per cell:
// velocities are zero below hextra (kernels_flux.h:98-117) and sqrt(h) is the
// reference's SQRTH array (kernels.h:178).
// z is the bed level (FP64 form) or the cell's FP32 offset from the FP64 base
// level of its 32x32 tile (FP32 form).
template <typename T>
struct CellQ {
  T h, qx, qy, z, sq, u, v;
  T hd;  // h*dx/2/dt, the limiter's bound: the same for the cell's four faces
};

// Result of one face: contributions to the owner (a) and to the neighbour (b),
// already scaled as rhs = dt*d/dx (kernels_flux.h:267-273).  'wet' is false for
// a dry-dry face (both scaled triples are then +0).
template <typename T>
struct FaceOut {
  T a0, a1, a2, b0, b1, b2;
};

// Step constants of the face solver: rdx = RN(1/dx) and rdt = RN(1/dt) turn
// the divisions by dx and dt into exact three-operation quotients.
template <typename T>
struct StepK {
  T dx, dt, rdx, rdt, hextra;
  bool dx_pow2;  // dx is a power of two: a / dx == a * rdx exactly (both round the same real)
};

// True for a positive normal power of two.
__host__ __device__ inline bool is_pow2(double x) {
  unsigned long long b;
#ifdef __CUDA_ARCH__
  b = (unsigned long long)__double_as_longlong(x);
#else
  __builtin_memcpy(&b, &x, 8);
#endif
  const unsigned long long e = b >> 52;
  return (b & 0x000FFFFFFFFFFFFFull) == 0 && e >= 1 && e <= 0x7FE;
}

template <typename T>
__host__ __device__ inline StepK<T> step_k(T dx, T dt, T rdx, T rdt, T hextra) {
  StepK<T> K;
  K.dx = dx;
  K.dt = dt;
  K.rdx = rdx;
  K.rdt = rdt;
  K.hextra = hextra;
  K.dx_pow2 = is_pow2((double)dx);
  return K;
}

// LINE: the FP64 straight-line forms, for cells that regular_cell() accepts.
template <typename T, bool LINE = false>
__device__ __forceinline__ CellQ<T> make_cell(T h, T qx, T qy, T z, const StepK<T>& K) {
  const T hextra = K.hextra;
  CellQ<T> c;
  c.h = h;
  c.qx = qx;
  c.qy = qy;
  c.z = z;
  c.hd = div_nz(h * K.dx * T(0.5), K.dt, K.rdt);
  if constexpr (LINE && sizeof(T) == 8) {
    const double hs = h > 0.0 ? h : 1.0;
    const double y = rsqrt_line(hs);
    const double s = sqrt_line(hs, y);
    const double rh = recip_line(hs, y * y);
    const bool flows = h >= hextra;
    c.sq = h > 0.0 ? s : 0.0;
    c.u = flows ? div_line(qx, hs, rh) : 0.0;
    c.v = flows ? div_line(qy, hs, rh) : 0.0;
    return c;
  }
  c.sq = dev_fmax(dev_sqrt(h), T(0));
  if constexpr (sizeof(T) == 4) {
    const T rh = recip(h);
    T u, v;
    mul2(rh, rh, qx, qy, &u, &v);
    c.u = h >= hextra ? u : T(0);
    c.v = h >= hextra ? v : T(0);
    return c;
  }
  if (h >= hextra) {
    const T rh = recip(h);
    c.u = div_shared(qx, h, rh);
    c.v = div_shared(qy, h, rh);
  } else {
    c.u = T(0);
    c.v = T(0);
  }
  return c;
}

// Products with the face normal (nx, ny) = (1,0) or (0,1): the component
// itself (the product with the zero component is a zero term).
template <typename T, bool XFACE>
__device__ __forceinline__ T n_dot(T a, T b) {  // a*nx + b*ny
  return XFACE ? a : b;
}
template <typename T, bool XFACE>
__device__ __forceinline__ T n_cross(T a, T b) {  // b*nx - a*ny
  return XFACE ? b : -a;
}

// A quotient by a shared divisor, its reciprocal given: straight-line or guarded.
template <bool LINE>
__device__ __forceinline__ double quot(double a, double b, double y) {
  return LINE ? div_line(a, b, y) : div_shared(a, b, y);
}
template <bool LINE>
__device__ __forceinline__ float quot(float a, float b, float y) {
  return div_shared(a, b, y);
}

// Two quotients by the same divisor.
template <bool LINE>
__device__ __forceinline__ void quot2(double a0, double a1, double b, double y, double* r0, double* r1) {
  *r0 = quot<LINE>(a0, b, y);
  *r1 = quot<LINE>(a1, b, y);
}
template <bool LINE>
__device__ __forceinline__ void quot2(float a0, float a1, float, float y, float* r0, float* r1) {
  mul2(y, y, a0, a1, r0, r1);
}

// cross, dzb (FP32 form): the cells lie in different bed tiles; base level of
// c2's minus that of c1's.
// LINE (FP64): both cells are regular (regular_cell), so square roots,
// reciprocals and shared quotients take their straight-line forms.
template <typename T, bool XFACE, bool LINE = false>
__device__ __forceinline__ FaceOut<T> face_flux(const CellQ<T>& c1, const CellQ<T>& c2, const StepK<T>& K,
                                                bool cross = false, double dzb = 0.0) {
  constexpr bool L64 = LINE && sizeof(T) == 8;
  const T dx = K.dx, dt = K.dt, hextra = K.hextra;
  const T G = T(kGravity), SG = T(kSqrtG), E12 = eps12<T>();
  FaceOut<T> out;
  out.a0 = out.a1 = out.a2 = out.b0 = out.b1 = out.b2 = T(0);

  const T h1 = c1.h, h2 = c2.h;
  const bool brink = !(h1 >= E12 && h2 >= E12);  // next to a dry cell, or one whose depth is no number
  if (brink && !(h1 > T(0) || h2 > T(0))) return out;

  const T u1 = c1.u, v1 = c1.v, u2 = c2.u, v2 = c2.v;
  const T sqh1 = c1.sq, sqh2 = c2.sq;

  // Roe-averaged state and wave speeds
  const T h12 = T(0.5) * (h1 + h2);
  const T dh = h2 - h1;
  const T ssq = sqh1 + sqh2;
  T c12, rc12, rssq;  // shared divisors: exact quotients via quot
  if constexpr (L64) {
    const T gh = G * h12;
    const T y = rsqrt_line(gh);
    c12 = sqrt_line(gh, y);
    rc12 = recip_line(c12, y);
    rssq = recip_line(ssq);
  } else {
    c12 = dev_sqrt(G * h12);
    rc12 = recip(c12);
    rssq = recip(ssq);
  }
  T u12, v12;
  T us1, vs1, us2, vs2;
  mul2(sqh1, sqh1, u1, v1, &us1, &vs1);
  mul2(sqh2, sqh2, u2, v2, &us2, &vs2);
  quot2<L64>(us1 + us2, vs1 + vs2, ssq, rssq, &u12, &v12);
  const T un = n_dot<T, XFACE>(u12, v12);
  T lam0 = un - c12, lam1 = un, lam2 = un + c12;
  T lamE0 = T(0), lamE2 = T(0);  // lamE1 is always zero
  bool fixed = false;

  // Harten-Hyman style entropy fix on the acoustic waves (rare: one branch)
  {
    const T un1 = n_dot<T, XFACE>(u1, v1), un2 = n_dot<T, XFACE>(u2, v2);
    T g1, g2;
    mul2(SG, SG, sqh1, sqh2, &g1, &g2);
    const T a1 = un1 - g1, a2 = un2 - g2, b1 = un1 + g1, b2 = un2 + g2;
    const bool fix0 = a1 < T(0) && a2 > T(0), fix2 = b1 < T(0) && b2 > T(0);
    fixed = fix0 || fix2;
    if (fixed) {
      if (fix0) {
        const T t = div_rare(a1 * (a2 - lam0), a2 - a1);
        lamE0 = lam0 - t;
        lam0 = t;
      }
      if (fix2) {
        const T t = div_rare(b2 * (lam2 - b1), b2 - b1);
        lamE2 = lam2 - t;
        lam2 = t;
      }
    }
  }

  // eigenvector components (row 0 and row 2 have a leading 1, row 1 a 0)
  // (components that are zero for this face direction are never used)
  const T r01 = XFACE ? u12 - c12 : u12, r02 = XFACE ? v12 : v12 - c12;
  const T r21 = XFACE ? u12 + c12 : u12, r22 = XFACE ? v12 : v12 + c12;

  // wave strengths
  const T dqx = c2.qx - c1.qx, dqy = c2.qy - c1.qy;
  T udh, vdh, aq, al1;
  mul2(dh, dh, u12, v12, &udh, &vdh);
  const T dx1 = dqx - udh, dy1 = dqy - vdh;
  quot2<L64>(n_dot<T, XFACE>(dx1, dy1), n_cross<T, XFACE>(dx1, dy1), c12, rc12, &aq, &al1);
  T al0, al2;
  mul2(T(0.5), T(0.5), dh - aq, dh + aq, &al0, &al2);

  // upwinded bed-step source, limited where the step is higher than the water
  T dz;
  bool above1, above2;  // z1 + h1 < z2, z2 + h2 < z1
  if (sizeof(T) == 8) {
    const T z1 = c1.z, z2 = c2.z;
    dz = z2 - z1;
    above1 = z1 + h1 < z2;
    above2 = z2 + h2 < z1;
  } else {
    // FP32 form: the bed step from both cells' bases and offsets, so
    // every evaluation of a face gets the same value (a face on a tile edge
    // is evaluated by both tiles, and mass is conserved only if both agree)
    dz = c2.z - c1.z;
    if (cross) dz = (T)(dzb + ((double)c2.z - (double)c1.z));
    above1 = h1 < dz;
    above2 = h2 < -dz;
  }
  T dzp = dz, hp;
  if (dz >= T(0)) {
    hp = h1;
    if (above1) dzp = h1;
  } else {
    hp = h2;
    if (above2) dzp = -h2;
  }
  T be0 = quot<L64>(T(0.5) * G * (hp - T(0.5) * dev_fabs(dzp)) * dzp, c12, rc12);

  // Waves 0, 1 and 2 with eigenvectors (1, r01, r02), (0, -c12 ny, c12 nx) and
  // (1, r21, r22) go to the neighbour's side (q) where their speed is
  // positive, else to the owner's (p).  Plain faces - subcritical, no entropy
  // fix, no dry cell - are nearly all: they send one acoustic wave each way and
  // are done in one short block without the terms that are zero there (flux
  // launch of rain on 1531x2049, FP64: 157 -> 148 us; on 4096^2, FP32: 448 ->
  // 404 us).
  T p0, p1, p2, q0, q1, q2;
  hp = h1 + al0;
  if (!brink && !fixed && lam0 < T(0) && lam2 > T(0)) {
    {  // positivity limiter
      const T lo = al0 * lam0 - c1.hd, hi = -al2 * lam2 + c2.hd;
      const bool limit = hp > T(0);
      if constexpr (L64) {  // be0 is NaN only over beds that are no numbers, which the callers catch
        be0 = limit && lo > be0 ? lo : be0;
        be0 = limit && hi < be0 ? hi : be0;
      } else {
        const T b = dev_fmin(dev_fmax(be0, lo), hi);
        be0 = limit ? b : be0;
      }
    }
    const T w1 = lam1 * al1, t = XFACE ? w1 * c12 : w1 * -c12;
    T w0, w2;
    mul2(lam0, lam2, al0, al2, &w0, &w2);
    p0 = w0 - be0;
    q0 = w2 + be0;
    mul2(r01, r21, p0, q0, &p1, &q1);
    mul2(r02, r22, p0, q0, &p2, &q2);
    if (lam1 > T(0)) {
      if (XFACE) q2 = t + q2; else q1 = t + q1;
    } else {
      if (XFACE) p2 = p2 + t; else p1 = p1 + t;
    }
  } else {
    if (lam0 * lam2 < T(0) && hp > T(0) && h1 > T(0) && h2 > T(0)) {
      T lo = al0 * lam0 - c1.hd, hi = -al2 * lam2 + c2.hd;
      if (fixed) {
        // lam/(lam + lamE) is exactly 1 without an entropy-fix part (lam != 0 here)
        const T f0 = lamE2 == T(0) ? T(1) : div_rare(lam0, lam0 + lamE2);
        const T f2 = lamE0 == T(0) ? T(1) : div_rare(lam2, lam2 + lamE0);
        lo = f0 * (lo + lamE2 * h2);
        hi = f2 * (hi + lamE0 * h1);
      }
      be0 = dev_fmax(be0, lo);
      be0 = dev_fmin(be0, hi);
    }
    const T be2 = -be0;
    const T w0 = lam0 * al0 - be0, w1 = lam1 * al1, w2 = lam2 * al2 - be2;
    // intermediate states decide whether mass is redirected from a dry side;
    // they only matter next to a dry cell, so they are formed only there.  The
    // rest is sorted wave by wave: by branches in FP64, by selections in FP32,
    // where a selection is one instruction.
    if (sizeof(T) == 4) {
      const bool right0 = lam0 > T(0), right2 = lam2 > T(0);
      const T x1 = w0 * r01, x2 = w0 * r02, y1 = w2 * r21, y2 = w2 * r22;
      const T t = XFACE ? w1 * c12 : w1 * -c12;
      p0 = (right0 ? T(0) : w0) + (right2 ? T(0) : w2);
      q0 = (right0 ? w0 : T(0)) + (right2 ? w2 : T(0));
      p1 = right0 ? T(0) : x1;
      p2 = right0 ? T(0) : x2;
      q1 = right0 ? x1 : T(0);
      q2 = right0 ? x2 : T(0);
      if (lam1 > T(0)) {
        if (XFACE) q2 += t; else q1 += t;
      } else {
        if (XFACE) p2 += t; else p1 += t;
      }
      p1 += right2 ? T(0) : y1;
      p2 += right2 ? T(0) : y2;
      q1 += right2 ? y1 : T(0);
      q2 += right2 ? y2 : T(0);
      if (brink) {
        const bool dry2 = h2 < E12 && hp + div_rare(be2, lam2) < -E12;
        const bool dry1 = !dry2 && h1 < E12 && hp - div_rare(be0, lam0) < -E12;
        if (dry1 || dry2) {
          const T m = w0 + w2;
          p0 = dry2 ? m : T(0);
          q0 = dry2 ? T(0) : m;
          p1 = p2 = q1 = q2 = T(0);
        }
      }
    } else {
      p0 = p1 = p2 = q0 = q1 = q2 = T(0);
      if (h2 < E12 && hp + div_rare(be2, lam2) < -E12) {
        p0 += w0 + w2;
      } else if (h1 < E12 && hp - div_rare(be0, lam0) < -E12) {
        q0 += w0 + w2;
      } else {
        if (lam0 > T(0)) {
          q0 += w0;
          q1 += w0 * r01;
          q2 += w0 * r02;
        } else {
          p0 += w0;
          p1 += w0 * r01;
          p2 += w0 * r02;
        }
        if (lam1 > T(0)) {
          if (XFACE) q2 += w1 * c12; else q1 += w1 * -c12;
        } else {
          if (XFACE) p2 += w1 * c12; else p1 += w1 * -c12;
        }
        if (lam2 > T(0)) {
          q0 += w2;
          q1 += w2 * r21;
          q2 += w2 * r22;
        } else {
          p0 += w2;
          p1 += w2 * r21;
          p2 += w2 * r22;
        }
      }
    }
    // entropy-fix parts (a wave without a fix contributes zeros; lamE1 is zero)
    if (lamE0 != T(0)) {
      const T w = lamE0 * al0;
      if (lamE0 > T(0)) {
        q0 += w * T(1);
        q1 += w * r01;
        q2 += w * r02;
      } else {
        p0 += w * T(1);
        p1 += w * r01;
        p2 += w * r02;
      }
    }
    if (lamE2 != T(0)) {
      const T w = lamE2 * al2;
      if (lamE2 > T(0)) {
        q0 += w * T(1);
        q1 += w * r21;
        q2 += w * r22;
      } else {
        p0 += w * T(1);
        p1 += w * r21;
        p2 += w * r22;
      }
    }
  }
  // flush tiny contributions, then scale to depth/discharge increments
  T th0 = E12;
  const T th1 = E12;
  if (sizeof(T) == 4) {
    // FP32 form: a mass contribution within the rounding noise of the terms
    // that formed it is noise.  1e-12 lies far above FP64 noise but far below
    // FP32 noise: at a shoreline the fluctuation into a dry cell cancels to
    // FP32 noise (~1e-9), which would leave 1e-11 m of water there, make the
    // cell count as wet and let water climb the bank.  (Momentum
    // contributions keep the absolute threshold only: zeroing those below
    // the noise of their terms deleted slow flows out of deep water every
    // step, and the FP32 run drained 2-5x further from FP64 in volume.)
    T s0 = dev_fabs(lam0 * al0) + dev_fabs(be0) + dev_fabs(lam2 * al2);
    if (fixed) s0 = s0 + dev_fabs(lamE0 * al0) + dev_fabs(lamE2 * al2);
    th0 = dev_fmax(E12, T(kNoise32) * s0);
  }
  if (sizeof(T) == 4 && th0 > E12) {
    // FP32 form: a mass contribution that is noise moves to the other side
    // instead of vanishing, so the face still conserves mass; the dry side of
    // a shoreline face gets exactly nothing
    const bool np = dev_fabs(p0) < th0, nq = dev_fabs(q0) < th0;
    if (nq && (!np || h1 >= h2)) {  // both noise: to the side with more water
      p0 += q0;
      q0 = T(0);
    } else if (np) {
      q0 += p0;
      p0 = T(0);
    }
  }
  if (dev_fabs(p0) < E12) p0 = T(0);
  if (dev_fabs(q0) < E12) q0 = T(0);
  if (dev_fabs(p1) < th1) p1 = T(0);
  if (dev_fabs(q1) < th1) q1 = T(0);
  if (dev_fabs(p2) < th1) p2 = T(0);
  if (dev_fabs(q2) < th1) q2 = T(0);
  // rhs = dt*p/dx (kernels_flux.h:267-273); dt*p is +0 or at least dt*1e-12
  if (sizeof(T) == 4 || K.dx_pow2) {  // uniform over the launch; in FP32 a / dx is a * rdx for any dx
    const T s = K.rdx;
    mul2(dt, dt, p0, q0, &p0, &q0);
    mul2(dt, dt, p1, q1, &p1, &q1);
    mul2(dt, dt, p2, q2, &p2, &q2);
    mul2(s, s, p0, q0, &out.a0, &out.b0);
    mul2(s, s, p1, q1, &out.a1, &out.b1);
    mul2(s, s, p2, q2, &out.a2, &out.b2);
  } else {
    out.a0 = div_nz(dt * p0, dx, K.rdx);
    out.a1 = div_nz(dt * p1, dx, K.rdx);
    out.a2 = div_nz(dt * p2, dx, K.rdx);
    out.b0 = div_nz(dt * q0, dx, K.rdx);
    out.b1 = div_nz(dt * q1, dx, K.rdx);
    out.b2 = div_nz(dt * q2, dx, K.rdx);
  }
  return out;
}

}  // namespace tri
