// The rotation of a pair of rows in the one-sided Jacobi kernels.
#pragma once
#include "tnc_common.cuh"

namespace tnc {

template <typename T>
struct Rot {
  typename traits<T>::real c, th;  // th = t |g|: the norms move to a - th, b + th
  T se, sec;
  bool apply;
  bool big;  // |g| > stol sqrt(a b): above the stage-stop tolerance
};

// Jacobi rotation from the 2x2 Gram entries (see tnc_svd.cu for the formula)
template <typename T>
__device__ __forceinline__ Rot<T> make_rot_ieee(typename traits<T>::real a, typename traits<T>::real b, T g,
                                                typename traits<T>::real rtol, typename traits<T>::real noise2,
                                                typename traits<T>::real stol) {
  typedef typename traits<T>::real R;
  Rot<T> r;
  const R h = abs_(g);
  const R sab = sqrt(a) * sqrt(b);
  // rows at the rounding-noise floor (or whose squared norm underflowed) count as converged
  r.apply = (a > noise2) && (b > noise2) && (a > 0) && (b > 0) && (h > rtol * sab);
  r.big = r.apply && h > stol * sab;
  if (!r.apply) { r.c = 1; r.th = 0; r.se = zero_<T>(); r.sec = zero_<T>(); return r; }
  const R tau = (b - a) / (2 * h);
  R t;
  if (fabs(tau) > (R)1e15) t = (R)0.5 / tau;
  else t = (tau >= 0 ? R(1) : R(-1)) / (fabs(tau) + sqrt(R(1) + tau * tau));
  r.c = R(1) / sqrt(R(1) + t * t);
  r.th = t * h;
  const R s = r.c * t;
  const R inv_h = R(1) / h;  // one division for both parts of e = g / |g|
  const T e = isfinite(inv_h) ? g * inv_h : div_real_(g, h);
  r.se = s * e;
  r.sec = s * conj_(e);
  return r;
}

// The same rotation for single-precision rows with a short dependency chain (it
// is on the critical path of every Jacobi step: square roots, reciprocals and a
// division in their IEEE forms took about 1,080 cycles of a 2,800-cycle step).
// With z = (b - a) / 2 and w = sign(z) / (|z| + sqrt(z^2 + |g|^2)):  t = |g| w,
// so neither |g| nor 1 / |g| is needed:  t |g| = |g|^2 w,  s e = c w g,
// c = 1 / sqrt(1 + |g|^2 w^2).  w may carry the hardware estimates' error (the
// angle is off by 1e-7 of itself, and the next sweep sees that), c may not: a
// rotation with a biased c^2 + s^2 drifts the norms.  c is the estimate y of
// 1 / sqrt(q) and one step of Newton's method for y^-2 = q, y + y (1 - q y^2) / 2
// (q y rounded, the residual and the last operation fused): below an ulp off, its
// mean about zero.
// Operands whose squares or products leave the comfortable FP32 range take the
// IEEE formula.
__device__ __forceinline__ float fast_rsqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <typename T>
__device__ __forceinline__ Rot<T> make_rot(typename traits<T>::real a, typename traits<T>::real b, T g,
                                           typename traits<T>::real rtol, typename traits<T>::real noise2,
                                           typename traits<T>::real stol = 0) {
  typedef typename traits<T>::real R;
  if constexpr (sizeof(R) != 4) {
    return make_rot_ieee<T>(a, b, g, rtol, noise2, stol);
  } else {
    const float h2 = abs2_(g), ab = a * b, z = 0.5f * (b - a);
    if (!(h2 > 1e-30f && h2 < 1e30f && ab > 1e-30f && ab < 1e30f && fabsf(z) < 1e15f))
      return make_rot_ieee<T>(a, b, g, rtol, noise2, stol);
    Rot<T> r;
    r.apply = (a > noise2) && (b > noise2) && (h2 > (rtol * rtol) * ab);
    r.big = r.apply && h2 > (stol * stol) * ab;
    if (!r.apply) { r.c = 1; r.th = 0; r.se = zero_<T>(); r.sec = zero_<T>(); return r; }
    const float r2 = fmaf(z, z, h2);
    const float w = copysignf(fast_rcp(fmaf(r2, fast_rsqrt(r2), fabsf(z))), z);
    r.th = h2 * w;
    const float q = fmaf(r.th, w, 1.f);
    const float y = fast_rsqrt(q);
    const float e = fmaf(-q * y, y, 1.f);
    const float c = fmaf(0.5f * y, e, y);
    r.c = c;
    const float cw = c * w;
    r.se = cw * g;
    r.sec = cw * conj_(g);
    return r;
  }
}

}  // namespace tnc
