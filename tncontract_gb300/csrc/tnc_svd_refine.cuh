// FP64 SVD of the triangular factor R in two precisions: a single-precision
// Jacobi finds the rotations, FP64 products bring them to FP64.
//
// GB300 runs an FP64 instruction of a warp in 64 cycles, an FP32 one in 1, so a
// Jacobi in FP64 is bound by its own scalar chains.  Here the block Jacobi of
// single-precision rows (tnc_jacobi32.cuh) rotates a rounded copy of R and
// accumulates J; then, in FP64, W = J R and a few steps of
//   G = W W^H,  delta = J J^H - I   (half each: one pass over both),
//   J <- (I + F) J,  W = J R,
// where F holds for every pair of rows the rotation that makes them orthogonal
// (all pairs at once: the angles are small) and half the defect delta that makes
// J unitary.  Both defects are squared by a step: 1e-6 after the Jacobi, then
// about 1e-10, then rounding.  F is small, so the products with it run in FP32
// (error 6e-8 |F|, which the next step sees); when it is below 1e-9, W takes its
// correction directly too.  The refinement ends when every pair meets the FP64
// Jacobi's own tolerance; what does not converge (clusters of nearly equal
// values) is left to that Jacobi, which starts from W and J and skips when
// nothing is left.
//
// Graded matrices: the single-precision copy keeps every row to its own relative
// precision, down to the FP64 noise floor, and delta is put on the row of larger
// norm (its component along the smaller one is removed), so that a small row's
// orthogonality to the large ones, which sits in small entries of J, is not
// disturbed by them.
//
// The FP64 Jacobi alone took 4.9 ms of a 64 x 64 float64 SVD's 5.5 and 46 of a
// 256 x 256 complex128 one's 57; the SVDs take 0.7 and 5.3 ms, and reconstruct the
// matrix to 1e-15 instead of 1e-14 to 8e-14 (fewer roundings an entry).
#pragma once
#include "tnc_gemm_tile.cuh"
#include "tnc_persist.cuh"

namespace tnc {

constexpr int kRefineSteps = 4;         // steps at most; one more look decides
constexpr float kRefineDirect = 1e-9f;  // |F| below which W takes F W in FP32
struct RefineState {
  unsigned rot, unit;  // pairs of rows / of J's rows above the tolerance
  unsigned hard;       // pairs whose rotation this step could not take
  float fmax;          // largest |F|
};
// Whether a step before `upto` found nothing to do.  Without J (accept >= 0), also
// whether one took an F below `accept`; a hard one is the last then, and the steps
// after it have not run.
__host__ __device__ __forceinline__ bool refine_done(const RefineState* st, int upto, float accept = -1.f) {
  for (int s = 0; s < upto; ++s) {
    if (st[s].rot == 0 && st[s].unit == 0) return true;
    if (accept >= 0.f && st[s].hard) return false;
    if (st[s].fmax < accept) return true;
  }
  return false;
}
// The same from inside step `step`, after its test.
__host__ __device__ __forceinline__ bool refine_idle(const RefineState* st, int step, float accept = -1.f) {
  return refine_done(st, step, accept) || (st[step].rot == 0 && st[step].unit == 0);
}
// A step with pairs that it cannot rotate leaves them to the FP64 Jacobi: the
// steps after it make J unitary and rotate nothing; without J such a step does
// nothing and is the last.
__host__ __device__ __forceinline__ bool refine_hard(const RefineState* st, int upto) {
  for (int s = 0; s < upto; ++s)
    if (st[s].hard) return true;
  return false;
}

template <typename T> struct narrow_of { typedef float type; };
template <> struct narrow_of<c128> { typedef c64 type; };


// Exponent k with |R|_F about 2^k: the single-precision copy is R 2^-k.
__device__ __forceinline__ int refine_exp(const double* f2) {
  const double f = f2[0];
  return (f > 0.0 && isfinite(f)) ? ilogb(sqrt(f)) : 0;
}
__device__ __forceinline__ float refine_narrow(double v) { return (float)v; }
__device__ __forceinline__ c64 refine_narrow(c128 v) { return c64((float)v.re, (float)v.im); }
__device__ __forceinline__ double refine_ldexp(double v, int k) { return ldexp(v, k); }
__device__ __forceinline__ c128 refine_ldexp(c128 v, int k) { return c128(ldexp(v.re, k), ldexp(v.im, k)); }
__device__ __forceinline__ double refine_widen(float v) { return (double)v; }
__device__ __forceinline__ c128 refine_widen(c64 v) { return c128((double)v.re, (double)v.im); }

// W32 = R 2^(23 - k), J32 = I.  f2[1] is what makes the Jacobi's noise floor
// (eps32^2 f2[1]) that of FP64.  At a norm of 2^23 the squares of every row above
// it, and their products, are FP32 numbers.
constexpr int kRefineLift = 23;
template <typename T>
__global__ void refine_split_kernel(int64_t n, const T* __restrict__ R, typename narrow_of<T>::type* __restrict__ W32,
                                    typename narrow_of<T>::type* __restrict__ J32, double* f2) {
  typedef typename narrow_of<T>::type S;
  const int k = refine_exp(f2);
  if (blockIdx.x == 0 && threadIdx.x == 0) f2[1] = ldexp(f2[0], 2 * (kRefineLift - 29 - k));  // eps64 = 2^-29 eps32
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n * n; e += (int64_t)gridDim.x * blockDim.x) {
    W32[e] = refine_narrow(refine_ldexp(R[e], kRefineLift - k));
    J32[e] = e / n == e % n ? one_<S>() : zero_<S>();
  }
}

template <typename T>
__global__ void refine_widen_kernel(int64_t n2, const typename narrow_of<T>::type* __restrict__ J32, T* __restrict__ J) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n2; e += (int64_t)gridDim.x * blockDim.x)
    J[e] = refine_widen(J32[e]);
}

// W = J R, R upper triangular: column tile n0 needs R's rows up to n0 + BN only.
// The long columns first, so that the short ones fill the last wave.
template <typename T>
__global__ void __launch_bounds__(TileS<T>::THR)
refine_product_kernel(int64_t n, const T* __restrict__ J, const T* __restrict__ R, T* __restrict__ W,
                      const RefineState* st, int upto) {
  typedef TileS<T> G;
  __shared__ __align__(16) T As[2][G::BK * G::LDA];
  __shared__ __align__(16) T Bs[2][G::BK * G::LDB];
  if (refine_done(st, upto) || (upto > 0 && st[upto - 1].fmax < kRefineDirect)) return;
  const int64_t rows = (n + G::BM - 1) / G::BM, cols = (n + G::BN - 1) / G::BN;
  const int64_t m0 = (int64_t)(blockIdx.x % rows) * G::BM, n0 = (cols - 1 - blockIdx.x / rows) * G::BN;
  T acc[G::TM][G::TN];
  const int64_t kk = n0 + G::BN < n ? n0 + G::BN : n;
  gemm_acc<T, G, true, false>(n, n, kk, false, false, J, n, R, n, m0, n0, As, Bs, acc);
  const int64_t gm = m0 + tile_row<G>(0), gn = n0 + tile_col<G>(0);
  if (gm < n && gn < n) W[gm * n + gn] = acc[0][0];
}

// X = W (blockIdx.y = 0) or J (1), n x n: <x_i, x_k> for i < k, G's above the diagonal of GF, delta's below it (at (k, i)); the diagonals
// to a and d.
template <typename T>
__global__ void __launch_bounds__(TileS<T>::THR)
refine_gram_kernel(int64_t n, const T* __restrict__ W, const T* __restrict__ J, T* __restrict__ GF,
                   typename traits<T>::real* __restrict__ a, typename traits<T>::real* __restrict__ d,
                   const RefineState* st, int upto, unsigned* rows_large) {
  typedef TileS<T> G;
  __shared__ __align__(16) T As[2][G::BK * G::LDA];
  __shared__ __align__(16) T Bs[2][G::BK * G::LDB];
  if (refine_done(st, upto)) return;
  if (blockIdx.y == 0)
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
      rows_large[i] = 0;
  // tiles (rb, cb) that reach the diagonal or lie above it: rows rb * 8 <= columns' end
  const int64_t cols = (n + G::BN - 1) / G::BN;
  int64_t t = blockIdx.x, cb = 0;
  for (; cb < cols; ++cb) {  // column cb has min(2 (cb + 1), rows) row tiles
    const int64_t cnt = 2 * (cb + 1), all = (n + G::BM - 1) / G::BM;
    const int64_t have = cnt < all ? cnt : all;
    if (t < have) break;
    t -= have;
  }
  if (cb >= cols) return;
  const int64_t m0 = t * G::BM, n0 = cb * G::BN;
  const T* X = blockIdx.y ? J : W;
  T acc[G::TM][G::TN];
  gemm_acc<T, G, true, true>(n, n, n, false, true, X, n, X, n, m0, n0, As, Bs, acc);
  const int64_t i = m0 + tile_row<G>(0), k = n0 + tile_col<G>(0);
  if (i > k || k >= n) return;
  const T v = acc[0][0];
  if (i == k) {
    if (blockIdx.y) d[i] = real_(v) - typename traits<T>::real(1);
    else a[i] = real_(v);
  } else if (blockIdx.y) {
    GF[k * n + i] = v;
  } else {
    GF[i * n + k] = v;
  }
}

// 2^-2k: the squared norms and products in units of |R|_F^2, where squares and
// products of them neither overflow nor, above the noise floor, underflow.
__device__ __forceinline__ double refine_scale2(const double* f2) {
  const int k = refine_exp(f2);
  return ldexp(1.0, k > -500 ? -2 * k : 1000);
}

// The pair's rotation x' = x - f y, y' = y + conj(f) x after the defect of J is put
// right (f = t e, e = g / |g|), and the tangent t; large: an angle above 1e-3.  a
// and b are the norms with J's defect taken out: two rows of one singular value
// then differ by second-order terms only, and their inner product is second order
// too, so a pair below `skip` (relative) is left as it is.  Only the differences
// need FP64: f may be off by 1e-7 of itself.  Scaled values; everything is taken
// relative to the larger row, so that FP32's range holds it (what underflows is
// below the tolerance).
template <typename S>
struct RefinePair {
  S f;
  float t;
  bool large;
};
template <typename T>
__device__ __forceinline__ RefinePair<typename narrow_of<T>::type> refine_pair(T g, T dl, double a, double b,
                                                                               double noise2, float skip) {
  typedef typename narrow_of<T>::type S;
  RefinePair<S> r;
  r.f = zero_<S>();
  r.t = 0.f;
  r.large = false;
  if (!(a > noise2 && b > noise2)) return r;
  const S gt = refine_narrow(g - dl * (a < b ? a : b));
  const float af = (float)a, bf = (float)b, m = 1.f / fmaxf(af, bf);
  const S gr = gt * m;
  const float zr = (float)(0.5 * (b - a)) * m, h2 = abs2_(gr);
  const float w = copysignf(1.f / (fabsf(zr) + sqrtf(fmaf(zr, zr, h2))), zr);
  if (!(h2 > skip * skip * (fminf(af, bf) * m)) || !isfinite(w)) return r;
  r.t = sqrtf(h2) * fabsf(w);
  r.f = gr * w;
  r.large = r.t > 1e-3f;
  return r;
}
// Relative inner products that a step leaves alone: half the tolerance, and with J
// the second order of the Jacobi's 1e-6 at first.
template <bool HASJ>
__device__ __forceinline__ float refine_skip(int step, double tol) {
  return HASJ && step == 0 ? 1e-9f : 0.5f * (float)tol;
}

// Whether a pair is above the tolerance (scaled squared norms and product).
template <typename T>
__device__ __forceinline__ bool refine_above(T g, double a, double b, double noise2, double tol2) {
  return a > noise2 && b > noise2 && abs2_(g) > tol2 * (a * b);
}

// Counts of the pairs above the tolerances, and for every row its pairs with a
// large angle (and its partner in the last).  A thread takes a pair i < k.  J is held to
// utol, rounding, whatever the caller's tolerance: U and VH are as unitary as J, and
// the singular values are second order in tol only if it is.  Without J, delta is
// nothing and d is not read.  Pairs of two rows from nkeep on are left alone.
template <typename T, bool HASJ>
__global__ void refine_test_kernel(int64_t n, const T* __restrict__ GF, const typename traits<T>::real* __restrict__ a,
                                   const typename traits<T>::real* __restrict__ d, const double* frob2, double tol,
                                   double utol, double eps, int64_t nkeep, RefineState* st, int step, float accept,
                                   unsigned* rows_large, unsigned* partner) {
  if (refine_done(st, step, accept) || (!HASJ && refine_hard(st, step))) return;
  const double sc = refine_scale2(frob2), noise2 = eps * eps * frob2[0] * sc, tol2 = tol * tol, utol2 = 16.0 * utol * utol;
  const float skip = refine_skip<HASJ>(step, tol);
  unsigned rot = 0, unit = 0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n * n; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / n, k = e - i * n;
    if (i > k) continue;
    if (i == k) {
      if (HASJ) unit += d[i] * d[i] > utol2;
      continue;
    }
    if (i >= nkeep) continue;
    const T g = GF[i * n + k] * sc, dl = HASJ ? GF[k * n + i] : zero_<T>();
    const double ai = a[i] * sc, ak = a[k] * sc, di = HASJ ? d[i] : 0.0, dk = HASJ ? d[k] : 0.0;
    if (HASJ) unit += abs2_(dl) > utol2;
    if (refine_above<T>(g, ai, ak, noise2, tol2)) {
      ++rot;
      if (refine_pair<T>(g, dl, ai - ai * di, ak - ak * dk, noise2, skip).large) {
        // two in a row: the simultaneous rotations do not hold for them
        const unsigned before = atomicAdd(&rows_large[i], 1u) + atomicAdd(&rows_large[k], 1u);
        if (before) atomicOr(&st[step].hard, 1u);
        if (partner) {  // read only where a row has one
          partner[i] = (unsigned)k;
          partner[k] = (unsigned)i;
        }
      }
    }
  }
  if (rot) atomicAdd(&st[step].rot, rot);
  if (unit) atomicAdd(&st[step].unit, unit);
}

// F^T in single precision, Ft[k][i] = F(i, k).  A pair takes its first-order
// rotation, or, when its angle is large, it is above the tolerance and neither row
// has another such pair, the full one (with its part of the diagonal; without J, refine_pairs_kernel does
// it in FP64).  Late steps take small angles only, so that what they leave of J's
// defect is below rounding.
template <typename T, bool HASJ>
__global__ void refine_f_kernel(int64_t n, const T* __restrict__ GF, const typename traits<T>::real* __restrict__ a,
                                const typename traits<T>::real* __restrict__ d, const double* frob2, double tol,
                                double eps, int64_t nkeep, RefineState* st, int step, float accept,
                                const unsigned* __restrict__ rows_large,
                                typename narrow_of<T>::type* __restrict__ Ft) {
  typedef typename narrow_of<T>::type S;
  if (refine_idle(st, step, accept) || (!HASJ && refine_hard(st, step + 1))) return;
  const double sc = refine_scale2(frob2), noise2 = eps * eps * frob2[0] * sc;
  const bool rotate = !refine_hard(st, step);
  const float skip = refine_skip<HASJ>(step, tol), top = step < 2 ? 2.f : step == 2 ? 1e-5f : 1e-7f;
  // a warp takes row i: its own F(i, k) for every k, and F(i, i)
  const int lane = threadIdx.x & 31;
  float fmax2 = 0.f;
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n;
       i += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    const double di = HASJ ? d[i] : 0.0, raw = a[i] * sc, ai = raw - raw * di;
    const unsigned li = rows_large[i];
    float diag = 0.f;
    for (int64_t k = lane; k < n; k += 32) {
      if (k == i) continue;
      const bool up = i < k;  // G above the diagonal, delta below it
      const T g = (up ? GF[i * n + k] : GF[k * n + i]) * sc;
      const T dl = !HASJ ? zero_<T>() : up ? GF[k * n + i] : GF[i * n + k];
      const double rk = a[k] * sc, ak = HASJ ? rk - rk * d[k] : rk;
      S f = zero_<S>();
      if (rotate && (i < nkeep || k < nkeep)) {
        RefinePair<S> r = refine_pair<T>(g, dl, up ? ai : ak, up ? ak : ai, noise2, skip);
        if ((r.large || (HASJ && r.t >= top)) && !refine_above<T>(g, raw, rk, noise2, tol * tol)) {
          r.f = zero_<S>();  // two nearly equal norms that meet the tolerance: the test has not counted the pair
        } else if (!HASJ && r.large && li == 1 && rows_large[k] == 1) {
          r.f = zero_<S>();
          fmax2 = 1.f;  // another look
        } else if (HASJ && r.large && li == 1 && rows_large[k] == 1 && r.t < top) {
          const float c = 1.f / sqrtf(fmaf(r.t, r.t, 1.f));
          diag -= r.t * r.t * c / (1.f + 1.f / c);  // c - 1
          r.f = r.f * c;
        } else if (r.large || (HASJ && r.t >= top)) {
          r.f = zero_<S>();
          atomicOr(&st[step].hard, 1u);
        }
        f = up ? -r.f : conj_(r.f);
      }
      const bool larger = up ? raw >= rk : raw > rk;
      if (HASJ && larger) f = f - refine_narrow(up ? dl : conj_(dl));
      Ft[k * n + i] = f;
      fmax2 = fmaxf(fmax2, abs2_(f));
    }
    diag = warp_sum(diag) - 0.5f * (float)di;
    if (lane == 0) Ft[i * n + i] = S(diag);
    fmax2 = fmaxf(fmax2, diag * diag);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) fmax2 = fmaxf(fmax2, __shfl_xor_sync(0xffffffffu, fmax2, o));
  if (lane == 0) atomicMax(reinterpret_cast<unsigned*>(&st[step].fmax), __float_as_uint(sqrtf(fmax2)));  // not negative
}

// X += F X for X = J (n x n) and, with a small F, W (blockIdx.y = 1), in place by
// columns: a CTA keeps C columns of X (rounded to FP32; W in units of 2^k) in
// shared memory and a thread takes rows of the result, reading F^T along them.
template <typename T, int C>
__global__ void __launch_bounds__(256)
refine_apply_kernel(int64_t n, const typename narrow_of<T>::type* __restrict__ Ft, T* __restrict__ J, T* __restrict__ W,
                    const double* frob2, const RefineState* st, int step) {
  typedef typename narrow_of<T>::type S;
  extern __shared__ __align__(16) unsigned char refine_smem[];
  S* s = reinterpret_cast<S*>(refine_smem);  // [n][C]
  if (refine_idle(st, step) || (blockIdx.y && !(st[step].fmax < kRefineDirect))) return;
  T* X = blockIdx.y ? W : J;
  const int e2 = blockIdx.y ? refine_exp(frob2) : 0;
  const int64_t c0 = (int64_t)blockIdx.x * C;
  for (int64_t e = threadIdx.x; e < n * C; e += blockDim.x) {
    const int64_t i = e / C, c = c0 + e % C;
    s[e] = c < n ? refine_narrow(refine_ldexp(X[i * n + c], -e2)) : zero_<S>();
  }
  __syncthreads();
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    S acc[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = zero_<S>();
#pragma unroll 8
    for (int64_t k = 0; k < n; ++k) {
      const S f = Ft[k * n + i];
#pragma unroll
      for (int c = 0; c < C; ++c) fma_(acc[c], f, s[k * C + c]);
    }
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (c0 + c < n) X[i * n + c0 + c] = X[i * n + c0 + c] + refine_ldexp(refine_widen(acc[c]), e2);
  }
}

// Row tiles of the half that refine_gram_kernel takes.
inline unsigned refine_half_tiles(int64_t n) {
  const int64_t rows = (n + 7) / 8, cols = (n + 15) / 16;
  int64_t half = 0;
  for (int64_t c = 0; c < cols; ++c) half += 2 * (c + 1) < rows ? 2 * (c + 1) : rows;
  return (unsigned)half;
}

}  // namespace tnc
