// The refinement's kernels (tnc_svd_refine.cuh) for rows in double-float without an
// accumulator: the finish of the sweep's bond cores.  Products and sums keep their
// rounding errors in FP32 (about 12 operations a term: TwoProd by FMA, TwoSum), so
// the FP64 pipe, which issues one FP32 operation's worth in 64 cycles, is left to
// the n^2 entries of the Gram matrix.
#pragma once
#include "tnc_df.cuh"
#include "tnc_svd_refine.cuh"

namespace tnc {

template <typename Tdf> struct df_parts;
template <> struct df_parts<dfr> { typedef float S; typedef double D; };
template <> struct df_parts<dfc> { typedef c64 S; typedef c128 D; };
__device__ __forceinline__ float df_hi(dfr v) { return v.h; }
__device__ __forceinline__ float df_lo(dfr v) { return v.l; }
__device__ __forceinline__ c64 df_hi(dfc v) { return c64(v.re.h, v.im.h); }
__device__ __forceinline__ c64 df_lo(dfc v) { return c64(v.re.l, v.im.l); }
__device__ __forceinline__ double df_value(dfr v) { return to_double(v); }
__device__ __forceinline__ c128 df_value(dfc v) { return c128(to_double(v.re), to_double(v.im)); }
__device__ __forceinline__ void df_set(dfr& v, double x) { v = dfr(x); }
__device__ __forceinline__ void df_set(dfc& v, c128 x) {
  v.re = dfr(x.re);
  v.im = dfr(x.im);
}

// (s, c) += (xh + xl) conj(yh + yl)
__device__ __forceinline__ void df_dot(float& s, float& c, float xh, float xl, float yh, float yl) {
  dot2_acc(s, c, xh, xl, yh, yl);
}
__device__ __forceinline__ void df_dot(c64& s, c64& c, c64 xh, c64 xl, c64 yh, c64 yl) {
  dot2_acc(s.re, c.re, xh.re, xl.re, yh.re, yl.re);
  dot2_acc(s.re, c.re, xh.im, xl.im, yh.im, yl.im);
  dot2_acc(s.im, c.im, xh.im, xl.im, yh.re, yl.re);
  dot2_acc(s.im, c.im, -xh.re, -xl.re, yh.im, yl.im);
}
__device__ __forceinline__ double df_sum(float s, float c) { return (double)s + (double)c; }
__device__ __forceinline__ c128 df_sum(c64 s, c64 c) { return c128(df_sum(s.re, c.re), df_sum(s.im, c.im)); }

// (s, c) += f (h + l)
__device__ __forceinline__ void df_axpy(float& s, float& c, float f, float h, float l) {
  const float p = __fmul_rn(f, h), e = __fmaf_rn(f, h, -p);
  float t;
  two_sum(s, p, s, t);
  c = __fadd_rn(c, __fadd_rn(t, e));
  c = __fmaf_rn(f, l, c);
}
__device__ __forceinline__ void df_axpy(c64& s, c64& c, c64 f, c64 h, c64 l) {
  df_axpy(s.re, c.re, f.re, h.re, l.re);
  df_axpy(s.re, c.re, -f.im, h.im, l.im);
  df_axpy(s.im, c.im, f.re, h.im, l.im);
  df_axpy(s.im, c.im, f.im, h.re, l.re);
}
// x + (s + c)
__device__ __forceinline__ dfr df_plus(dfr x, float s, float c) { return df_add(x, df_norm(s, c)); }
__device__ __forceinline__ dfc df_plus(dfc x, c64 s, c64 c) {
  x.re = df_add(x.re, df_norm(s.re, c.re));
  x.im = df_add(x.im, df_norm(s.im, c.im));
  return x;
}

// G(i, k) = <w_i, w_k> for i < k, the diagonal to a; 32 x 32 tiles on or above the
// diagonal, 2 x 2 outputs a thread.  Bound by the FP32 pipe.  (As an FP64 product it
// kept the whole chip's FP64 pipe busy for 480 us at 512 rows of 512 complex64
// elements: the finish took 1.5 ms instead of 1.0, and twelve sweeps at a time 13 %
// more.)
constexpr int kDfTile = 32, kDfK = 16;
template <typename Tdf>
__global__ void __launch_bounds__(256)
df_gram_kernel(int64_t n, int64_t K, const Tdf* __restrict__ W, typename df_parts<Tdf>::D* __restrict__ G,
               double* __restrict__ a, const RefineState* st, int upto, float accept, unsigned* rows_large) {
  typedef typename df_parts<Tdf>::S S;
  __shared__ Tdf xs[kDfTile][kDfK + 1], ys[kDfTile][kDfK + 1];
  if (refine_done(st, upto, accept) || refine_hard(st, upto)) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    rows_large[i] = 0;
  int64_t t = blockIdx.x, cb = 0;  // column cb has cb + 1 tiles
  while (t > cb) t -= ++cb;
  const int64_t m0 = t * kDfTile, n0 = cb * kDfTile;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  S s[2][2], c[2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) s[i][j] = c[i][j] = zero_<S>();
  for (int64_t k0 = 0; k0 < K; k0 += kDfK) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = ty + 16 * h;
      const bool in = k0 + tx < K;
      Tdf z = {};
      xs[r][tx] = in && m0 + r < n ? W[(m0 + r) * K + k0 + tx] : z;
      ys[r][tx] = in && n0 + r < n ? W[(n0 + r) * K + k0 + tx] : z;
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < kDfK; ++k) {
      S xh[2], xl[2], yh[2], yl[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const Tdf x = xs[ty + 16 * i][k], y = ys[tx + 16 * i][k];
        xh[i] = df_hi(x);
        xl[i] = df_lo(x);
        yh[i] = df_hi(y);
        yl[i] = df_lo(y);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) df_dot(s[i][j], c[i][j], xh[i], xl[i], yh[j], yl[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int64_t gi = m0 + ty + 16 * i, gk = n0 + tx + 16 * j;
      if (gi > gk || gk >= n) continue;
      const auto v = df_sum(s[i][j], c[i][j]);
      if (gi == gk) a[gi] = real_(v);
      else G[gi * n + gk] = v;
    }
}

// W += F W + F F W / 2: I + F + F^2 / 2 is unitary to |F|^4, and F W is summed as
// exactly as W is held (F may reach 1e-3, and FP32 sums would leave 6e-8 of that
// in the singular values).  In place by columns: a CTA keeps C columns of W in
// shared memory and a thread takes up to four rows of the result (n <= 1024),
// reading F^T along them.
template <typename Tdf, int C>
__global__ void __launch_bounds__(256)
df_rotate_kernel(int64_t n, int64_t cols, const typename df_parts<Tdf>::S* __restrict__ Ft, Tdf* __restrict__ W,
                 const RefineState* st, int step, float accept) {
  typedef typename df_parts<Tdf>::S S;
  extern __shared__ __align__(16) unsigned char df_smem[];
  S* h = reinterpret_cast<S*>(df_smem);  // [n][C] high parts
  S* l = h + n * C;                      // low parts
  if (refine_idle(st, step, accept) || refine_hard(st, step + 1)) return;
  const int64_t c0 = (int64_t)blockIdx.x * C;
  for (int64_t e = threadIdx.x; e < n * C; e += blockDim.x) {
    const int64_t i = e / C, c = c0 + e % C;
    Tdf v = {};
    if (c < cols) v = W[i * cols + c];
    h[e] = df_hi(v);
    l[e] = df_lo(v);
  }
  __syncthreads();
  S z[4][C];  // F W / 2
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t i = threadIdx.x + 256 * r;
#pragma unroll
    for (int c = 0; c < C; ++c) z[r][c] = zero_<S>();
    if (i >= n) continue;
#pragma unroll 8
    for (int64_t k = 0; k < n; ++k) {
      const S f = 0.5f * Ft[k * n + i];
#pragma unroll
      for (int c = 0; c < C; ++c) fma_(z[r][c], f, h[k * C + c]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t i = threadIdx.x + 256 * r;
    if (i >= n) continue;
#pragma unroll
    for (int c = 0; c < C; ++c) l[i * C + c] = l[i * C + c] + z[r][c];  // the small part joins the low one
  }
  __syncthreads();
#pragma unroll 1
  for (int64_t i = threadIdx.x; i < n; i += 256) {
    S acc[C], err[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = err[c] = zero_<S>();
#pragma unroll 4
    for (int64_t k = 0; k < n; ++k) {
      const S f = Ft[k * n + i];
#pragma unroll
      for (int c = 0; c < C; ++c) df_axpy(acc[c], err[c], f, h[k * C + c], l[k * C + c]);
    }
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (c0 + c < cols) W[i * cols + c0 + c] = df_plus(W[i * cols + c0 + c], acc[c], err[c]);
  }
}

// The rotations of large angle whose rows have no other, in FP64: a warp takes the
// pair of its row.
template <typename Tdf>
__global__ void df_pairs_kernel(int64_t n, int64_t cols, const typename df_parts<Tdf>::D* __restrict__ G,
                                const double* __restrict__ a, Tdf* __restrict__ W, const RefineState* st, int step,
                                float accept, const unsigned* __restrict__ rows_large,
                                const unsigned* __restrict__ partner) {
  typedef typename df_parts<Tdf>::D D;
  if (refine_idle(st, step, accept) || refine_hard(st, step + 1)) return;
  const int lane = threadIdx.x & 31;
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n;
       i += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    if (rows_large[i] != 1) continue;
    const int64_t k = partner[i];
    if (k <= i || rows_large[k] != 1) continue;
    const D g = G[i * n + k];
    const double h = abs_(g), tau = (a[k] - a[i]) / (2 * h);
    const double t = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
    const double c = 1.0 / sqrt(1.0 + t * t), s = c * t;
    const D se = s * div_real_(g, h);
    Tdf *x = W + i * cols, *y = W + k * cols;
    for (int64_t e = lane; e < cols; e += 32) {
      const D xv = df_value(x[e]), yv = df_value(y[e]);
      df_set(x[e], c * xv - se * yv);
      df_set(y[e], conj_(se) * xv + c * yv);
    }
  }
}

}  // namespace tnc
