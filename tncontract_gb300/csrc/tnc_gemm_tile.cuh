// The output tile of the CUDA-core GEMM (tnc_gemm.cu), and of the products of
// the SVD refinement (tnc_svd_refine.cuh).
#pragma once
#include "tnc_common.cuh"

namespace tnc {

template <typename T>
__device__ __forceinline__ T maybe_conj(T v, bool c) { return c ? conj_(v) : v; }

// four consecutive elements of a 16-byte-aligned shared-memory row
__device__ __forceinline__ void lds4(const float* p, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void lds4(const c64* p, c64 (&v)[4]) {
  const float4 q0 = reinterpret_cast<const float4*>(p)[0], q1 = reinterpret_cast<const float4*>(p)[1];
  v[0] = c64(q0.x, q0.y); v[1] = c64(q0.z, q0.w); v[2] = c64(q1.x, q1.y); v[3] = c64(q1.z, q1.w);
}

// Output tile BM x BN of a CTA, TM x TN of it a thread, K slices of BK.
// FP32 threads take 4 x 4 consecutive outputs (16-byte shared-memory loads feed
// the FMAs).  FP64 ones take outputs BM / TM rows and BN / TN columns apart: an
// FP64 instruction holds a scheduler for 64 cycles, so loads are free beside it
// and any tile runs at the pipe's rate; only the balance over the SMs counts.
template <typename T, int BM_, int BN_, int TM_, int TN_>
struct GemmTile {
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_;
  static constexpr int THR = (BM / TM) * (BN / TN);
  static constexpr bool WIDE = sizeof(typename traits<T>::real) == 8;
  static constexpr int BK = 16;
  static constexpr int PAD = WIDE ? 1 : 16 / (int)sizeof(T);  // FP32 rows stay 16-byte aligned
  static constexpr int LDA = BM + PAD, LDB = BN + PAD;
  static constexpr int PA = BM * BK / THR, PB = BN * BK / THR;  // tile elements each thread moves
};
template <typename T> using Tile64 = GemmTile<T, 64, 64, 4, 4>;  // FP32
template <typename T> using Tile32 = GemmTile<T, 32, 32, 4, 4>;  // FP32, narrow products, K split over a cluster
template <typename T> using TileL = GemmTile<T, 32, 32, 4, 2>;   // FP64, 128 threads each
template <typename T> using TileM = GemmTile<T, 16, 16, 2, 1>;
template <typename T> using TileS = GemmTile<T, 8, 16, 1, 1>;

// Fetch the BK-slice at k0 of a BR-row operand tile into registers.
// KMAJOR: element (r, k) at X[r * ld + k] (lanes run along k);
// else:   element (r, k) at X[k * ld + r] (lanes run along r).
template <typename T, int BR, int BK, int THR, bool KMAJOR, int PER>
__device__ __forceinline__ void tile_fetch(const T* __restrict__ X, int64_t ld, int64_t r0, int64_t R, int64_t k0,
                                           int64_t K, T (&v)[PER]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    int r, k;
    if (KMAJOR) { k = t % BK; r = t / BK + (THR / BK) * j; }
    else { r = t % BR; k = t / BR + (THR / BR) * j; }
    const int64_t gr = r0 + r, gk = k0 + k;
    v[j] = (gr < R && gk < K) ? (KMAJOR ? X[gr * ld + gk] : X[gk * ld + gr]) : zero_<T>();
  }
}

template <typename T, int BR, int BK, int LD, int THR, bool KMAJOR, int PER>
__device__ __forceinline__ void tile_store(T* s, const T (&v)[PER], bool cj) {
  const int t = threadIdx.x;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    int r, k;
    if (KMAJOR) { k = t % BK; r = t / BK + (THR / BK) * j; }
    else { r = t % BR; k = t / BR + (THR / BR) * j; }
    s[k * LD + r] = maybe_conj(v[j], cj);
  }
}

// Row and column in the tile of a thread's output (i, j).
template <typename G> __device__ __forceinline__ int tile_row(int i) {
  const int ty = threadIdx.x / (G::BN / G::TN);
  return G::WIDE ? ty + (G::BM / G::TM) * i : ty * G::TM + i;
}
template <typename G> __device__ __forceinline__ int tile_col(int j) {
  const int tx = threadIdx.x % (G::BN / G::TN);
  return G::WIDE ? tx + (G::BN / G::TN) * j : tx * G::TN + j;
}

// The products of one output tile (rows m0.., columns n0..) of op(A) op(B).  The
// terms of an output are added in the order of k by every tile shape.
template <typename T, typename G, bool AK, bool BKM>
__device__ __forceinline__ void gemm_acc(int64_t M, int64_t N, int64_t K, bool aC, bool bC, const T* __restrict__ Ab,
                                         int64_t lda, const T* __restrict__ Bb, int64_t ldb, int64_t m0, int64_t n0,
                                         T (*As)[G::BK * G::LDA], T (*Bs)[G::BK * G::LDB], T (&acc)[G::TM][G::TN]) {
  constexpr int TM = G::TM, TN = G::TN, BK = G::BK;
  const int tid = threadIdx.x;
  const int tx = tid % (G::BN / TN), ty = tid / (G::BN / TN);
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = zero_<T>();

  T va[G::PA], vb[G::PB];
  auto fetch = [&](int64_t k0) {
    tile_fetch<T, G::BM, BK, G::THR, AK>(Ab, lda, m0, M, k0, K, va);
    tile_fetch<T, G::BN, BK, G::THR, BKM>(Bb, ldb, n0, N, k0, K, vb);
  };
  auto store = [&](int buf) {
    tile_store<T, G::BM, BK, G::LDA, G::THR, AK>(As[buf], va, aC);
    tile_store<T, G::BN, BK, G::LDB, G::THR, BKM>(Bs[buf], vb, bC);
  };
  fetch(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int64_t k0 = 0; k0 < K; k0 += BK) {
    const bool more = k0 + BK < K;
    if (more) fetch(k0 + BK);
    const T* as = As[buf];
    const T* bs = Bs[buf];
    auto step = [&](int kk) {
      T a[TM], b[TN];
      if constexpr (G::WIDE) {
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = as[kk * G::LDA + ty + (G::BM / TM) * i];
#pragma unroll
        for (int j = 0; j < TN; ++j) b[j] = bs[kk * G::LDB + tx + (G::BN / TN) * j];
      } else {
        lds4(as + kk * G::LDA + ty * TM, a);
        lds4(bs + kk * G::LDB + tx * TN, b);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) fma_(acc[i][j], a[i], b[j]);
    };
    const int kn = (K - k0) < BK ? (int)(K - k0) : BK;
    if (!G::WIDE || kn == BK) {
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) step(kk);
    } else {  // no FP64 products with the padding
      for (int kk = 0; kk < kn; ++kk) step(kk);
    }
    if (more) store(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }
}

// One output tile of C = alpha op(A) op(B) + beta C.
template <typename T, typename G, bool AK, bool BKM>
__device__ __forceinline__ void gemm_tile(int64_t M, int64_t N, int64_t K, bool aC, bool bC, T alpha,
                                          const T* __restrict__ Ab, int64_t lda, const T* __restrict__ Bb,
                                          int64_t ldb, T beta, T* __restrict__ Cb, int64_t ldc, int64_t m0,
                                          int64_t n0, T (*As)[G::BK * G::LDA], T (*Bs)[G::BK * G::LDB]) {
  const bool beta_zero = (abs2_(beta) == 0);
  T acc[G::TM][G::TN];
  gemm_acc<T, G, AK, BKM>(M, N, K, aC, bC, Ab, lda, Bb, ldb, m0, n0, As, Bs, acc);
#pragma unroll
  for (int i = 0; i < G::TM; ++i) {
    const int64_t gm = m0 + tile_row<G>(i);
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < G::TN; ++j) {
      const int64_t gn = n0 + tile_col<G>(j);
      if (gn >= N) continue;
      T v = alpha * acc[i][j];
      if (!beta_zero) v += beta * Cb[gm * ldc + gn];
      Cb[gm * ldc + gn] = v;
    }
  }
}

}  // namespace tnc
