// Batched GEMM on row-major operands with transpose / conjugate options
// (the product inside np.tensordot, tncontract/tensor.py:735).
//
// CUDA-core tiled kernel: an output tile per CTA (64 x 64 with a 4x4 register
// micro-tile per thread in FP32, smaller ones in FP64), K in slices of BK
// staged in shared memory k-major (so an FP32 thread reads its 4 consecutive
// values of each operand with 16-byte loads).  Two shared-memory buffers: the
// next slice is fetched into registers while the current one is multiplied,
// then stored to the other buffer -- one CTA barrier per slice and the
// global-load latency hidden behind the FMAs.  Whether an operand's contiguous
// axis is K (A: N/R, B: T/C) or M/N (A: T/C, B: N/R) is a template parameter,
// so each tile load is a coalesced, branch-free pattern.  This is the FP64 /
// complex128 path (GB300 runs FP64 on the CUDA cores) and the general path for
// small or odd shapes; FP32-class products that tolerate its digit split can
// use the tcgen05 kernel.
#include "tnc_gemm_tile.cuh"

namespace tnc {

template <typename T, typename G, bool AK, bool BKM>
__global__ void __launch_bounds__(G::THR)
gemm_simt_kernel(int64_t M, int64_t N, int64_t K, bool aC, bool bC, T alpha, const T* __restrict__ A, int64_t lda,
                 int64_t sA, const T* __restrict__ B, int64_t ldb, int64_t sB, T beta, T* __restrict__ C,
                 int64_t ldc, int64_t sC, int64_t batch) {
  __shared__ __align__(16) T As[2][G::BK * G::LDA];
  __shared__ __align__(16) T Bs[2][G::BK * G::LDB];
  const int64_t n0 = (int64_t)blockIdx.x * G::BN;
  for (int64_t bz = blockIdx.z; bz < batch; bz += gridDim.z)
    for (int64_t m0 = (int64_t)blockIdx.y * G::BM; m0 < M; m0 += (int64_t)gridDim.y * G::BM) {
      gemm_tile<T, G, AK, BKM>(M, N, K, aC, bC, alpha, A + bz * sA, lda, B + bz * sB, ldb, beta, C + bz * sC, ldc, m0,
                               n0, As, Bs);
      __syncthreads();  // the next tile reuses the shared tiles
    }
}

// FP32 tile with K split over the S CTAs of a cluster: every CTA multiplies its
// run of K slices, leaves its sums in shared memory (where its slices were), and
// adds up (in the order of K) and writes 1 / S of the tile's rows from all of them.
template <typename T, typename G>
struct SplitSmem {
  static constexpr int A = 2 * G::BK * G::LDA, B = 2 * G::BK * G::LDB;
  static_assert(A + B >= G::BM * G::BN, "the sums lie over the slices");
  T v[A + B];
};
template <typename T, typename G, bool AK, bool BKM>
__device__ __forceinline__ void split_tile(int64_t M, int64_t N, int64_t K, bool aC, bool bC, T alpha, const T* A,
                                           int64_t lda, const T* B, int64_t ldb, T beta, T* C, int64_t ldc, int64_t m0,
                                           int64_t n0, int S, int rank, SplitSmem<T, G>& sm) {
  T(*As)[G::BK * G::LDA] = reinterpret_cast<T(*)[G::BK * G::LDA]>(sm.v);
  T(*Bs)[G::BK * G::LDB] = reinterpret_cast<T(*)[G::BK * G::LDB]>(sm.v + SplitSmem<T, G>::A);
  T* part = sm.v;
  const int64_t slices = (K + G::BK - 1) / G::BK;
  const int64_t k0 = slices * rank / S * G::BK, k1 = slices * (rank + 1) / S * G::BK, kn = (k1 < K ? k1 : K) - k0;
  T acc[G::TM][G::TN];
#pragma unroll
  for (int i = 0; i < G::TM; ++i)
#pragma unroll
    for (int j = 0; j < G::TN; ++j) acc[i][j] = zero_<T>();
  if (kn > 0)
    gemm_acc<T, G, AK, BKM>(M, N, kn, aC, bC, AK ? A + k0 : A + k0 * lda, lda, BKM ? B + k0 : B + k0 * ldb, ldb, m0, n0,
                            As, Bs, acc);
#pragma unroll
  for (int i = 0; i < G::TM; ++i)
#pragma unroll
    for (int j = 0; j < G::TN; ++j) part[tile_row<G>(i) * G::BN + tile_col<G>(j)] = acc[i][j];
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const bool beta_zero = (abs2_(beta) == 0);
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(part);
  const int rows = G::BM / S;
  for (int e = threadIdx.x; e < rows * G::BN; e += G::THR) {
    const int r = rank * rows + e / G::BN, c = e % G::BN;
    const int64_t gm = m0 + r, gn = n0 + c;
    if (gm >= M || gn >= N) continue;
    T sum = zero_<T>();
    for (int q = 0; q < S; ++q) {
      uint32_t at;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(base + (uint32_t)((r * G::BN + c) * sizeof(T))), "r"(q));
      T v;
      if constexpr (traits<T>::is_complex)
        asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.re), "=f"(v.im) : "r"(at) : "memory");
      else
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
      sum += v;
    }
    T v = alpha * sum;
    if (!beta_zero) v += beta * C[gm * ldc + gn];
    C[gm * ldc + gn] = v;
  }
  // no CTA leaves, or starts its next tile, while another reads its sums
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ int split_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return (int)r;
}

template <typename T, typename G, bool AK, bool BKM>
__global__ void __launch_bounds__(G::THR)
gemm_split_kernel(int64_t M, int64_t N, int64_t K, bool aC, bool bC, T alpha, const T* __restrict__ A, int64_t lda,
                  int64_t sA, const T* __restrict__ B, int64_t ldb, int64_t sB, T beta, T* C, int64_t ldc, int64_t sC,
                  int64_t batch, int S) {
  __shared__ __align__(16) SplitSmem<T, G> sm;
  const int64_t n0 = (int64_t)(blockIdx.x / (unsigned)S) * G::BN;
  const int rank = split_rank();
  for (int64_t bz = blockIdx.z; bz < batch; bz += gridDim.z)
    for (int64_t m0 = (int64_t)blockIdx.y * G::BM; m0 < M; m0 += (int64_t)gridDim.y * G::BM)
      split_tile<T, G, AK, BKM>(M, N, K, aC, bC, alpha, A + bz * sA, lda, B + bz * sB, ldb, beta, C + bz * sC, ldc, m0, n0,
                                S, rank, sm);
}

// CTAs of the cluster that splits K when the 64 x 64 tiles would not fill the chip
// (0: they do, or K is too short to split): two slices or more each, and two CTAs
// of 64 x 64 an SM or four of 32 x 32 (the two larger products of a chi = 256,
// D = 3 environment update: 128 us in 32 x 32 tiles, two warps each, 107 in parts of
// 64 x 64 ones, from a cold cache).
template <typename Count>
static int split_of(Count tiles, int64_t k, bool small) {
  if (tiles(64, 64) >= 152) return 0;
  const int64_t t = small ? tiles(32, 32) : tiles(64, 64), most = small ? 152 * 4 : 152 * 2;
  int s = 1;
  while (s < 8 && t * s * 2 <= most && k >= 64 * s) s *= 2;
  return s;
}
// Products with a side of at most 32 take the 32 x 32 tile.
static bool split_small(int64_t m, int64_t n) { return m <= 32 || n <= 32; }

static cudaLaunchConfig_t split_config(dim3 grid, int threads, int S, cudaStream_t st, cudaLaunchAttribute* attr) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = (unsigned)S;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// FP64 tile of a set of products by the time of the busiest SM: tiles are dealt
// to 152 SMs and a tile takes BM BN K / 2 cycles of its SM (four times that in
// complex), so the cost is ceil(tiles / 152) BM BN; the larger tile among equals
// (fewer loads).  One 64 x 64 tile shape left most SMs without work: a 32 x 16 x
// 32 complex128 product took 70 us in one CTA, a 513 x 203 x 291 float64 one 220
// in 45.  ``tiles`` counts the tiles of a shape.
enum { kTileS, kTileM, kTileL };
template <typename Count>
static int wide_tile(Count tiles) {
  const int64_t cl = (tiles(32, 32) + 151) / 152 * 1024, cm = (tiles(16, 16) + 151) / 152 * 256,
                cs = (tiles(8, 16) + 151) / 152 * 128;
  if (cl <= cm && cl <= cs) return kTileL;
  return cm <= cs ? kTileM : kTileS;
}

// Independent products of different shapes in one launch: the CTAs of the
// grid are dealt out to the problems' output tiles (problem q owns tiles
// [tile0_q, tile0_{q+1})), each problem with its own operand layouts.
struct GroupProblem {
  int64_t m, n, k, lda, ldb, ldc, tile0, tiles_n;
  const void* A;
  const void* B;
  void* C;
  double alpha[2], beta[2];
  int opA, opB;
};
constexpr int kGroupMax = 16;
struct GemmGroup {
  int count;
  GroupProblem p[kGroupMax];
};

template <typename T, typename G>
__global__ void __launch_bounds__(G::THR) gemm_grouped_kernel(const __grid_constant__ GemmGroup g) {
  __shared__ __align__(16) T As[2][G::BK * G::LDA];
  __shared__ __align__(16) T Bs[2][G::BK * G::LDB];
  int q = 0;
  while (q + 1 < g.count && (int64_t)blockIdx.x >= g.p[q + 1].tile0) ++q;
  const GroupProblem& P = g.p[q];
  const int64_t t = (int64_t)blockIdx.x - P.tile0;
  const int64_t m0 = (t / P.tiles_n) * G::BM, n0 = (t % P.tiles_n) * G::BN;
  const T alpha = from_pair<T>(P.alpha), beta = from_pair<T>(P.beta);
  const bool aK = (P.opA == TNC_OP_N || P.opA == TNC_OP_R), bK = (P.opB == TNC_OP_T || P.opB == TNC_OP_C);
  const bool aC = (P.opA == TNC_OP_C || P.opA == TNC_OP_R), bC = (P.opB == TNC_OP_C || P.opB == TNC_OP_R);
  const T* A = (const T*)P.A;
  const T* B = (const T*)P.B;
  T* C = (T*)P.C;
  if (aK && bK) gemm_tile<T, G, true, true>(P.m, P.n, P.k, aC, bC, alpha, A, P.lda, B, P.ldb, beta, C, P.ldc, m0, n0, As, Bs);
  else if (aK) gemm_tile<T, G, true, false>(P.m, P.n, P.k, aC, bC, alpha, A, P.lda, B, P.ldb, beta, C, P.ldc, m0, n0, As, Bs);
  else if (bK) gemm_tile<T, G, false, true>(P.m, P.n, P.k, aC, bC, alpha, A, P.lda, B, P.ldb, beta, C, P.ldc, m0, n0, As, Bs);
  else gemm_tile<T, G, false, false>(P.m, P.n, P.k, aC, bC, alpha, A, P.lda, B, P.ldb, beta, C, P.ldc, m0, n0, As, Bs);
}

template <typename T, typename G>
__global__ void __launch_bounds__(G::THR) gemm_grouped_split_kernel(const __grid_constant__ GemmGroup g, int S) {
  __shared__ __align__(16) SplitSmem<T, G> sm;
  const int64_t tile = blockIdx.x / (unsigned)S;
  int q = 0;
  while (q + 1 < g.count && tile >= g.p[q + 1].tile0) ++q;
  const GroupProblem& P = g.p[q];
  const int64_t t = tile - P.tile0;
  const int64_t m0 = (t / P.tiles_n) * G::BM, n0 = (t % P.tiles_n) * G::BN;
  const T alpha = from_pair<T>(P.alpha), beta = from_pair<T>(P.beta);
  const bool aK = (P.opA == TNC_OP_N || P.opA == TNC_OP_R), bK = (P.opB == TNC_OP_T || P.opB == TNC_OP_C);
  const bool aC = (P.opA == TNC_OP_C || P.opA == TNC_OP_R), bC = (P.opB == TNC_OP_C || P.opB == TNC_OP_R);
  const T* A = (const T*)P.A;
  const T* B = (const T*)P.B;
  T* C = (T*)P.C;
  const int rank = split_rank();
  if (aK && bK) split_tile<T, G, true, true>(P.m, P.n, P.k, aC, bC, alpha, A, P.lda, B, P.ldb, beta, C, P.ldc, m0, n0, S, rank, sm);
  else if (aK) split_tile<T, G, true, false>(P.m, P.n, P.k, aC, bC, alpha, A, P.lda, B, P.ldb, beta, C, P.ldc, m0, n0, S, rank, sm);
  else if (bK) split_tile<T, G, false, true>(P.m, P.n, P.k, aC, bC, alpha, A, P.lda, B, P.ldb, beta, C, P.ldc, m0, n0, S, rank, sm);
  else split_tile<T, G, false, false>(P.m, P.n, P.k, aC, bC, alpha, A, P.lda, B, P.ldb, beta, C, P.ldc, m0, n0, S, rank, sm);
}

// Tiles of a shape over the problems of a group, laid out for the kernel.
template <typename G>
static int64_t group_tiles(GemmGroup& g) {
  int64_t tiles = 0;
  for (int i = 0; i < g.count; ++i) {
    GroupProblem& q = g.p[i];
    q.tiles_n = (q.n + G::BN - 1) / G::BN;
    q.tile0 = tiles;
    tiles += q.tiles_n * ((q.m + G::BM - 1) / G::BM);
  }
  return tiles;
}

template <typename T, typename G>
static int grouped_launch(GemmGroup& g, cudaStream_t st) {
  const int64_t tiles = group_tiles<G>(g);
  if (tiles > 0x7fffffff) return TNC_ERR_ARG;
  gemm_grouped_kernel<T, G><<<(unsigned)tiles, G::THR, 0, st>>>(g);
  return launch_status();
}

template <typename T>
int gemm_grouped_launch(int count, const tnc_gemm_problem* probs, cudaStream_t st) {
  if (count <= 0 || count > kGroupMax || !probs) return TNC_ERR_ARG;
  GemmGroup g;
  g.count = 0;
  for (int i = 0; i < count; ++i) {
    const tnc_gemm_problem& p = probs[i];
    if (p.m < 0 || p.n < 0 || p.k <= 0 || p.opA < 0 || p.opA > 3 || p.opB < 0 || p.opB > 3 || p.ldc < p.n)
      return TNC_ERR_ARG;
    if (p.m == 0 || p.n == 0) continue;
    if (!p.A || !p.B || !p.C) return TNC_ERR_ARG;
    GroupProblem& q = g.p[g.count++];
    q.m = p.m; q.n = p.n; q.k = p.k; q.lda = p.lda; q.ldb = p.ldb; q.ldc = p.ldc;
    q.A = p.A; q.B = p.B; q.C = p.C; q.opA = p.opA; q.opB = p.opB;
    q.alpha[0] = p.alpha[0]; q.alpha[1] = p.alpha[1]; q.beta[0] = p.beta[0]; q.beta[1] = p.beta[1];
  }
  if (g.count == 0) return TNC_OK;
  auto count_tiles = [&](int bm, int bn) {
    int64_t t = 0;
    for (int i = 0; i < g.count; ++i) t += ((g.p[i].m + bm - 1) / bm) * ((g.p[i].n + bn - 1) / bn);
    return t;
  };
  if constexpr (Tile64<T>::WIDE) {
    switch (wide_tile(count_tiles)) {
      case kTileS: return grouped_launch<T, TileS<T>>(g, st);
      case kTileM: return grouped_launch<T, TileM<T>>(g, st);
      default: return grouped_launch<T, TileL<T>>(g, st);
    }
  } else {
    int64_t k = 0;
    bool small = true;  // of all problems
    for (int i = 0; i < g.count; ++i) {
      k = g.p[i].k > k ? g.p[i].k : k;
      small = small && split_small(g.p[i].m, g.p[i].n);
    }
    const int S = split_of(count_tiles, k, small);
    if (S == 0) return grouped_launch<T, Tile64<T>>(g, st);
    cudaLaunchAttribute attr;
    const int64_t tiles = small ? group_tiles<Tile32<T>>(g) : group_tiles<Tile64<T>>(g);  // a few hundred at most
    const cudaLaunchConfig_t cfg =
        split_config(dim3((unsigned)(tiles * S)), small ? Tile32<T>::THR : Tile64<T>::THR, S, st, &attr);
    const auto fn = small ? gemm_grouped_split_kernel<T, Tile32<T>> : gemm_grouped_split_kernel<T, Tile64<T>>;
    if (cudaLaunchKernelEx(&cfg, fn, g, S) != cudaSuccess) return TNC_ERR_CUDA;
    return launch_status();
  }
}

// C = beta*C when K == 0 (np.tensordot over no axes still has the outer
// product shape; with K == 0 the product is zero)
template <typename T>
__global__ void gemm_scale_c(int64_t M, int64_t N, T beta, T* C, int64_t ldc, int64_t sC, int64_t batch) {
  const int64_t total = M * N * batch;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t b = e / (M * N), r = e - b * M * N;
    int64_t i = r / N, j = r - i * N;
    T* c = C + b * sC + i * ldc + j;
    *c = (abs2_(beta) == 0) ? zero_<T>() : beta * *c;
  }
}

template <typename T, typename G>
static int simt_launch(int opA, int opB, int64_t m, int64_t n, int64_t k, T alpha, const T* A, int64_t lda, int64_t sA,
                       const T* B, int64_t ldb, int64_t sB, T beta, T* C, int64_t ldc, int64_t sC, int64_t batch,
                       cudaStream_t st) {
  const int64_t gy = (m + G::BM - 1) / G::BM, gx = (n + G::BN - 1) / G::BN;
  if (gx > 0x7fffffff) return TNC_ERR_ARG;
  const dim3 grid((unsigned)gx, (unsigned)(gy < 65535 ? gy : 65535), (unsigned)(batch < 65535 ? batch : 65535));
  // A is K-contiguous for N / R, B for T / C
  const bool aK = (opA == TNC_OP_N || opA == TNC_OP_R), bK = (opB == TNC_OP_T || opB == TNC_OP_C);
  const bool aC = (opA == TNC_OP_C || opA == TNC_OP_R), bC = (opB == TNC_OP_C || opB == TNC_OP_R);
#define TNC_GEMM_LAUNCH(AKV, BKV)                                                                                  \
  gemm_simt_kernel<T, G, AKV, BKV><<<grid, G::THR, 0, st>>>(m, n, k, aC, bC, alpha, A, lda, sA, B, ldb, sB, beta, C, \
                                                            ldc, sC, batch)
  if (aK && bK) TNC_GEMM_LAUNCH(true, true);
  else if (aK) TNC_GEMM_LAUNCH(true, false);
  else if (bK) TNC_GEMM_LAUNCH(false, true);
  else TNC_GEMM_LAUNCH(false, false);
#undef TNC_GEMM_LAUNCH
  return launch_status();
}

// Fewer than 152 tiles of 64 x 64: every count of the grid is small.
template <typename T, typename G>
static int split_launch(int opA, int opB, int64_t m, int64_t n, int64_t k, T alpha, const T* A, int64_t lda, int64_t sA,
                        const T* B, int64_t ldb, int64_t sB, T beta, T* C, int64_t ldc, int64_t sC, int64_t batch, int S,
                        cudaStream_t st) {
  const dim3 grid((unsigned)((n + G::BN - 1) / G::BN * S), (unsigned)((m + G::BM - 1) / G::BM), (unsigned)batch);
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = split_config(grid, G::THR, S, st, &attr);
  const bool aK = (opA == TNC_OP_N || opA == TNC_OP_R), bK = (opB == TNC_OP_T || opB == TNC_OP_C);
  const bool aC = (opA == TNC_OP_C || opA == TNC_OP_R), bC = (opB == TNC_OP_C || opB == TNC_OP_R);
  const auto fn = aK ? (bK ? gemm_split_kernel<T, G, true, true> : gemm_split_kernel<T, G, true, false>)
                     : (bK ? gemm_split_kernel<T, G, false, true> : gemm_split_kernel<T, G, false, false>);
  if (cudaLaunchKernelEx(&cfg, fn, m, n, k, aC, bC, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, S) !=
      cudaSuccess)
    return TNC_ERR_CUDA;
  return launch_status();
}

template <typename T>
int gemm_launch(int opA, int opB, int64_t m, int64_t n, int64_t k, T alpha, const T* A, int64_t lda,
                int64_t sA, const T* B, int64_t ldb, int64_t sB, T beta, T* C, int64_t ldc, int64_t sC,
                int64_t batch, cudaStream_t st) {
  if (m < 0 || n < 0 || k < 0 || batch < 0 || opA < 0 || opA > 3 || opB < 0 || opB > 3) return TNC_ERR_ARG;
  if (m == 0 || n == 0 || batch == 0) return TNC_OK;
  if (ldc < n) return TNC_ERR_ARG;
  if (k == 0) {
    gemm_scale_c<T><<<grid1d(m * n * batch, 256), 256, 0, st>>>(m, n, beta, C, ldc, sC, batch);
    return launch_status();
  }
  if ((m + 63) / 64 > 65535) return TNC_ERR_ARG;
  auto tiles = [&](int bm, int bn) { return ((m + bm - 1) / bm) * ((n + bn - 1) / bn) * batch; };
  if constexpr (Tile64<T>::WIDE) {
    switch (wide_tile(tiles)) {
      case kTileS: return simt_launch<T, TileS<T>>(opA, opB, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, st);
      case kTileM: return simt_launch<T, TileM<T>>(opA, opB, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, st);
      default: return simt_launch<T, TileL<T>>(opA, opB, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, st);
    }
  } else {
    const bool small = split_small(m, n);
    const int S = split_of(tiles, k, small);
    if (S == 0) return simt_launch<T, Tile64<T>>(opA, opB, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, st);
    if (small) return split_launch<T, Tile32<T>>(opA, opB, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, S, st);
    return split_launch<T, Tile64<T>>(opA, opB, m, n, k, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch, S, st);
  }
}

template int gemm_launch<float>(int, int, int64_t, int64_t, int64_t, float, const float*, int64_t, int64_t,
                                const float*, int64_t, int64_t, float, float*, int64_t, int64_t, int64_t,
                                cudaStream_t);
template int gemm_launch<double>(int, int, int64_t, int64_t, int64_t, double, const double*, int64_t, int64_t,
                                 const double*, int64_t, int64_t, double, double*, int64_t, int64_t, int64_t,
                                 cudaStream_t);
template int gemm_launch<c64>(int, int, int64_t, int64_t, int64_t, c64, const c64*, int64_t, int64_t, const c64*,
                              int64_t, int64_t, c64, c64*, int64_t, int64_t, int64_t, cudaStream_t);
template int gemm_launch<c128>(int, int, int64_t, int64_t, int64_t, c128, const c128*, int64_t, int64_t,
                               const c128*, int64_t, int64_t, c128, c128*, int64_t, int64_t, int64_t,
                               cudaStream_t);

}  // namespace tnc

using namespace tnc;

extern "C" int tnc_gemm(int dtype, int opA, int opB, int64_t m, int64_t n, int64_t k, const double* alpha,
                        const void* A, int64_t lda, int64_t strideA, const void* B, int64_t ldb,
                        int64_t strideB, const double* beta, void* C, int64_t ldc, int64_t strideC,
                        int64_t batch, void* stream) {
  if (!alpha || !beta) return TNC_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  TNC_DISPATCH(dtype, T,
               return gemm_launch<T>(opA, opB, m, n, k, from_pair<T>(alpha), (const T*)A, lda, strideA,
                                     (const T*)B, ldb, strideB, from_pair<T>(beta), (T*)C, ldc, strideC, batch,
                                     st));
  return TNC_ERR_ARG;
}

extern "C" int tnc_gemm_grouped(int dtype, int count, const tnc_gemm_problem* problems, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  TNC_DISPATCH(dtype, T, return gemm_grouped_launch<T>(count, problems, st));
  return TNC_ERR_ARG;
}
