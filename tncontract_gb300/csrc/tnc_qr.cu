// Reduced QR (np.linalg.qr(mode="reduced") in tensor_qr, tncontract/tensor.py:1044).
//
// Householder QR in LAPACK's convention (geqrf + ungqr: Q = H_0 ... H_{k-1},
// H_c = I - tau_c v_c v_c^H, v_c[c] = 1, R's diagonal real for complex input).
// Up to kQrPanelRows rows it runs in panels (tnc_qr_block.cuh): one cluster
// factors a panel and forms its block reflector's T, one launch applies it to
// the remaining columns, and Q is formed by the same block reflectors in
// reverse.  Longer matrices run the general kernels below: a cooperative
// column-owner dataflow, where every column of A is owned by one warp;
// reflector c is published (with a flag) by the owner of column c as soon as
// reflectors 0..c-1 have been applied to that column, and each warp applies
// the published reflectors to its own columns in order, the owner of column
// c+1 first (look-ahead).
//
// Working layout: Bt = A^T (row c of Bt is column c of A, contiguous), so
// every warp streams its own column and the published reflector with
// coalesced loads.
#include "tnc_persist.cuh"
#include "tnc_qr_block.cuh"

#include <atomic>
#include <type_traits>

namespace tnc {

constexpr int kQrWarps = 4;  // warps per CTA

template <typename T> __device__ __forceinline__ typename traits<T>::real imag_(T v) {
  if constexpr (traits<T>::is_complex) return v.im; else return 0;
}

// Reflector for column c (row c of Bt), LAPACK larfg convention.
template <typename T>
__device__ void make_reflector(T* col, int64_t c, int64_t m, T* tau_out) {
  typedef typename traits<T>::real R;
  const int lane = threadIdx.x & 31;
  R xn = 0;
  for (int64_t i = c + 1 + lane; i < m; i += 32) xn += abs2_(col[i]);
  xn = warp_sum(xn);
  T alpha = col[c];
  T tau = zero_<T>();
  if (!(xn == R(0) && imag_(alpha) == R(0))) {
    R ar = real_(alpha);
    R beta = -copysign(sqrt(abs2_(alpha) + xn), ar);
    T betaT = from_real<T>(beta);
    tau = qr_div<T>(betaT - alpha, betaT);
    T scal = qr_div<T>(one_<T>(), alpha - betaT);
    for (int64_t i = c + 1 + lane; i < m; i += 32) col[i] = scal * col[i];
    __syncwarp();
    if (lane == 0) col[c] = betaT;
  }
  if (lane == 0) *tau_out = tau;
  __syncwarp();
}

// col[i] -= conj(tau) * (v^H col) * v[i], i >= c  (applies H_c^H)
template <typename T>
__device__ __forceinline__ void apply_reflector_h(T* col, const T* v, T tau, int64_t c, int64_t m) {
  const T w = warp_reflector_dot(v, col, c, m);
  __syncwarp();
  warp_reflector_axpy(v, col, conj_(tau) * w, c, m);
  __syncwarp();
}

template <typename T>
__global__ void __launch_bounds__(kQrWarps * 32)
qr_factor_kernel(T* Bt, int64_t m, int64_t n, int64_t ld, T* tau, int* flags, SyncWords* sw) {
  const int64_t k = m < n ? m : n;
  const int64_t nwarps = (int64_t)gridDim.x * kQrWarps;
  const int64_t wid = (int64_t)blockIdx.x * kQrWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (wid >= n) return;
  // my columns: wid, wid + nwarps, ...
  if (wid == 0) {  // column 0 needs no earlier reflector
    make_reflector(Bt, 0, m, tau);
    __threadfence();
    if (lane == 0) atomicExch(&flags[0], 1);
  }
  int64_t first = wid;  // first own column not yet past all reflectors
  for (int64_t c = 0; c < k; ++c) {
    // skip own columns <= c: they are final (their reflector is published)
    while (first <= c) first += nwarps;
    if (first >= n) break;  // nothing left to update
    if (!warp_wait_flag(&flags[c], sw)) return;
    const T* v = Bt + c * ld;
    const T tc = ldcg(tau + c);
    for (int64_t j = first; j < n; j += nwarps) {
      apply_reflector_h(Bt + j * ld, v, tc, c, m);
      if (j == c + 1 && j < k) {  // look-ahead: publish the next reflector now
        make_reflector(Bt + j * ld, j, m, tau + j);
        __threadfence();
        if (lane == 0) atomicExch(&flags[j], 1);
      }
    }
  }
}

// Qt[j] = H_{min(j,k-1)} ... H_0 e_j  (row j of Qt = column j of Q)
template <typename T>
__global__ void __launch_bounds__(kQrWarps * 32)
qr_form_q_kernel(const T* __restrict__ Bt, int64_t m, int64_t k, const T* __restrict__ tau, T* __restrict__ Qt) {
  const int64_t nwarps = (int64_t)gridDim.x * kQrWarps;
  const int lane = threadIdx.x & 31;
  for (int64_t j = (int64_t)blockIdx.x * kQrWarps + (threadIdx.x >> 5); j < k; j += nwarps) {
    T* q = Qt + j * m;
    for (int64_t i = lane; i < m; i += 32) q[i] = (i == j) ? one_<T>() : zero_<T>();
    __syncwarp();
    for (int64_t c = j; c >= 0; --c) {
      const T* v = Bt + c * m;
      const T tc = tau[c];
      // q -= tau * (v^H q) * v  (H_c, not conjugated)
      const T w = warp_reflector_dot(v, q, c, m);
      __syncwarp();
      warp_reflector_axpy(v, q, tc * w, c, m);
      __syncwarp();
    }
  }
}

// R[i][j] = Bt[j][i] for i <= j, 0 below (R is k x n)
template <typename T>
__global__ void qr_extract_r(const T* __restrict__ Bt, int64_t m, int64_t n, int64_t k, T* __restrict__ R) {
  const int64_t total = k * n;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t i = e / n, j = e - i * n;
    R[e] = (i <= j) ? Bt[j * m + i] : zero_<T>();
  }
}

static size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// ---------------------------------------------------------------------------
// Workspace.  `blocked` (k >= kQrBlockedMin) has room for the general path's
// products; the panels' T factors (nb x nb each) lie in its `sm` area, or in an
// area of their own for a smaller k.
template <typename T>
static int dtype_of() {
  return sizeof(T) == 4 ? TNC_F32 : (sizeof(T) == 8 ? (traits<T>::is_complex ? TNC_C64 : TNC_F64) : TNC_C128);
}

constexpr int64_t kQrNB = 64;                 // panel width of the general path
constexpr int64_t kQrBlockedMin = 2 * kQrNB;  // k below this: its unblocked dataflow only

constexpr int64_t kQrSplitK = 128;  // K chunk of the split-K products

struct QrLayout {
  size_t bt, tau, flags, sync, qt, vt, sm, wt, w2t, part, tf, total;
  bool blocked;
};
// t_area = false: the caller keeps the T factors (at most k x k elements) elsewhere.
static QrLayout qr_layout(int64_t m, int64_t n, int dt, bool t_area = true) {
  const size_t es = (size_t)elem_size(dt);
  int64_t k = m < n ? m : n;
  QrLayout L;
  size_t off = 0;
  L.blocked = k >= kQrBlockedMin;
  L.bt = off; off = align256(off + (size_t)n * m * es);
  L.tau = off; off = align256(off + (size_t)k * es);
  L.flags = off; off = align256(off + (size_t)k * sizeof(int));
  L.sync = off; off = align256(off + sizeof(SyncWords));
  L.qt = off; off = align256(off + (size_t)k * m * es);
  L.vt = L.sm = L.wt = L.w2t = L.part = off;
  if (L.blocked) {
    const int64_t nblk = (k + kQrNB - 1) / kQrNB;
    const int64_t rows = n > k ? n : k;
    L.vt = off; off = align256(off + (size_t)kQrNB * m * es);
    L.sm = off; off = align256(off + (size_t)nblk * kQrNB * kQrNB * es);
    L.wt = off; off = align256(off + (size_t)rows * kQrNB * es);
    L.w2t = off; off = align256(off + (size_t)rows * kQrNB * es);
    L.part = off; off = align256(off + (size_t)((m + kQrSplitK - 1) / kQrSplitK) * rows * kQrNB * es);
    L.tf = L.sm;
  } else {
    L.tf = off;
    if (t_area) off = align256(off + (size_t)k * (k < kQrNB ? k : kQrNB) * es);
  }
  L.total = off;
  return L;
}

// Vt[j][i] = reflector j of a panel (i = row within the panel's sub-matrix):
// 0 above the diagonal, 1 on it, the stored entries below
template <typename T>
__global__ void qr_extract_vt(const T* __restrict__ Bt, int64_t ld, int64_t nbb, int64_t ms, T* __restrict__ Vt) {
  const int64_t total = nbb * ms;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = e / ms, i = e - j * ms;
    Vt[e] = (i < j) ? zero_<T>() : (i == j ? one_<T>() : Bt[j * ld + i]);
  }
}

template <typename T> __device__ __forceinline__ bool is_zero_(T v) {
  if constexpr (traits<T>::is_complex) return v.re == 0 && v.im == 0; else return v == 0;
}

// The block reflector's T enters only as T^H W (trailing update) and T W (Q
// formation).  For Householder blocks T^-1 = U = striu(S) + diag(1/tau) with
// S = V^H V (from Q = I - V T V^H unitary: T^-1 + T^-H = V^H V, T^-1 upper
// triangular), so both products are triangular solves against S:
//   adjoint: U^H W2 = W (forward),   else: U W2 = W (backward).
// A reflector with tau = 0 (H = I) drops out of the product: its component
// of W2 is 0 and it is skipped by the others.  Rows of Wt / W2t are columns
// of W / W2 (rows x nbb); one warp per row, lane l holding components l and
// l + 32, S and tau staged in shared memory (nbb * nbb + nbb elements).
template <typename T>
__global__ void qr_apply_tinv(const T* __restrict__ S, const T* __restrict__ tau, int64_t nbb, const T* __restrict__ Wt,
                              T* __restrict__ W2t, int64_t rows, int adjoint) {
  extern __shared__ __align__(16) unsigned char qr_t_smem[];
  T* sS = reinterpret_cast<T*>(qr_t_smem);
  T* st = sS + nbb * nbb;
  for (int64_t e = threadIdx.x; e < nbb * nbb; e += blockDim.x) sS[e] = S[e];
  for (int64_t e = threadIdx.x; e < nbb; e += blockDim.x) st[e] = tau[e];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int n = (int)nbb;
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += nwarps) {
    const T* wr = Wt + r * nbb;
    T a0 = zero_<T>(), a1 = zero_<T>();
    if (adjoint) {
      for (int i = 0; i < n; ++i) {
        T p = zero_<T>();
        if (lane < i) p = conj_(sS[lane * n + i]) * a0;
        if (lane + 32 < i) p += conj_(sS[(lane + 32) * n + i]) * a1;
        p = warp_sum(p);
        const T ti = st[i];
        const T val = is_zero_(ti) ? zero_<T>() : (wr[i] - p) * conj_(ti);
        if (lane == i) a0 = val;
        if (lane + 32 == i) a1 = val;
      }
    } else {
      for (int i = n - 1; i >= 0; --i) {
        T p = zero_<T>();
        if (lane > i && lane < n) p = sS[i * n + lane] * a0;
        if (lane + 32 > i && lane + 32 < n) p += sS[i * n + lane + 32] * a1;
        p = warp_sum(p);
        const T ti = st[i];
        const T val = is_zero_(ti) ? zero_<T>() : (wr[i] - p) * ti;
        if (lane == i) a0 = val;
        if (lane + 32 == i) a1 = val;
      }
    }
    if (lane < n) W2t[r * nbb + lane] = a0;
    if (lane + 32 < n) W2t[r * nbb + lane + 32] = a1;
  }
}

// Dynamic shared memory of qr_apply_tinv beyond the 48 KB default
// (complex128): raised once per device.
template <typename T>
static int ensure_tinv_smem() {
  constexpr size_t bytes = (size_t)(kQrNB * kQrNB + kQrNB) * sizeof(T);
  if constexpr (bytes <= 48 * 1024) {
    return TNC_OK;
  } else {
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return TNC_ERR_CUDA;
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load() & bit) return TNC_OK;
    if (cudaFuncSetAttribute((const void*)qr_apply_tinv<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) !=
        cudaSuccess)
      return TNC_ERR_CUDA;
    done.fetch_or(bit);
    return TNC_OK;
  }
}

// C (rows x cols, ld ldc) = sum over nparts of P[p] (rows x cols, dense)
template <typename T>
__global__ void qr_sum_parts(const T* __restrict__ P, int64_t nparts, int64_t rows, int64_t cols, T* __restrict__ C,
                             int64_t ldc) {
  const int64_t total = rows * cols;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    T acc = zero_<T>();
    for (int64_t p = 0; p < nparts; ++p) acc += P[p * total + e];
    const int64_t r = e / cols, c = e - r * cols;
    C[r * ldc + c] = acc;
  }
}

// Qt = the first k rows of the m x m identity
template <typename T>
__global__ void qr_eye_rows(T* Qt, int64_t k, int64_t m) {
  const int64_t total = k * m;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = e / m, i = e - j * m;
    Qt[e] = (i == j) ? one_<T>() : zero_<T>();
  }
}

// C (M x N, ld ldc) = op(A) op(B) with A (M x K, row-major, opA N or R) and B
// (N x K, row-major, opB T or C): the K range is cut into chunks of kQrSplitK,
// each chunk one member of a batched CUDA-core GEMM into P, then the partial
// products are summed -- enough CTAs for the long-K, narrow products of the
// blocked QR, at FP32 accuracy.
template <typename T>
static int qr_gemm_splitk(int opA, int opB, int64_t M, int64_t N, int64_t K, const T* A, int64_t lda, const T* B,
                          int64_t ldb, T* C, int64_t ldc, T* P, cudaStream_t st) {
  const int64_t nparts = (K + kQrSplitK - 1) / kQrSplitK;
  const int64_t full = K / kQrSplitK;  // chunks of full length
  const T one = one_<T>(), zero = zero_<T>();
  if (full > 0) {
    if (int rc = gemm_launch<T>(opA, opB, M, N, kQrSplitK, one, A, lda, kQrSplitK, B, ldb, kQrSplitK, zero, P, N, M * N,
                                full, st))
      return rc;
  }
  if (full < nparts) {  // the ragged last chunk
    const int64_t k0 = full * kQrSplitK;
    if (int rc = gemm_launch<T>(opA, opB, M, N, K - k0, one, A + k0, lda, 0, B + k0, ldb, 0, zero, P + full * M * N, N,
                                0, 1, st))
      return rc;
  }
  qr_sum_parts<T><<<grid1d(M * N, 256), 256, 0, st>>>(P, nparts, M, N, C, ldc);
  return launch_status(1);
}

// Unblocked dataflow factorisation of the m x n matrix whose transpose is at
// Bt (row stride ld): reflectors in place, tau, per-column flags (zeroed by
// the caller), errors in sw.
template <typename T>
static int qr_dataflow(int64_t m, int64_t n, int64_t ld, T* Bt, T* tau, int* flags, SyncWords* sw, cudaStream_t st) {
  void* args[] = {(void*)&Bt, (void*)&m, (void*)&n, (void*)&ld, (void*)&tau, (void*)&flags, (void*)&sw};
  const int threads = kQrWarps * 32;
  int cap = coop_capacity((const void*)qr_factor_kernel<T>, threads, 0);
  if (cap <= 0) return TNC_ERR_CUDA;
  int64_t want = (n + kQrWarps - 1) / kQrWarps;
  int grid = (int)(want < cap ? want : cap);
  if (cudaLaunchCooperativeKernel((const void*)qr_factor_kernel<T>, dim3(grid), dim3(threads), args, 0, st) !=
      cudaSuccess)
    return TNC_ERR_CUDA;
  return launch_status(1);
}

// A kernel's dynamic shared memory (and cluster sizes above 8), once per device.
static int cluster_attrs(const void* fn, size_t smem, std::atomic<unsigned long long>& done) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return TNC_ERR_CUDA;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load() & bit) return TNC_OK;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return TNC_ERR_CUDA;
  done.fetch_or(bit);
  return TNC_OK;
}

static cudaLaunchConfig_t cluster_config(unsigned ctas, unsigned cluster, int threads, size_t smem, cudaStream_t st,
                                         cudaLaunchAttribute* attr) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = cluster;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

static int pow2_at_least(int64_t v) {
  int p = 1;
  while (p < v) p *= 2;
  return p;
}

template <typename T, int R>
static int launch_panel(T* P, int64_t ld, int m, int nb, T* tau, T* Tout, int* info, cudaStream_t st) {
  static std::atomic<unsigned long long> done{0};
  const size_t smem = qr_panel_smem<T>(R);
  if (int rc = cluster_attrs((const void*)qr_panel_kernel<T, R>, smem, done)) return rc;
  const int cs = pow2_at_least((m + 32 * R - 1) / (32 * R));
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cluster_config(cs, cs, QrShape<T>::NW * 32, smem, st, &attr);
  return cudaLaunchKernelEx(&cfg, qr_panel_kernel<T, R>, P, ld, m, nb, tau, Tout, cs, info) == cudaSuccess ? TNC_OK
                                                                                                         : TNC_ERR_CUDA;
}

// Rows of a lane (R; a CTA holds 32 R) by the panel's length.  FP32: a step's
// arithmetic grows with R, its exchange with the CTAs, and empty rows cost as
// much as full ones.  So R goes in steps of one for complex types (real ones
// pack rows in pairs and gain nothing from an odd R beyond 3), on 4 CTAs up to
// 512 rows (1024 for real types) and else on 8, the portable cluster (16 CTAs of
// half the rows: 3.30 ms for 1536 x 768 complex64, 2.84 on 8).  Against R of 2,
// 4, 6 and 8 on 8 CTAs: 1536 x 768 complex64 2.83 -> 2.78 ms, 768 x 512 1.47 ->
// 1.43, 1280 x 64 0.238 -> 0.225; float32 512 x 256 0.606 -> 0.559, 768 x 64
// 0.186 -> 0.177.  FP64 panels spread over 16 CTAs as soon as possible, their
// arithmetic being the longer part.
template <typename T>
static int qr_panel(T* P, int64_t ld, int64_t m, int64_t nb, T* tau, T* Tout, int* info, cudaStream_t st) {
  const int rows = (int)m, n = (int)nb;
  constexpr bool cplx = traits<T>::is_complex;
  if constexpr (sizeof(typename traits<T>::real) == 4) {
    if (m <= (cplx ? 256 : 128)) return launch_panel<T, 2>(P, ld, rows, n, tau, Tout, info, st);
    if (m > 256 && m <= 384) return launch_panel<T, 3>(P, ld, rows, n, tau, Tout, info, st);
    if (m <= 512) return launch_panel<T, 4>(P, ld, rows, n, tau, Tout, info, st);
    if (m <= 768) return launch_panel<T, cplx ? 3 : 6>(P, ld, rows, n, tau, Tout, info, st);
    if (m <= 1024) return launch_panel<T, cplx ? 4 : 8>(P, ld, rows, n, tau, Tout, info, st);
    if (cplx && m <= 1280) return launch_panel<T, cplx ? 5 : 6>(P, ld, rows, n, tau, Tout, info, st);
    if (m <= 1536) return launch_panel<T, 6>(P, ld, rows, n, tau, Tout, info, st);
    if (cplx && m <= 1792) return launch_panel<T, cplx ? 7 : 8>(P, ld, rows, n, tau, Tout, info, st);
  } else {
    if (m <= 512) return launch_panel<T, 1>(P, ld, rows, n, tau, Tout, info, st);
    if (m <= 1024) return launch_panel<T, 2>(P, ld, rows, n, tau, Tout, info, st);
    if (m <= 2048) return launch_panel<T, 4>(P, ld, rows, n, tau, Tout, info, st);
  }
  return launch_panel<T, 8>(P, ld, rows, n, tau, Tout, info, st);
}

// X (nc columns, ms rows) <- (I - V op(T) V^H) X.  Clusters of up to 8 CTAs of
// 64 rows or more, 32 where that leaves SMs idle, as many as shared memory
// holds at most.
template <typename T>
static int qr_apply(const T* V, int64_t ldv, int64_t nb, int64_t ms, const T* Tm, T* X, int64_t ldx, int64_t nc,
                    int adjoint, cudaStream_t st) {
  constexpr int kRows = std::is_same<T, c64>::value ? 192 : 256;
  static std::atomic<unsigned long long> done{0};
  if (int rc = cluster_attrs((const void*)qr_apply_kernel<T>, qr_apply_smem<T>(kRows), done)) return rc;
  const int64_t blocks = (nc + QrShape<T>::NC - 1) / QrShape<T>::NC;
  int cs = pow2_at_least((ms + 63) / 64);
  if (cs > 8) cs = 8;
  while (cs < 8 && 32 * cs < ms && blocks * cs < 152) cs *= 2;
  int64_t rows = ((ms + cs - 1) / cs + 31) / 32 * 32;
  if (rows < QrShape<T>::NB) rows = QrShape<T>::NB;
  if (rows > kRows) rows = kRows;
  if (blocks * cs > 0x7fffffff) return TNC_ERR_ARG;
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cluster_config((unsigned)(blocks * cs), cs, QrShape<T>::ATHR,
                                                qr_apply_smem<T>((int)rows), st, &attr);
  return cudaLaunchKernelEx(&cfg, qr_apply_kernel<T>, V, ldv, (int)nb, ms, Tm, X, ldx, nc, (int)rows, cs, adjoint) ==
                 cudaSuccess
             ? TNC_OK
             : TNC_ERR_CUDA;
}

// Householder factorisation of the m x n matrix X whose transpose is already
// in Bt (n x m, dense).  R (k x n) is always extracted; the rows of Q^T
// (k x m, in the workspace at L.qt) are formed when want_qt or Q is set, and
// Q = (Q^T)^T (m x k) is written when Q is not null.
template <typename T>
static int qr_factor_bt(int64_t m, int64_t n, T* Q, bool want_qt, T* R, const QrLayout& L, char* w, T* tf, int* info,
                        cudaStream_t st) {
  const int64_t k = m < n ? m : n;
  T* Bt = (T*)(w + L.bt);
  T* tau = (T*)(w + L.tau);
  int* flags = (int*)(w + L.flags);
  SyncWords* sw = (SyncWords*)(w + L.sync);
  T* Qt = (T*)(w + L.qt);
  const bool form_q = (Q != nullptr || want_qt);
  if (m <= kQrPanelRows) {
    constexpr int64_t NB = QrShape<T>::NB;
    if (cudaMemsetAsync(info, 0, sizeof(int), st) != cudaSuccess) return TNC_ERR_CUDA;
    int launches = 1;  // extract R
    for (int64_t c0 = 0; c0 < k; c0 += NB) {
      const int64_t nb = (k - c0) < NB ? (k - c0) : NB, ms = m - c0, n2 = n - c0 - nb;
      T* panel = Bt + c0 * m + c0;
      if (int rc = qr_panel<T>(panel, m, ms, nb, tau + c0, tf + c0 * NB, info, st)) return rc;
      ++launches;
      if (n2 > 0) {
        if (int rc = qr_apply<T>(panel, m, nb, ms, tf + c0 * NB, panel + nb * m, m, n2, 1, st)) return rc;
        ++launches;
      }
    }
    qr_extract_r<T><<<grid1d(k * n, 256), 256, 0, st>>>(Bt, m, n, k, R);
    if (form_q) {
      qr_eye_rows<T><<<grid1d(k * m, 256), 256, 0, st>>>(Qt, k, m);
      ++launches;
      for (int64_t c0 = (k - 1) / NB * NB; c0 >= 0; c0 -= NB) {
        const int64_t nb = (k - c0) < NB ? (k - c0) : NB;
        if (int rc = qr_apply<T>(Bt + c0 * m + c0, m, nb, m - c0, tf + c0 * NB, Qt + c0 * m + c0, m, k - c0, 0, st))
          return rc;
        ++launches;
      }
    }
    if (launch_status(launches)) return TNC_ERR_CUDA;
    if (Q == nullptr) return TNC_OK;
    const int64_t shp[2] = {k, m};
    const int perm[2] = {1, 0};
    return tnc_permute(dtype_of<T>(), Qt, Q, 2, shp, perm, 0, st);
  }
  if (cudaMemsetAsync(flags, 0, (size_t)k * sizeof(int), st) != cudaSuccess) return TNC_ERR_CUDA;
  if (cudaMemsetAsync(sw, 0, sizeof(SyncWords), st) != cudaSuccess) return TNC_ERR_CUDA;
  if (cudaMemsetAsync(info, 0, sizeof(int), st) != cudaSuccess) return TNC_ERR_CUDA;
  if (!L.blocked) {
    if (int rc = qr_dataflow<T>(m, n, m, Bt, tau, flags, sw, st)) return rc;
    copy_sync_error<<<1, 1, 0, st>>>(sw, info);
    int launches = 2;  // error copy, extract R
    if (form_q) {
      const int threads = kQrWarps * 32;
      int64_t gq = (k + kQrWarps - 1) / kQrWarps;
      if (gq > 152 * 16) gq = 152 * 16;
      qr_form_q_kernel<T><<<(unsigned)gq, threads, 0, st>>>(Bt, m, k, tau, Qt);
      ++launches;
    }
    qr_extract_r<T><<<grid1d(k * n, 256), 256, 0, st>>>(Bt, m, n, k, R);
    if (launch_status(launches)) return TNC_ERR_CUDA;
  } else {
    T* Vt = (T*)(w + L.vt);
    T* Sall = (T*)(w + L.sm);  // S = V^H V of every panel
    T* Wt = (T*)(w + L.wt);
    T* W2t = (T*)(w + L.w2t);
    T* P = (T*)(w + L.part);
    const T one = one_<T>(), mone = zero_<T>() - one_<T>();
    const int64_t nblk = (k + kQrNB - 1) / kQrNB;
    if (int rc = ensure_tinv_smem<T>()) return rc;
    const size_t tinv_smem = (size_t)(kQrNB * kQrNB + kQrNB) * sizeof(T);
    for (int64_t b = 0; b < nblk; ++b) {
      const int64_t c0 = b * kQrNB;
      const int64_t nbb = (k - c0) < kQrNB ? (k - c0) : kQrNB;
      const int64_t ms = m - c0;
      T* panel = Bt + c0 * m + c0;
      if (int rc = qr_dataflow<T>(ms, nbb, m, panel, tau + c0, flags + c0, sw, st)) return rc;
      const int64_t n2 = n - c0 - nbb;
      const bool need_t = form_q || n2 > 0;
      if (!need_t) continue;
      qr_extract_vt<T><<<grid1d(nbb * ms, 256), 256, 0, st>>>(panel, m, nbb, ms, Vt);
      // S = V^H V = conj(Vt) Vt^T, kept per panel for the Q formation
      T* Sb = Sall + b * kQrNB * kQrNB;
      if (int rc = qr_gemm_splitk<T>(TNC_OP_R, TNC_OP_T, nbb, nbb, ms, Vt, ms, Vt, ms, Sb, nbb, P, st)) return rc;
      if (launch_status(1)) return TNC_ERR_CUDA;
      if (n2 > 0) {
        T* X2t = Bt + (c0 + nbb) * m + c0;  // trailing columns, rows c0.. (n2 x ms, ld m)
        if (int rc = qr_gemm_splitk<T>(TNC_OP_N, TNC_OP_C, n2, nbb, ms, X2t, m, Vt, ms, Wt, nbb, P, st)) return rc;
        // W2 = T^H W
        qr_apply_tinv<T><<<grid1d(n2 * 32, 256, 152 * 8), 256, tinv_smem, st>>>(Sb, tau + c0, nbb, Wt, W2t, n2, 1);
        if (launch_status(1)) return TNC_ERR_CUDA;
        if (int rc = gemm_launch<T>(TNC_OP_N, TNC_OP_N, n2, ms, nbb, mone, W2t, nbb, 0, Vt, ms, 0, one, X2t, m, 0, 1,
                                    st))
          return rc;
      }
    }
    copy_sync_error<<<1, 1, 0, st>>>(sw, info);
    qr_extract_r<T><<<grid1d(k * n, 256), 256, 0, st>>>(Bt, m, n, k, R);
    if (launch_status(2)) return TNC_ERR_CUDA;
    if (form_q) {
      qr_eye_rows<T><<<grid1d(k * m, 256), 256, 0, st>>>(Qt, k, m);
      if (launch_status(1)) return TNC_ERR_CUDA;
      for (int64_t b = nblk - 1; b >= 0; --b) {
        const int64_t c0 = b * kQrNB;
        const int64_t nbb = (k - c0) < kQrNB ? (k - c0) : kQrNB;
        const int64_t ms = m - c0;
        const int64_t nq = k - c0;            // columns of Q touched
        T* Qs = Qt + c0 * m + c0;             // nq x ms, ld m
        const T* Sb = Sall + b * kQrNB * kQrNB;
        qr_extract_vt<T><<<grid1d(nbb * ms, 256), 256, 0, st>>>(Bt + c0 * m + c0, m, nbb, ms, Vt);
        if (launch_status(1)) return TNC_ERR_CUDA;
        if (int rc = qr_gemm_splitk<T>(TNC_OP_N, TNC_OP_C, nq, nbb, ms, Qs, m, Vt, ms, Wt, nbb, P, st)) return rc;
        // W2 = T W
        qr_apply_tinv<T><<<grid1d(nq * 32, 256, 152 * 8), 256, tinv_smem, st>>>(Sb, tau + c0, nbb, Wt, W2t, nq, 0);
        if (launch_status(1)) return TNC_ERR_CUDA;
        if (int rc = gemm_launch<T>(TNC_OP_N, TNC_OP_N, nq, ms, nbb, mone, W2t, nbb, 0, Vt, ms, 0, one, Qs, m, 0, 1, st))
          return rc;
      }
    }
  }
  if (Q == nullptr) return TNC_OK;
  // Q = Qt^T
  int64_t shp[2] = {k, m};
  int perm[2] = {1, 0};
  return tnc_permute(dtype_of<T>(), Qt, Q, 2, shp, perm, 0, st);
}

template <typename T>
static int qr_impl(int64_t m, int64_t n, const T* A, int64_t lda, T* Q, T* R, void* work, size_t wb,
                   int* info, cudaStream_t st) {
  if (m <= 0 || n <= 0 || lda < n || !A || !Q || !R || !work || !info) return TNC_ERR_ARG;
  if (lda != n) return TNC_ERR_ARG;
  QrLayout L = qr_layout(m, n, dtype_of<T>());
  if (wb < L.total) return TNC_ERR_WORKSPACE;
  char* w = (char*)work;
  // Bt = A^T
  int64_t shp[2] = {m, n};
  int perm[2] = {1, 0};
  if (int s = tnc_permute(dtype_of<T>(), A, (T*)(w + L.bt), 2, shp, perm, 0, st)) return s;
  return qr_factor_bt<T>(m, n, Q, false, R, L, w, (T*)(w + L.tf), info, st);
}

// R factor only, of A (m x n) or, with adjoint, of A^H (n x m).  For A^H the
// transposed copy the factorisation works on is conj(A) itself, so no
// transpose runs.
template <typename T>
static int qr_r_impl(int64_t m, int64_t n, const T* A, int adjoint, T* R, void* work, size_t wb, int* info,
                     cudaStream_t st) {
  if (m <= 0 || n <= 0 || !A || !R || !work || !info) return TNC_ERR_ARG;
  const int64_t fm = adjoint ? n : m, fn = adjoint ? m : n;  // the factorised matrix is fm x fn
  QrLayout L = qr_layout(fm, fn, dtype_of<T>());
  if (wb < L.total) return TNC_ERR_WORKSPACE;
  char* w = (char*)work;
  if (adjoint) {
    int64_t shp[2] = {m, n};
    int perm[2] = {0, 1};
    if (int s = tnc_permute(dtype_of<T>(), A, (T*)(w + L.bt), 2, shp, perm, traits<T>::is_complex ? 1 : 0, st))
      return s;
  } else {
    int64_t shp[2] = {m, n};
    int perm[2] = {1, 0};
    if (int s = tnc_permute(dtype_of<T>(), A, (T*)(w + L.bt), 2, shp, perm, 0, st)) return s;
  }
  return qr_factor_bt<T>(fm, fn, (T*)nullptr, false, R, L, w, (T*)(w + L.tf), info, st);
}

}  // namespace tnc

namespace tnc {

size_t qr_qt_workspace(int64_t fm, int64_t fn, int dt) { return qr_layout(fm, fn, dt, false).total; }

template <typename T>
int qr_qt(int64_t fm, int64_t fn, const T* A, int adjoint, bool want_qt, T* R, void* work, size_t wb, T* tf, int* info,
          cudaStream_t st, T** qt) {
  if (fm <= 0 || fn <= 0 || !A || !R || !work || !info) return TNC_ERR_ARG;
  QrLayout L = qr_layout(fm, fn, dtype_of<T>(), false);
  if (wb < L.total) return TNC_ERR_WORKSPACE;
  char* w = (char*)work;
  // Bt = X^T: for X = A^H that is conj(A) as stored (A is fn x fm)
  int64_t shp[2] = {adjoint ? fn : fm, adjoint ? fm : fn};
  int perm_id[2] = {0, 1}, perm_t[2] = {1, 0};
  if (int s = tnc_permute(dtype_of<T>(), A, (T*)(w + L.bt), 2, shp, adjoint ? perm_id : perm_t,
                          (adjoint && traits<T>::is_complex) ? 1 : 0, st))
    return s;
  if (qt) *qt = (T*)(w + L.qt);
  return qr_factor_bt<T>(fm, fn, (T*)nullptr, want_qt, R, L, w, L.blocked ? (T*)(w + L.tf) : tf, info, st);
}

template int qr_qt<float>(int64_t, int64_t, const float*, int, bool, float*, void*, size_t, float*, int*, cudaStream_t, float**);
template int qr_qt<double>(int64_t, int64_t, const double*, int, bool, double*, void*, size_t, double*, int*, cudaStream_t, double**);
template int qr_qt<c64>(int64_t, int64_t, const c64*, int, bool, c64*, void*, size_t, c64*, int*, cudaStream_t, c64**);
template int qr_qt<c128>(int64_t, int64_t, const c128*, int, bool, c128*, void*, size_t, c128*, int*, cudaStream_t, c128**);

TNC_DEFINE_SPIN_SETTER(spin_limit_set_qr)

// Self-test: the panel's wait for bytes that never come.
__global__ void qr_selftest_kernel(int* info) {
  __shared__ __align__(8) unsigned long long bar;
  if (threadIdx.x == 0) {
    qr_bar_init(qr_smem(&bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    qr_bar_expect(qr_smem(&bar), 16);
  }
  __syncthreads();
  const bool here = qr_bar_wait(qr_smem(&bar), 0, qr_wait_limit());
  if (!__syncthreads_and(here) && threadIdx.x == 0) info[0] = TNC_ERR_TIMEOUT;
}
int qr_wait_selftest(int* info, cudaStream_t st) {
  qr_selftest_kernel<<<1, 64, 0, st>>>(info);
  return launch_status(1);
}

}  // namespace tnc

using namespace tnc;

extern "C" int tnc_qr_workspace_size(int dtype, int64_t m, int64_t n, size_t* bytes) {
  if (!elem_size(dtype) || m <= 0 || n <= 0 || !bytes) return TNC_ERR_ARG;
  *bytes = qr_layout(m, n, dtype).total;
  return TNC_OK;
}

extern "C" int tnc_qr(int dtype, int64_t m, int64_t n, const void* A, int64_t lda, void* Q, void* R, void* work,
                      size_t work_bytes, int* info, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  TNC_DISPATCH(dtype, T, return qr_impl<T>(m, n, (const T*)A, lda, (T*)Q, (T*)R, work, work_bytes, info, st));
  return TNC_ERR_ARG;
}

extern "C" int tnc_qr_r_workspace_size(int dtype, int64_t m, int64_t n, int adjoint, size_t* bytes) {
  if (!elem_size(dtype) || m <= 0 || n <= 0 || !bytes) return TNC_ERR_ARG;
  *bytes = adjoint ? qr_layout(n, m, dtype).total : qr_layout(m, n, dtype).total;
  return TNC_OK;
}

extern "C" int tnc_qr_r(int dtype, int64_t m, int64_t n, const void* A, int adjoint, void* R, void* work,
                        size_t work_bytes, int* info, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  TNC_DISPATCH(dtype, T, return qr_r_impl<T>(m, n, (const T*)A, adjoint, (T*)R, work, work_bytes, info, st));
  return TNC_ERR_ARG;
}
