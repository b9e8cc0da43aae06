// Host side of the single-precision block Jacobi (tnc_jacobi32.cuh).
#include "tnc_jacobi32.cuh"

#include <atomic>

namespace tnc {

constexpr size_t kJ32MaxSmem = 200 * 1024;

template <typename T, int E, bool ACC, int MAXT>
static int j32_launch(J32Args a, cudaStream_t st) {
  static std::atomic<unsigned long long> done{0};
  const void* fn = (const void*)jacobi32_kernel<T, E, ACC, MAXT>;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return TNC_ERR_CUDA;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(done.load() & bit)) {  // never lowered: callers with other row lengths share the setting
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kJ32MaxSmem) != cudaSuccess)
      return TNC_ERR_CUDA;
    done.fetch_or(bit);
  }
  const size_t smem = (size_t)2 * a.h * 32 * E * sizeof(T) * (ACC ? 2 : 1);
  if (smem > kJ32MaxSmem || 32 * a.h > MAXT) return TNC_ERR_ARG;
  const int threads = 32 * a.h, cap = coop_capacity(fn, threads, smem);
  if (cap < a.N / 2) return TNC_ERR_CUDA;  // every half-block pair has its CTA
  void* args[] = {(void*)&a};
  if (cudaLaunchCooperativeKernel(fn, dim3((unsigned)(a.N / 2)), dim3(threads), args, smem, st) != cudaSuccess)
    return TNC_ERR_CUDA;
  return TNC_OK;
}

template <typename T>
int jacobi32_rows(T* W, T* J, int64_t nr, int64_t L, int h, int max_sweeps, double tol, double stop_tol,
                  const double* frob2, float* Dn, unsigned* counters, SyncWords* sw, int* info, int64_t nkeep,
                  cudaStream_t st) {
  if (nr <= 0 || L > 1024 || nr > L || (J && L > 512)) return TNC_ERR_ARG;
  if (h != 2 && h != 4 && h != 8 && h != 16) h = 8;
  if (h == 16 && (L > 512 || J)) h = 8;
  while (h > 2 && h / 2 >= nr) h >>= 1;
  if (max_sweeps > kJ32MaxSweeps) max_sweeps = kJ32MaxSweeps;
  const int64_t nb = (nr + h - 1) / h;
  J32Args a;
  a.W = W;
  a.J = J;
  a.nr = (int)nr;
  a.L = (int)L;
  a.h = h;
  a.N = (int)(nb + (nb & 1));
  a.kb = (int)((nkeep < nr ? nkeep : nr) + h - 1) / h;
  a.max_sweeps = max_sweeps;
  a.vec = (L * (int64_t)sizeof(T)) % 16 == 0 && (uintptr_t)W % 16 == 0 && (uintptr_t)J % 16 == 0;
  a.rtol = (float)tol;
  a.stol = (float)stop_tol;
  a.staged = stop_tol > 0;
  a.frob2 = frob2;
  a.Dn = Dn;
  a.counters = counters;
  a.ver = counters + 2 * kJ32MaxSweeps;
  a.sw = sw;
  a.info = info;
  if (J) {
    if (L <= 128) return j32_launch<T, 4, true, 256>(a, st);
    if (L <= 256) return j32_launch<T, 8, true, 256>(a, st);
    return j32_launch<T, 16, true, 256>(a, st);
  }
  if (h == 16) {
    if (L <= 128) return j32_launch<T, 4, false, 512>(a, st);
    if (L <= 256) return j32_launch<T, 8, false, 512>(a, st);
    return j32_launch<T, 16, false, 512>(a, st);
  }
  if (L <= 128) return j32_launch<T, 4, false, 256>(a, st);
  if (L <= 256) return j32_launch<T, 8, false, 256>(a, st);
  if (L <= 512) return j32_launch<T, 16, false, 256>(a, st);
  return j32_launch<T, 32, false, 256>(a, st);
}

template int jacobi32_rows<float>(float*, float*, int64_t, int64_t, int, int, double, double, const double*, float*,
                                  unsigned*, SyncWords*, int*, int64_t, cudaStream_t);
template int jacobi32_rows<c64>(c64*, c64*, int64_t, int64_t, int, int, double, double, const double*, float*,
                                unsigned*, SyncWords*, int*, int64_t, cudaStream_t);

TNC_DEFINE_SPIN_SETTER(spin_limit_set_j32)

// Self-test: a warp waits for a row nobody gives.
__global__ void j32_selftest_kernel(const unsigned* counter, SyncWords* sw, int* info) {
  j32_wait_row(counter, 1u, sw);
  if (threadIdx.x == 0) info[0] = ld_volatile(&sw->err);
}
int j32_wait_selftest(const unsigned* counter, SyncWords* sw, int* info, cudaStream_t st) {
  j32_selftest_kernel<<<1, 32, 0, st>>>(counter, sw, info);
  return launch_status(1);
}

}  // namespace tnc
