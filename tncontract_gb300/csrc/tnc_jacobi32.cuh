// One-sided block Jacobi of single-precision rows (float, complex64): the rows
// of W are rotated in pairs until they are mutually orthogonal; with an
// accumulator J (rows of the same length, ACC) the rotations are applied to its
// rows too.  The host side is jacobi32_rows (tnc_jacobi32.cu).
//
// A CTA works on two half-blocks of h rows (h = warps per CTA): the right-mover
// in registers (warp i holds row i), the left-mover in shared memory.  A sweep is
//   phase 0 -- the pairs inside the two half-blocks (an h-point round-robin);
//   rounds  -- h steps a round, step s rotating row i of the one with row
//              (i + s) mod h of the other.
// The half-blocks meet by odd-even transposition: they stand in a line, every
// round the neighbours (2i, 2i + 1) or (2i + 1, 2i + 2) meet and pass each
// other, and after N rounds (N half-blocks) all pairs have met once.  A CTA keeps
// one of its two half-blocks from a round to the next and exchanges the other, by
// rows: warp i stores its row, publishes that row's step counter, and waits for
// the counter of the row it takes.  (A round-robin tournament moved both
// half-blocks every round through barriers of the whole CTA: 9,600 of a round's
// 29,000 cycles at 512 x 512 complex64.)
//
// Lanes hold 16-byte pieces (V elements) of a row; rows are padded to 32 E
// elements with zeros, which rotations keep, so the inner loops test nothing.
// Every wait is bounded; a CTA whose wait gives up (or finds that another's has)
// records TNC_ERR_TIMEOUT, goes through the sweep without waiting again and leaves
// before its grid barrier, at which the others then leave too.
#pragma once
#include "tnc_persist.cuh"
#include "tnc_rot.cuh"

namespace tnc {

constexpr int kJ32MaxSweeps = 100;  // as kRowsMaxSweeps: rotation counts, large-rotation counts, then a step counter a row

// d += a b on both halves (one issue slot)
__device__ __forceinline__ void fma2_(float2& d, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}
__device__ __forceinline__ float2 mul2_(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return d;
}

// A lane's share of a row: P pairs of floats (a complex64 element, or two floats).
// <x, y> = sum x conj(y) over the first D pairs.
template <bool CPLX, int P, int D>
__device__ __forceinline__ void j32_dot(const float2 (&x)[P], const float2 (&y)[P], float& re, float& im) {
  float2 s0 = make_float2(0.f, 0.f), s1 = s0;
  if constexpr (CPLX) {
    float i0 = 0.f, i1 = 0.f;
#pragma unroll
    for (int u = 0; u < D; u += 2) {
      fma2_(s0, x[u], y[u]);
      i0 = fmaf(x[u].y, y[u].x, i0);
      i1 = fmaf(-x[u].x, y[u].y, i1);
      fma2_(s1, x[u + 1], y[u + 1]);
      i0 = fmaf(x[u + 1].y, y[u + 1].x, i0);
      i1 = fmaf(-x[u + 1].x, y[u + 1].y, i1);
    }
    im = i0 + i1;
  } else {
#pragma unroll
    for (int u = 0; u < D; u += 2) {
      fma2_(s0, x[u], y[u]);
      fma2_(s1, x[u + 1], y[u + 1]);
    }
    im = 0.f;
  }
  re = (s0.x + s1.x) + (s0.y + s1.y);
}

// x' = c x - se y,  y' = conj(se) x + c y
template <bool CPLX, int P>
__device__ __forceinline__ void j32_rotate(float2 (&x)[P], float2 (&y)[P], float c, float ser, float sei) {
  const float2 c2 = make_float2(c, c), p2 = make_float2(ser, ser), m2 = make_float2(-ser, -ser);
#pragma unroll
  for (int u = 0; u < P; ++u) {
    const float2 xo = x[u], yo = y[u];
    float2 a = mul2_(c2, xo), b = mul2_(c2, yo);
    fma2_(a, m2, yo);
    fma2_(b, p2, xo);
    if constexpr (CPLX) {
      a.x = fmaf(sei, yo.y, a.x);
      a.y = fmaf(-sei, yo.x, a.y);
      b.x = fmaf(sei, xo.y, b.x);
      b.y = fmaf(-sei, xo.x, b.y);
    }
    x[u] = a;
    y[u] = b;
  }
}

// Rows in shared memory: piece u of a row at float4 index u * 32 + lane.
template <int P>
__device__ __forceinline__ void j32_lds(const float4* row, float2 (&v)[P]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int u = 0; u < P / 2; ++u) {
    const float4 q = row[u * 32 + lane];
    v[2 * u] = make_float2(q.x, q.y);
    v[2 * u + 1] = make_float2(q.z, q.w);
  }
}
template <int P>
__device__ __forceinline__ void j32_sts(float4* row, const float2 (&v)[P]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int u = 0; u < P / 2; ++u) row[u * 32 + lane] = make_float4(v[2 * u].x, v[2 * u].y, v[2 * u + 1].x, v[2 * u + 1].y);
}

// Pairs [0, D) of a row in global memory (L elements; vec: 16-byte pieces).
template <typename T, int P, int D, int OFF>
__device__ __forceinline__ void j32_ldg(const T* row, int L, bool vec, float2 (&v)[P]) {
  constexpr int V = 16 / sizeof(T);
  const int lane = threadIdx.x & 31;
  if (vec) {
#pragma unroll
    for (int u = 0; u < D / 2; ++u) {
      const int e = (u * 32 + lane) * V;
      const float4 q = e < L ? __ldcg(reinterpret_cast<const float4*>(row + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[OFF + 2 * u] = make_float2(q.x, q.y);
      v[OFF + 2 * u + 1] = make_float2(q.z, q.w);
    }
  } else {
#pragma unroll
    for (int u = 0; u < D; ++u) {
      const int e = ((u / 2) * 32 + lane) * V + (u & 1) * (V / 2);
      if constexpr (traits<T>::is_complex) {
        v[OFF + u] = e < L ? __ldcg(reinterpret_cast<const float2*>(row + e)) : make_float2(0.f, 0.f);
      } else {
        v[OFF + u].x = e < L ? __ldcg(reinterpret_cast<const float*>(row) + e) : 0.f;
        v[OFF + u].y = e + 1 < L ? __ldcg(reinterpret_cast<const float*>(row) + e + 1) : 0.f;
      }
    }
  }
}
template <typename T, int P, int D, int OFF>
__device__ __forceinline__ void j32_stg(T* row, int L, bool vec, const float2 (&v)[P]) {
  constexpr int V = 16 / sizeof(T);
  const int lane = threadIdx.x & 31;
  if (vec) {
#pragma unroll
    for (int u = 0; u < D / 2; ++u) {
      const int e = (u * 32 + lane) * V;
      if (e < L)
        __stcg(reinterpret_cast<float4*>(row + e),
               make_float4(v[OFF + 2 * u].x, v[OFF + 2 * u].y, v[OFF + 2 * u + 1].x, v[OFF + 2 * u + 1].y));
    }
  } else {
#pragma unroll
    for (int u = 0; u < D; ++u) {
      const int e = ((u / 2) * 32 + lane) * V + (u & 1) * (V / 2);
      if constexpr (traits<T>::is_complex) {
        if (e < L) __stcg(reinterpret_cast<float2*>(row + e), v[OFF + u]);
      } else {
        if (e < L) __stcg(reinterpret_cast<float*>(row) + e, v[OFF + u].x);
        if (e + 1 < L) __stcg(reinterpret_cast<float*>(row) + e + 1, v[OFF + u].y);
      }
    }
  }
}

// Step counters: the store publishes what the warp stored before it, the load takes
// what was published (rows are read through L2, so no fence follows it).
__device__ __forceinline__ void j32_publish(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned j32_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// A warp waits until a row's counter has reached `step`; false on error / timeout.
__device__ __forceinline__ bool j32_wait_row(const unsigned* counter, unsigned step, SyncWords* sw) {
  int good = 1;
  if ((threadIdx.x & 31) == 0) {
    const long long limit = spin_limit();
    for (long long spins = 0; j32_acquire(counter) < step; ++spins) {
      if (ld_volatile(&sw->err)) { good = 0; break; }
      if (spins > limit) { atomicCAS(&sw->err, 0, TNC_ERR_TIMEOUT); good = 0; break; }
    }
  }
  good = __shfl_sync(0xffffffffu, good, 0);
  __syncwarp();
  return good != 0;
}

struct J32Args {
  void *W, *J;  // rows of L elements each (J: ACC only)
  int nr, L, h, N, kb, max_sweeps, vec;  // N: half-blocks, padded to even; kb: half-blocks with kept rows
  float rtol, stol;
  int staged;  // stop after a sweep without a rotation above stol
  const double* frob2;
  float* Dn;  // squared row norms between rounds
  unsigned *counters, *ver;
  SyncWords* sw;
  int* info;
};

// E elements a lane of a row of W (and as many of J's with ACC).
template <typename T, int E, bool ACC, int MAXT>
__global__ void __launch_bounds__(MAXT, (MAXT == 256 && E * sizeof(T) * (ACC ? 2 : 1) <= 128) ? 2 : 1)
jacobi32_kernel(const J32Args p) {
  constexpr bool CPLX = traits<T>::is_complex;
  constexpr int D = E * (int)sizeof(T) / 8, P = ACC ? 2 * D : D;  // float2 pairs of W, of the whole row
  extern __shared__ __align__(16) unsigned char j32_smem[];
  float4* sL = reinterpret_cast<float4*>(j32_smem);  // [h] rows of 16 P floats x 32 lanes
  float4* sR = sL + (size_t)p.h * (P / 2) * 32;
  __shared__ float nL[16], nR[16];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = p.h, N = p.N, nb = (p.nr + h - 1) / h, cta = blockIdx.x;
  const bool vec = p.vec != 0;
  T* W = static_cast<T*>(p.W);
  T* J = static_cast<T*>(p.J);
  const float noise2 = noise_floor2<T>(p.frob2);
  constexpr int kRow = (P / 2) * 32;  // float4s of a row
  float2 x[P], y[P];
  float an = 0.f;
  bool ok = true;
  int sweep = 0;
  bool converged = false, staged = false;
  unsigned last_rot = 0;

  auto load_row = [&](int row, float2 (&v)[P]) {
    j32_ldg<T, P, D, 0>(W + (int64_t)row * p.L, p.L, vec, v);
    if constexpr (ACC) j32_ldg<T, P, D, D>(J + (int64_t)row * p.L, p.L, vec, v);
  };
  // store a row, then its step counter (one warp)
  auto give_row = [&](int row, const float2 (&v)[P], float n2, unsigned step) {
    j32_stg<T, P, D, 0>(W + (int64_t)row * p.L, p.L, vec, v);
    if constexpr (ACC) j32_stg<T, P, D, D>(J + (int64_t)row * p.L, p.L, vec, v);
    if (lane == 0) __stcg(p.Dn + row, n2);
    __syncwarp();
    if (lane == 0) j32_publish(p.ver + row, step);
  };
  auto take_row = [&](int row, unsigned step) { ok = ok && j32_wait_row(p.ver + row, step, p.sw); };
  // rotate the pair (x, y); returns 0, 1 or 3 (above stol), the norms moved by *th
  auto rotate = [&](float a, float b, float2 (&xx)[P], float2 (&yy)[P], float& th) -> int {
    float re, im;
    j32_dot<CPLX, P, D>(xx, yy, re, im);
    re = warp_sum(re);
    if constexpr (CPLX) im = warp_sum(im);
    Rot<T> r;
    if constexpr (CPLX) r = make_rot<T>(a, b, T(re, im), p.rtol, noise2, p.stol);
    else r = make_rot<T>(a, b, re, p.rtol, noise2, p.stol);
    if (!r.apply) return 0;
    float sei = 0.f;
    if constexpr (CPLX) sei = r.se.im;
    j32_rotate<CPLX, P>(xx, yy, r.c, real_(r.se), sei);
    th = r.th;
    return r.big ? 3 : 1;
  };
  // half-block at position q and time t (mod 2N), moving right or left
  auto mover = [&](int q, int t) {
    int c = q - t;
    if (c < 0) c += 2 * N;
    return c < N ? c : 2 * N - 1 - c;
  };

  for (; sweep < p.max_sweeps; ++sweep) {
    unsigned rot = 0, rotb = 0;
    const unsigned t0 = (unsigned)sweep * (unsigned)N;
    const int base = (sweep & 1) * N;  // t0 mod 2N
    // phase 0; the grid barrier before it has ordered every earlier store
    int hR = mover(2 * cta, base), hL = mover(2 * N - 1 - (2 * cta + 1), base);
    {
      const int rowR = hR * h + warp, rowL = hL * h + warp;
      const bool inR = hR < nb && rowR < p.nr, inL = hL < nb && rowL < p.nr;
#pragma unroll
      for (int u = 0; u < P; ++u) x[u] = y[u] = make_float2(0.f, 0.f);
      if (inR) load_row(rowR, x);
      if (inL) load_row(rowL, y);
      float s = 0.f, t = 0.f;
#pragma unroll
      for (int u = 0; u < D; ++u) {
        s = fmaf(x[u].x, x[u].x, s);
        s = fmaf(x[u].y, x[u].y, s);
        t = fmaf(y[u].x, y[u].x, t);
        t = fmaf(y[u].y, y[u].y, t);
      }
      s = warp_sum(s);
      t = warp_sum(t);
      j32_sts<P>(sR + warp * kRow, x);
      j32_sts<P>(sL + warp * kRow, y);
      if (lane == 0) { nR[warp] = s; nL[warp] = t; }
      __syncthreads();
      // warps [0, h / 2) take the pairs of R, the others those of L
      const bool left = warp >= h / 2;
      const int pw = left ? warp - h / 2 : warp, blk = left ? hL : hR;
      float4* sb = left ? sL : sR;
      float* nn = left ? nL : nR;
      const int cnt = blk < nb && blk < p.kb ? ((p.nr - blk * h) < h ? p.nr - blk * h : h) : 0;
      for (int r = 0; r < h - 1; ++r) {
        const int mod = h - 1;
        int a = r, b = mod;
        if (pw) { a = (r + pw) % mod; b = (r - pw + mod) % mod; }
        if (pw < h / 2 && a < cnt && b < cnt) {
          j32_lds<P>(sb + a * kRow, x);
          j32_lds<P>(sb + b * kRow, y);
          const float na = nn[a], nc = nn[b];
          float th = 0.f;
          const int k = rotate(na, nc, x, y, th);
          if (k) {
            j32_sts<P>(sb + a * kRow, x);
            j32_sts<P>(sb + b * kRow, y);
            __syncwarp();
            if (lane == 0) { nn[a] = na - th; nn[b] = nc + th; }
          }
          rot += (unsigned)(k & 1);
          rotb += (unsigned)(k >> 1);
        }
        __syncthreads();
      }
      j32_lds<P>(sR + warp * kRow, x);
      an = nR[warp];
    }
    // rounds
    for (int r = 0; r < N; ++r) {
      const bool odd = (r & 1) != 0, active = !odd || cta < N / 2 - 1;
      const int q = 2 * cta + (odd ? 1 : 0), tm = base + r;
      const int idR = active ? mover(q, tm) : -1, idL = active ? mover(2 * N - 2 - q, tm) : -1;
      if (r > 0) {
        const unsigned step = t0 + (unsigned)r;
        if (hL != idL) {
          if (hL >= 0 && hL < nb && hL * h + warp < p.nr) {
            j32_lds<P>(sL + warp * kRow, y);
            give_row(hL * h + warp, y, nL[warp], step);
          }
        }
        if (hR != idR) {
          if (hR >= 0 && hR < nb && hR * h + warp < p.nr) give_row(hR * h + warp, x, an, step);
        }
        // a half-block that stood at an end of the line was given a round earlier
        if (hL != idL && idL >= 0 && idL < nb && idL * h + warp < p.nr) {
          const int row = idL * h + warp;
          take_row(row, step - (!odd && cta == N / 2 - 1 ? 1u : 0u));
          load_row(row, y);
          j32_sts<P>(sL + warp * kRow, y);
          if (lane == 0) nL[warp] = __ldcg(p.Dn + row);
          __syncwarp();
        }
        if (hR != idR && idR >= 0 && idR < nb && idR * h + warp < p.nr) {
          const int row = idR * h + warp;
          take_row(row, step - (!odd && cta == 0 ? 1u : 0u));
          load_row(row, x);
          an = __ldcg(p.Dn + row);
        }
        hR = idR;
        hL = idL;
      }
      if (!active || hR >= nb || hL >= nb || (hR >= p.kb && hL >= p.kb)) continue;
      const bool inR = hR * h + warp < p.nr;
      const int cntL = (p.nr - hL * h) < h ? p.nr - hL * h : h;
      for (int s = 0; s < h; ++s) {
        const int j = (warp + s) & (h - 1);
        if (inR && j < cntL) {
          const float b = nL[j];
          j32_lds<P>(sL + j * kRow, y);
          float th = 0.f;
          const int k = rotate(an, b, x, y, th);
          if (k) {
            j32_sts<P>(sL + j * kRow, y);
            __syncwarp();
            if (lane == 0) nL[j] = b + th;
            an -= th;
          }
          rot += (unsigned)(k & 1);
          rotb += (unsigned)(k >> 1);
        }
        __syncthreads();
      }
    }
    {  // every half-block back to memory
      const unsigned step = t0 + (unsigned)N;
      if (hL >= 0 && hL < nb && hL * h + warp < p.nr) {
        j32_lds<P>(sL + warp * kRow, y);
        give_row(hL * h + warp, y, nL[warp], step);
      }
      if (hR >= 0 && hR < nb && hR * h + warp < p.nr) give_row(hR * h + warp, x, an, step);
    }
    if (lane == 0 && rot) atomicAdd(&p.counters[sweep], rot);
    if (lane == 0 && rotb) atomicAdd(&p.counters[kJ32MaxSweeps + sweep], rotb);
    if (!__syncthreads_and(ok) || !grid_barrier(p.sw, gridDim.x)) return;
    last_rot = ld_volatile(&p.counters[sweep]);
    if (last_rot == 0) { converged = true; ++sweep; break; }
    if (p.staged && ld_volatile(&p.counters[kJ32MaxSweeps + sweep]) == 0) { staged = true; ++sweep; break; }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    p.info[0] = (converged || staged) ? TNC_OK : TNC_ERR_NOT_CONVERGED;
    p.info[1] = sweep;
    p.info[2] = (int)last_rot;
    p.info[3] = staged ? 1 : 0;
  }
}

}  // namespace tnc
