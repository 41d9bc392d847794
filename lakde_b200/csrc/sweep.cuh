// Shared core of the dense kernels x points sweeps on the FP32 / FP64 pipes
// (chol_quad_form, the predictive density and its backward): a CTA keeps P
// points per thread and walks a chunk of kernels whose packed factors are
// staged two groups deep in shared memory by element-wise cp.async, so the
// next group's loads run under this group's arithmetic.
//
//   y_i = sum_{j <= i} U[j][i] (x_m[j] - x_n[j]),  Q = sum_i y_i^2,  U = W_triu_n
//
// What bounds it is the broadcast shared-memory read of U against the FMA
// pipe: one 16-byte read feeds 4 P float FMAs.  Measured on the B200, FMA rate
// of that loop with 1 / 2 / 4 points per thread: 34 / 51 / 62 TFLOP/s, and 37 /
// 58 / 64 with the column pair (i, i + 1) packed into one fma.rn.f32x2 (half
// the issue slots; the FMA pipe itself peaks at 72-74 either way).  So: four
// points at DP <= 16, two above, packed pairs for float32, one point for
// float64 above 16 dimensions (a 16-byte read feeds two DFMAs of two cycles
// each).  Every y_i and Q is accumulated in ascending order by itself, so the
// result does not depend on P or on the packing.
//
// Up to 32 dimensions the loop over (j, i) is unrolled with the points in
// registers.  Above that the unrolled body (2,080 FMAs and 544 loads at 64)
// does not fit the instruction cache, so the columns go in two blocks through a
// rolled loop over j, the points in a shared-memory column of their own.
#pragma once

#include "common.cuh"

namespace lakde {
namespace sweep {

constexpr int THREADS = 128;

template <typename T, int DP, bool ROLL = (DP > 32)>
struct Cfg {
  static constexpr bool ROLLED = ROLL;
  static constexpr int V = 16 / (int)sizeof(T);
  static constexpr int DPV = DP < V ? V : DP;  // columns of the packed layout
  static constexpr int CB = DP / 2;            // columns of a block (rolled layout: two blocks)
  static constexpr int P = sizeof(T) == 4 ? (DP <= 16 ? 4 : 2) : (DP <= 16 ? 2 : 1);
  static constexpr int TILE = THREADS * P;  // points per CTA
  // floats of the packed factor of one kernel
  static constexpr int US = ROLLED ? 3 * CB * CB : V * (DPV / V) * (DPV + V) / 2;
  static constexpr int X0 = US;         // centre (DPV)
  static constexpr int S0 = US + DPV;   // two scalars of the kernel
  static constexpr int KS = US + DPV + V;
  // kernels per staged group: about 20 KB a stage (a CTA synchronises twice per group)
  static constexpr int KT = ROLLED ? 1 : (DP <= 8 ? 32 : DP <= 16 ? 16 : 8);
  static constexpr size_t ybytes = ROLLED ? (size_t)DP * TILE * sizeof(T) : 0;
  static constexpr size_t smem = 2 * (size_t)KT * KS * sizeof(T) + ybytes;
  // resident CTAs an SM is asked for (the registers then fit).  The rolled form's
  // two fit the shared memory but for float64 at 64 dimensions, whose 115,744
  // bytes leave one (32 bytes too many), and the chunk rules count two there
  static constexpr int OCC = ROLLED ? 2 : sizeof(T) == 4 ? (DP <= 8 ? 4 : 3) : (DP <= 8 ? 4 : 3);

  // Element (j, i), j <= i, of the packed factor: row j from column V (j / V)
  // on, rows one after the other; rolled: block c = i / CB holds rows 0 ..
  // CB (c + 1) - 1 of its CB columns.
  __host__ __device__ static constexpr int at(int j, int i) {
    if (ROLLED) {
      const int c = i / CB;
      return c * CB * CB + j * CB + i - c * CB;
    }
    const int q = j / V, r = j % V;
    return V * (q * DPV - V * q * (q - 1) / 2) + r * (DPV - V * q) + i - V * q;
  }
};

template <typename T>
__device__ __forceinline__ void cp_async_elem(T *dst, const T *src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if constexpr (sizeof(T) == 4)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Issues the copies of kernels n0 .. n0 + cnt - 1 into a stage (upper triangle
// and centre; the padding of the stage stays zero).
template <typename T, int DP, typename C = Cfg<T, DP>>
__device__ __forceinline__ void stage_kernels(T *__restrict__ dst, const T *__restrict__ W, int64_t ws0, int64_t ws1,
                                              int64_t ws2, const T *__restrict__ Xn, int64_t xs0, int64_t xs1,
                                              int64_t n0, int cnt, int D, int tid) {
  // thread: column i of RPP rows apart, so addresses only step
  constexpr int LW = DP <= 2 ? 2 : DP <= 4 ? 4 : DP <= 8 ? 8 : DP <= 16 ? 16 : DP <= 32 ? 32 : 64;
  constexpr int RPP = THREADS / LW;
  const int i = tid & (LW - 1), r = tid / LW;
  if constexpr (RPP >= DP) {
    // RPP / DP kernels a pass, one element each (RPP and DP are powers of two here)
    const int j = r % DP;
    if (i < D && j <= i) {
      const int at = C::at(j, i);
      const T *src = W + (n0 + r / DP) * ws0 + j * ws1 + i * ws2;
      for (int k = r / DP; k < cnt; k += RPP / DP, src += (RPP / DP) * ws0) cp_async_elem(dst + k * C::KS + at, src);
    }
  } else if (i < D) {
    for (int k = 0; k < cnt; ++k) {
      const T *src = W + (n0 + k) * ws0 + r * ws1 + i * ws2;
      T *d = dst + k * C::KS;
      for (int j = r; j <= i; j += RPP, src += RPP * ws1) cp_async_elem(d + C::at(j, i), src);
    }
  }
  for (int f = tid; f < cnt * DP; f += THREADS) {
    const int d = f % DP, k = f / DP;
    if (d < D) cp_async_elem(dst + k * C::KS + C::X0 + d, Xn + (n0 + k) * xs0 + d * xs1);
  }
}

// Accumulators of two adjacent columns.
template <typename T>
struct Pair {
  T a, b;
  __device__ __forceinline__ void zero() { a = b = T(0); }
  __device__ __forceinline__ void fma2(const T *u, T d) {
    a = fma(u[0], d, a);
    b = fma(u[1], d, b);
  }
  __device__ __forceinline__ void fma_hi(const T *u, T d) { b = fma(u[1], d, b); }
  __device__ __forceinline__ T lo() const { return a; }
  __device__ __forceinline__ T hi() const { return b; }
};
template <>
struct Pair<float> {
  unsigned long long v;
  __device__ __forceinline__ void zero() { v = 0ull; }
  __device__ __forceinline__ void fma2(const float *u, float d) {
    unsigned long long uu, dd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(uu) : "f"(u[0]), "f"(u[1]));
    asm("mov.b64 %0, {%1, %1};" : "=l"(dd) : "f"(d));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(uu), "l"(dd));
  }
  __device__ __forceinline__ void fma_hi(const float *u, float d) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    y = fmaf(u[1], d, y);
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  }
  __device__ __forceinline__ float lo() const {
    return __uint_as_float((unsigned)v);
  }
  __device__ __forceinline__ float hi() const {
    return __uint_as_float((unsigned)(v >> 32));
  }
};

template <typename T>
__device__ __forceinline__ void load_vec(const T *p, T (&u)[16 / sizeof(T)]) {
  using VT = typename Vec<T>::type;
  const VT w = *reinterpret_cast<const VT *>(p);
  const T *s = reinterpret_cast<const T *>(&w);
#pragma unroll
  for (int k = 0; k < (int)(16 / sizeof(T)); ++k) u[k] = s[k];
}

// y_i of P points for one staged kernel, all DP columns (unrolled form);
// coordinate j of point p is coord(p, j).  C: layout of the staged factor.
template <typename C, typename T, int DP, int P, typename F>
__device__ __forceinline__ void products(const T *__restrict__ sk, F &&coord, Pair<T> (&acc)[P][(DP + 1) / 2]) {
  constexpr int V = C::V;
#pragma unroll
  for (int p = 0; p < P; ++p)
#pragma unroll
    for (int e = 0; e < (DP + 1) / 2; ++e) acc[p][e].zero();
  T xv[V];
#pragma unroll
  for (int j = 0; j < DP; ++j) {
    // bounds how far the loads are hoisted (registers)
    if (j % 4 == 0) asm volatile("" ::: "memory");
    if (j % V == 0) load_vec<T>(sk + C::X0 + j, xv);
    T dl[P];
#pragma unroll
    for (int p = 0; p < P; ++p) dl[p] = coord(p, j) - xv[j % V];
#pragma unroll
    for (int i0 = V * (j / V); i0 < C::DPV; i0 += V) {
      T u[V];
      load_vec<T>(sk + C::at(j, i0), u);
#pragma unroll
      for (int v = 0; v < V; v += 2) {
        const int i = i0 + v;
        if (i + 1 < j || i >= DP) continue;  // j > i + 1: both below the diagonal
#pragma unroll
        for (int p = 0; p < P; ++p) {
          if (i >= j)
            acc[p][i / 2].fma2(u + v, dl[p]);
          else
            acc[p][i / 2].fma_hi(u + v, dl[p]);
        }
      }
    }
  }
}

template <typename T, int DP, int P>
__device__ __forceinline__ void squares(const Pair<T> (&acc)[P][(DP + 1) / 2], T (&q)[P]) {
#pragma unroll
  for (int p = 0; p < P; ++p) {
    q[p] = T(0);
#pragma unroll
    for (int e = 0; e < (DP + 1) / 2; ++e) {
      q[p] = fma(acc[p][e].lo(), acc[p][e].lo(), q[p]);
      if (2 * e + 1 < DP) q[p] = fma(acc[p][e].hi(), acc[p][e].hi(), q[p]);
    }
  }
}

// Q of P points, CB columns at a time; the points' coordinates at ys + d TILE
// + p (this thread's shared-memory column).
template <typename T, int DP, int P>
__device__ __forceinline__ void quad_rolled(const T *__restrict__ sk, const T *__restrict__ ys, int D, T (&q)[P]) {
  using C = Cfg<T, DP>;
  constexpr int V = C::V, CB = C::CB;
#pragma unroll
  for (int p = 0; p < P; ++p) q[p] = T(0);
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    const T *u0 = sk + c * CB * CB;
    Pair<T> acc[P][CB / 2];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int e = 0; e < CB / 2; ++e) acc[p][e].zero();
#pragma unroll 1
    for (int j0 = 0; j0 < c * CB; j0 += V) {
      T xv[V];
      load_vec<T>(sk + C::X0 + j0, xv);
#pragma unroll
      for (int jj = 0; jj < V; ++jj) {
        const int j = j0 + jj;
        T dl[P];
#pragma unroll
        for (int p = 0; p < P; ++p) dl[p] = ys[j * C::TILE + p] - xv[jj];
#pragma unroll
        for (int i = 0; i < CB; i += V) {
          T u[V];
          load_vec<T>(u0 + j * CB + i, u);
#pragma unroll
          for (int v = 0; v < V; v += 2)
#pragma unroll
            for (int p = 0; p < P; ++p) acc[p][(i + v) / 2].fma2(u + v, dl[p]);
        }
      }
    }
    // the diagonal block
    T xv[V];
#pragma unroll
    for (int jj = 0; jj < CB; ++jj) {
      const int j = c * CB + jj;
      if (jj % V == 0) load_vec<T>(sk + C::X0 + j, xv);
      T dl[P];
#pragma unroll
      for (int p = 0; p < P; ++p) dl[p] = ys[j * C::TILE + p] - xv[jj % V];
#pragma unroll
      for (int i0 = V * (jj / V); i0 < CB; i0 += V) {
        T u[V];
        load_vec<T>(u0 + j * CB + i0, u);
#pragma unroll
        for (int v = 0; v < V; v += 2) {
          const int i = i0 + v;
          if (i + 1 < jj) continue;
#pragma unroll
          for (int p = 0; p < P; ++p) {
            if (i >= jj)
              acc[p][i / 2].fma2(u + v, dl[p]);
            else
              acc[p][i / 2].fma_hi(u + v, dl[p]);
          }
        }
      }
    }
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int e = 0; e < CB / 2; ++e) {
        q[p] = fma(acc[p][e].lo(), acc[p][e].lo(), q[p]);
        q[p] = fma(acc[p][e].hi(), acc[p][e].hi(), q[p]);
      }
  }
}

// The P points of a thread: registers (unrolled form) or its shared-memory
// column (rolled form).  Point p of thread t is point t + p THREADS of the tile.
template <typename T, int DP>
struct Points {
  using C = Cfg<T, DP>;
  static constexpr int R = C::ROLLED ? 1 : DP;
  T y[C::P][R];
  T *col;

  __device__ __forceinline__ void load(const T *__restrict__ X, int64_t s0, int64_t s1, int64_t m0, int64_t M, int D,
                                       T *ys, int tid) {
    col = ys + tid * C::P;
#pragma unroll
    for (int p = 0; p < C::P; ++p) {
      const int64_t m = m0 + tid + (int64_t)p * THREADS;
      if constexpr (C::ROLLED) {
#pragma unroll 8
        for (int d = 0; d < DP; ++d) col[d * C::TILE + p] = (m < M && d < D) ? X[m * s0 + d * s1] : T(0);
      } else {
#pragma unroll
        for (int d = 0; d < DP; ++d) y[p][d] = (m < M && d < D) ? X[m * s0 + d * s1] : T(0);
      }
    }
  }

  __device__ __forceinline__ void quad(const T *__restrict__ sk, int D, T (&q)[C::P]) const {
    if constexpr (C::ROLLED) {
      quad_rolled<T, DP, C::P>(sk, col, D, q);
    } else {
      Pair<T> acc[C::P][(DP + 1) / 2];
      products<C, T, DP, C::P>(sk, [&](int p, int j) { return y[p][j]; }, acc);
      squares<T, DP, C::P>(acc, q);
    }
  }
};

// Zeroes what a chunk of `kernels` will stage of both stages once: the padding
// is never written again.
template <typename T, typename C, int KT = C::KT>
__device__ __forceinline__ void clear_stages(T *st, int64_t kernels, int tid) {
  static_assert(C::KS % C::V == 0, "whole 16-byte vectors");
  const int end = (int)(kernels < 2 * KT ? kernels : 2 * KT) * C::KS;
  using VT = typename Vec<T>::type;
  VT zero;
  T *z = reinterpret_cast<T *>(&zero);
#pragma unroll
  for (int k = 0; k < C::V; ++k) z[k] = T(0);
  for (int e = tid * C::V; e < end; e += THREADS * C::V) *reinterpret_cast<VT *>(st + e) = zero;
}

// Kernels per CTA so that tiles x chunks is about `ctas`; whole groups of kt
// once a chunk is longer than one.
inline int64_t chunk_len(int64_t N, int64_t tiles, int64_t ctas, int kt) {
  int64_t nchunks = (ctas + tiles - 1) / tiles;
  if (nchunks < 1) nchunks = 1;
  const int64_t chunk = (N + nchunks - 1) / nchunks;
  return chunk > kt ? ((chunk + kt - 1) / kt) * kt : (chunk < 1 ? 1 : chunk);
}

// out[q] = -log N + logsumexp over the chunks' (max, sum) partials [nchunks, Nq]:
// 32 queries a block (coalesced reads), eight threads dealing a query's chunks
// between them (one thread walking all of them waited on its own loads: 72 us
// at 148 chunks x 5,000 queries).
template <typename T>
__global__ void __launch_bounds__(256) fold_kernel(const T *__restrict__ ws_m, const T *__restrict__ ws_s,
                                                   T *__restrict__ out, int64_t Nq, int64_t nchunks, T log_n) {
  constexpr int G = 8;
  __shared__ T sm[G][32], ss[G][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int64_t q = blockIdx.x * (int64_t)32 + lane;
  T m = neg_inf<T>();
  if (q < Nq) {
#pragma unroll 4
    for (int64_t c = g; c < nchunks; c += G) m = fmax(m, ws_m[c * Nq + q]);
  }
  sm[g][lane] = m;
  __syncthreads();
  T M = sm[0][lane];
#pragma unroll
  for (int k = 1; k < G; ++k) M = fmax(M, sm[k][lane]);
  T s = T(0);
  if (q < Nq && M != neg_inf<T>()) {
#pragma unroll 4
    for (int64_t c = g; c < nchunks; c += G) s += ws_s[c * Nq + q] * exp(ws_m[c * Nq + q] - M);
  }
  ss[g][lane] = s;
  __syncthreads();
  if (g != 0 || q >= Nq) return;
  T S = T(0);
#pragma unroll
  for (int k = 0; k < G; ++k) S += ss[k][lane];
  out[q] = (M == neg_inf<T>()) ? M : (M + log(S)) - log_n;
}

}  // namespace sweep
}  // namespace lakde
