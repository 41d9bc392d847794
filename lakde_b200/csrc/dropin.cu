// The three ops of the reference extension, rewritten for sm_100a:
//   ind2ptr         — CSR row pointers by per-row binary search
//   chol_quad_form  — dense Cholesky quad forms (the sweep of sweep.cuh)
//   W_inv           — CSR responsibility-weighted scatter covariance (M-step)
#include "common.cuh"
#include "factor_dmma.cuh"
#include "sweep.cuh"

namespace lakde {

// ---------------------------------------------------------------------------
// ind2ptr: out[i] = #{p : ind[p] < i}.  One thread per output entry, binary
// search over the sorted index vector; reads stay inside [0, nnz).
// ---------------------------------------------------------------------------
template <typename I, typename P>
__global__ void ind2ptr_kernel(const I *__restrict__ ind, int64_t nnz, int64_t M, P *__restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= M;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = 0, hi = nnz;
    while (lo < hi) {
      int64_t mid = (lo + hi) >> 1;
      if ((int64_t)ind[mid] < i)
        lo = mid + 1;
      else
        hi = mid;
    }
    out[i] = (P)lo;
  }
}

// ---------------------------------------------------------------------------
// Dense quad form: the kernels x points sweep of sweep.cuh, each Q written to
// out[n, m] (consecutive threads: consecutive points).  512 kernels x 20,011
// points, float32: d = 63 3.33 -> 1.00 ms (43 TFLOP/s), d = 21 289 -> 184 us
// against one point per thread with the factors loaded between barriers;
// float64 d = 63 6.17 -> 3.9 ms.
// ---------------------------------------------------------------------------
template <typename T, int DP>
__global__ void __launch_bounds__(sweep::THREADS, sweep::Cfg<T, DP>::OCC) quad_dense_kernel(
    const T *__restrict__ W, int64_t ws0, int64_t ws1, int64_t ws2, const T *__restrict__ Xn, int64_t xns0,
    int64_t xns1, const T *__restrict__ Xm, int64_t xms0, int64_t xms1, T *__restrict__ out, int64_t os0, int64_t os1,
    int64_t N, int64_t M, int D, int64_t chunk, int64_t m_tiles) {
  using C = sweep::Cfg<T, DP>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *st = reinterpret_cast<T *>(smem_raw);
  const int tid = threadIdx.x;
  const int64_t m0 = (blockIdx.x % m_tiles) * C::TILE;
  const int64_t n_begin = (blockIdx.x / m_tiles) * chunk;
  const int64_t n_end = (n_begin + chunk < N) ? n_begin + chunk : N;
  auto count = [&](int64_t n0) { return (int)((n_end - n0) < C::KT ? (n_end - n0) : C::KT); };
  sweep::clear_stages<T, C>(st, n_end - n_begin, tid);
  __syncthreads();
  sweep::stage_kernels<T, DP>(st, W, ws0, ws1, ws2, Xn, xns0, xns1, n_begin, count(n_begin), D, tid);
  sweep::cp_async_commit();
  sweep::Points<T, DP> pts;
  pts.load(Xm, xms0, xms1, m0, M, D, st + 2 * C::KT * C::KS, tid);
  int s = 0;
  for (int64_t n0 = n_begin; n0 < n_end; n0 += C::KT, s ^= 1) {
    const int64_t nn = n0 + C::KT;
    if (nn < n_end)
      sweep::stage_kernels<T, DP>(st + (s ^ 1) * C::KT * C::KS, W, ws0, ws1, ws2, Xn, xns0, xns1, nn, count(nn), D,
                                  tid);
    sweep::cp_async_commit();
    sweep::cp_async_wait<1>();
    __syncthreads();
    const int cnt = count(n0);
    for (int k = 0; k < cnt; ++k) {
      T q[C::P];
      pts.quad(st + (s * C::KT + k) * C::KS, D, q);
#pragma unroll
      for (int p = 0; p < C::P; ++p) {
        const int64_t m = m0 + tid + (int64_t)p * sweep::THREADS;
        if (m < M) out[(n0 + k) * os0 + m * os1] = q[p];
      }
    }
    __syncthreads();  // the stage is refilled in the next iteration
  }
}

// ---------------------------------------------------------------------------
// Scatter covariance, small D (<= 16): one warp per kernel row.  Pairs are
// staged 32 at a time as centred differences in the warp's shared slice;
// every lane owns up to 5 entries of the lower triangle.
// ---------------------------------------------------------------------------
template <typename T, typename RP, typename CI, int DP>
__global__ void __launch_bounds__(256) scatter_cov_warp(const RP *__restrict__ rowptr, const CI *__restrict__ col,
                                                        const T *__restrict__ val, const T *__restrict__ Xn,
                                                        const T *__restrict__ Xm, T *__restrict__ out, int64_t N,
                                                        int64_t M, int D, T *__restrict__ nu_out, T nu0) {
  constexpr int TT = DP * (DP + 1) / 2;
  constexpr int KE = (TT + 31) / 32;
  __shared__ T sd[8][32][DP + 1];
  __shared__ T sv[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 8 + warp;
  if (row >= N) return;

  int ei[KE], ej[KE];
  {
    int e = 0;
#pragma unroll
    for (int k = 0; k < KE; ++k) ei[k] = ej[k] = -1;
    for (int i = 0; i < DP; ++i)
      for (int j = 0; j <= i; ++j, ++e)
        if ((e & 31) == lane && (e >> 5) < KE) {
          ei[e >> 5] = i;
          ej[e >> 5] = j;
        }
  }
  const int64_t start = (int64_t)rowptr[row], end = (int64_t)rowptr[row + 1];
  bool bad = end < start;
  T acc[KE];
#pragma unroll
  for (int k = 0; k < KE; ++k) acc[k] = T(0);
  T vsum = T(0);

  for (int64_t base = start; base < end; base += 32) {
    const int64_t p = base + lane;
    const bool valid = p < end;
    int64_t c = valid ? (int64_t)col[p] : 0;
    T v = valid ? val[p] : T(0);
    if (valid && (c < 0 || c >= M)) {
      bad = true;
      c = 0;
      v = T(0);
    }
#pragma unroll
    for (int d = 0; d < DP; ++d)
      sd[warp][lane][d] = (valid && d < D) ? Xm[c * D + d] - Xn[row * D + d] : T(0);
    sv[warp][lane] = v;
    vsum += v;
    __syncwarp();
    const int cnt = (int)((end - base) < 32 ? (end - base) : 32);
    for (int q = 0; q < cnt; ++q) {
      const T vq = sv[warp][q];
#pragma unroll
      for (int k = 0; k < KE; ++k) {
        if (ei[k] >= 0) {
          const T di = sd[warp][q][ei[k]];
          const T dj = sd[warp][q][ej[k]];
          acc[k] = fma(vq * di, dj, acc[k]);
        }
      }
    }
    __syncwarp();
  }
  bad = __any_sync(0xffffffffu, bad);
  if (nu_out) {
    vsum = warp_sum(vsum);
    if (lane == 0) nu_out[row] = bad ? T(NAN) : nu0 + vsum;
  }
  T *o = out + row * (int64_t)D * D;
#pragma unroll
  for (int k = 0; k < KE; ++k) {
    const int i = ei[k], j = ej[k];
    if (i >= 0 && i < D) {
      const T v = bad ? T(NAN) : acc[k];
      o[i * D + j] = v;
      o[j * D + i] = v;
    }
  }
}

// ---------------------------------------------------------------------------
// Scatter covariance in float32, D in (16, 64]: one CTA per kernel row; each thread owns
// one 4x4 block of the lower triangle and updates it from 64-pair chunks of
// centred differences staged in shared memory (two 16-byte loads per pair).
// ---------------------------------------------------------------------------
template <typename T, int DP>
struct CtaScatterCfg {
  static constexpr int NB = DP / 4;
  static constexpr int NBLK = NB * (NB + 1) / 2;
  static constexpr int THREADS = ((NBLK + 31) / 32) * 32;
  static constexpr int CH = 64;
  static constexpr int LD = DP + 4;
  static constexpr size_t smem = (size_t)CH * LD * sizeof(T) + CH * sizeof(T) + CH * sizeof(int64_t) +
                                 DP * sizeof(T);
};

template <typename T, typename RP, typename CI, int DP>
__global__ void scatter_cov_cta(const RP *__restrict__ rowptr, const CI *__restrict__ col,
                                const T *__restrict__ val, const T *__restrict__ Xn, const T *__restrict__ Xm,
                                T *__restrict__ out, int64_t N, int64_t M, int D, T *__restrict__ nu_out,
                                T nu0) {
  using C = CtaScatterCfg<T, DP>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *sd = reinterpret_cast<T *>(smem_raw);
  T *sv = sd + C::CH * C::LD;
  int64_t *sc = reinterpret_cast<int64_t *>(sv + C::CH);
  T *sxn = reinterpret_cast<T *>(sc + C::CH);
  __shared__ int s_bad;

  const int64_t row = blockIdx.x;
  const int tid = threadIdx.x;
  int bi = -1, bj = -1;
  {
    int e = 0;
    for (int i = 0; i < C::NB; ++i)
      for (int j = 0; j <= i; ++j, ++e)
        if (e == tid) {
          bi = i;
          bj = j;
        }
  }
  if (tid == 0) s_bad = 0;
  for (int d = tid; d < DP; d += blockDim.x) sxn[d] = d < D ? Xn[row * D + d] : T(0);
  const int64_t start = (int64_t)rowptr[row], end = (int64_t)rowptr[row + 1];
  __syncthreads();
  if (end < start && tid == 0) s_bad = 1;

  T acc[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q] = T(0);

  T vsum = T(0);  // row sum of the weights, accumulated by thread 0
  for (int64_t base = start; base < end; base += C::CH) {
    const int cnt = (int)((end - base) < C::CH ? (end - base) : C::CH);
    for (int pp = tid; pp < C::CH; pp += blockDim.x) {
      int64_t c = 0;
      T v = T(0);
      if (pp < cnt) {
        c = (int64_t)col[base + pp];
        v = val[base + pp];
        if (c < 0 || c >= M) {
          s_bad = 1;
          c = 0;
          v = T(0);
        }
      }
      sc[pp] = c;
      sv[pp] = v;
    }
    __syncthreads();
    if (tid == 0)
      for (int pp = 0; pp < cnt; ++pp) vsum += sv[pp];
    for (int e = tid; e < C::CH * DP; e += blockDim.x) {
      const int pp = e / DP, d = e % DP;
      sd[pp * C::LD + d] = (pp < cnt && d < D) ? Xm[sc[pp] * D + d] - sxn[d] : T(0);
    }
    __syncthreads();
    if (bi >= 0) {
      for (int pp = 0; pp < cnt; ++pp) {
        const T v = sv[pp];
        T a[4], b[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          a[p] = sd[pp * C::LD + 4 * bi + p];
          b[p] = v * sd[pp * C::LD + 4 * bj + p];
        }
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[p][q] = fma(b[q], a[p], acc[p][q]);
      }
    }
    __syncthreads();
  }
  __syncthreads();
  if (nu_out && tid == 0) nu_out[row] = s_bad ? T(NAN) : nu0 + vsum;
  if (bi < 0) return;
  const bool bad = s_bad != 0;
  T *o = out + row * (int64_t)D * D;
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = 4 * bi + p, j = 4 * bj + q;
      if (i >= D || j > i) continue;
      const T v = bad ? T(NAN) : acc[p][q];
      o[i * D + j] = v;
      o[j * D + i] = v;
    }
}

// ---------------------------------------------------------------------------
// Scatter covariance in float64, D in (16, 64]: one warp per kernel row on the
// FP64 tensor cores, the lower 8 x 8 tiles of S_n in registers.  A step takes
// four pairs: lane l gathers the entries 8 I + l / 4 of pair l % 4's point,
// whose centred differences are the A fragment of row block I and, times the
// weight, the B fragment of column block I, so nothing passes through shared
// memory; the next step's gather is in flight under a step's products.
// Blocks of one warp: with several rows a block, the short ones wait for the
// longest.
//
// Bound by the FP64 tensor pipe (NT (NT + 1) / 2 MMAs of 16 cycles a step) and
// the gather from L2.  20,000 rows of 80 pairs on average at d = 43: 698 -> 259
// us, the tensor pipe 46 % busy (a fifth of the time is the longest rows' tail);
// d = 63 1278 -> 450, d = 24 2211 -> 121 (the CTA form above, whose 4 x 4
// register blocks read both operands from shared memory; it is still the
// float32 form, 417 us at d = 43, and has not been tried against this one there).
// ---------------------------------------------------------------------------
template <typename RP, typename CI, int DP>
__global__ void __launch_bounds__(32, DP <= 32 ? 16 : DP <= 48 ? 12 : 8)
    scatter_cov_mma(const RP *__restrict__ rowptr, const CI *__restrict__ col, const double *__restrict__ val,
                    const double *__restrict__ Xn, const double *__restrict__ Xm, double *__restrict__ out, int64_t M,
                    int D, double *__restrict__ nu_out, double nu0) {
  constexpr int NT = DP / 8;
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x, g = lane >> 2, t = lane & 3;
  const int64_t row = blockIdx.x;
  const int64_t start = (int64_t)rowptr[row], end = (int64_t)rowptr[row + 1];
  bool bad = end < start;

  double xn[NT];
#pragma unroll
  for (int I = 0; I < NT; ++I) xn[I] = 8 * I + g < D ? Xn[row * D + 8 * I + g] : 0.0;
  double c[NT * (NT + 1) / 2][2];
#pragma unroll
  for (int e = 0; e < NT * (NT + 1) / 2; ++e) c[e][0] = c[e][1] = 0.0;
  double vsum = 0.0;

  // pair base + lane of 32: its point (-1: none) and weight; the next 32's are loaded ahead
  int64_t ci = -1, ci1 = -1;
  double v = 0.0, v1 = 0.0;
  auto load_pairs = [&](int64_t base) {
    const int64_t p = base + lane;
    ci1 = -1;
    v1 = 0.0;
    if (p < end) {
      ci1 = (int64_t)col[p];
      v1 = val[p];
    }
  };
  auto take_pairs = [&](int64_t base) {
    ci = ci1;
    v = v1;
    if (base + lane < end && (ci < 0 || ci >= M)) {
      bad = true;
      ci = -1;
      v = 0.0;
    }
    vsum += v;
    load_pairs(base + 32);
  };
  double x[NT], w;
  bool ok;
  auto gather = [&](int s) {  // pairs 4 s .. 4 s + 3 of the 32
    const int64_t cs = __shfl_sync(FULL, ci, 4 * s + t);
    w = __shfl_sync(FULL, v, 4 * s + t);
    ok = cs >= 0;
#pragma unroll
    for (int I = 0; I < NT; ++I) x[I] = ok && 8 * I + g < D ? Xm[cs * D + 8 * I + g] : 0.0;
  };
  if (start < end) {
    load_pairs(start);
    take_pairs(start);
    gather(0);
    for (int64_t p = start; p < end;) {
      double dl[NT], b[NT];
#pragma unroll
      for (int I = 0; I < NT; ++I) {
        dl[I] = ok ? x[I] - xn[I] : 0.0;
        b[I] = w * dl[I];
      }
      p += 4;
      if (p < end) {
        const int s = (int)((p - start) >> 2) & 7;
        if (s == 0) take_pairs(p);
        gather(s);
      }
#pragma unroll
      for (int I = 0; I < NT; ++I)
#pragma unroll
        for (int J = 0; J <= I; ++J) {
          double *t = c[I * (I + 1) / 2 + J];
          dmma::mma(t[0], t[1], dl[I], b[J]);
        }
    }
  }
  bad = __any_sync(FULL, bad);
  if (nu_out) {
    vsum = warp_sum(vsum);
    if (lane == 0) nu_out[row] = bad ? (double)NAN : nu0 + vsum;
  }
  double *o = out + row * (int64_t)D * D;
#pragma unroll
  for (int I = 0; I < NT; ++I)
#pragma unroll
    for (int J = 0; J <= I; ++J)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = 8 * I + g, j = 8 * J + 2 * t + h;
        if (i >= D || j > i) continue;
        const double s = bad ? (double)NAN : c[I * (I + 1) / 2 + J][h];
        o[i * D + j] = s;
        o[j * D + i] = s;
      }
}

template <typename K>
static int set_smem(K kernel, size_t bytes) {
  if (bytes > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) {
      set_error("cudaFuncSetAttribute(%zu bytes): %s", bytes, cudaGetErrorString(e));
      return LAKDE_ECUDA;
    }
  }
  return LAKDE_OK;
}

}  // namespace lakde

using namespace lakde;

extern "C" int lakde_ind2ptr(const void *ind, int ind_dtype, int64_t nnz, int64_t M, void *out, int out_dtype,
                             void *stream) {
  clear_error();
  if (M < 0 || nnz < 0 || !out || (nnz > 0 && !ind)) {
    set_error("ind2ptr: invalid arguments (nnz=%lld, M=%lld)", (long long)nnz, (long long)M);
    return LAKDE_EINVAL;
  }
  if (int st = bind_device("ind2ptr", {out, nnz > 0 ? ind : nullptr})) return st;
  return dispatch_index(ind_dtype, [&](auto i0) {
    using I = decltype(i0);
    return dispatch_index(out_dtype, [&](auto p0) {
      using P = decltype(p0);
      const int threads = 256;
      int64_t blocks = (M + 1 + threads - 1) / threads;
      if (blocks > 148 * 64) blocks = 148 * 64;
      ind2ptr_kernel<I, P><<<(unsigned)blocks, threads, 0, as_stream(stream)>>>(
          static_cast<const I *>(ind), nnz, M, static_cast<P *>(out));
      return check_launch("ind2ptr");
    });
  });
}

extern "C" int lakde_chol_quad_form(int dtype, const void *W_triu, const int64_t *ws, const void *Xn,
                                    const int64_t *xns, const void *Xm, const int64_t *xms, void *out,
                                    const int64_t *os, int64_t N, int64_t M, int64_t D, void *stream) {
  clear_error();
  if (N < 0 || M < 0 || D < 1 || !ws || !xns || !xms || !os) {
    set_error("chol_quad_form: invalid sizes (N=%lld, M=%lld, D=%lld)", (long long)N, (long long)M,
              (long long)D);
    return LAKDE_EINVAL;
  }
  if (N == 0 || M == 0) return LAKDE_OK;
  if (!W_triu || !Xn || !Xm || !out) {
    set_error("chol_quad_form: null pointer");
    return LAKDE_EINVAL;
  }
  if (int st = bind_device("chol_quad_form", {out, W_triu, Xn, Xm})) return st;
  return dispatch_float(dtype, [&](auto t0) {
    using T = decltype(t0);
    return dispatch_dp(D, [&](auto dp) {
      constexpr int DP = decltype(dp)::value;
      using C = sweep::Cfg<T, DP>;
      auto kern = quad_dense_kernel<T, DP>;
      int st = set_smem(kern, C::smem);
      if (st) return st;
      // about six waves of resident CTAs: the last wave costs little, and a
      // CTA still shares its points over its chunk.  Of more than two CTAs an SM
      // at a kernel each, at least eight kernels a CTA while that leaves two
      // CTAs an SM, else four: a CTA's set-up (its points, the first stage, the
      // code's way into the instruction cache) takes as long as several kernels
      // up to 48 dimensions.  us, chunk as by the waves alone / 4 / 8 /
      // 16: float32 512 x 4,096 (chunk 2) at d = 16 48 / 32 / 29 / 27, at d = 8 17 /
      // 12 / 11 / 10; float64 64 x 2,000 (1) at d = 32 41 / 20 / 19 / 32, at d = 48
      // 57 / 36 / 36 / 65; 1,000 x 1 (1) at d = 40 34 / 30 / 33 / 63; 34 x 336 (1) at
      // d = 63 21 / 29.
      const int64_t m_tiles = (M + C::TILE - 1) / C::TILE;
      const int64_t least = m_tiles * N <= 2 * 148 ? 1 : m_tiles * ((N + 7) / 8) >= 2 * 148 ? 8 : 4;
      int64_t chunk = sweep::chunk_len(N, m_tiles, 148 * 6 * C::OCC, C::KT);
      chunk = chunk < least ? least : chunk;
      const int64_t tiles = m_tiles * ((N + chunk - 1) / chunk);
      if (tiles > 0x7fffffffLL) {
        set_error("chol_quad_form: problem too large (%lld tiles)", (long long)tiles);
        return (int)LAKDE_EUNSUPPORTED;
      }
      kern<<<(unsigned)tiles, sweep::THREADS, C::smem, as_stream(stream)>>>(
          static_cast<const T *>(W_triu), ws[0], ws[1], ws[2], static_cast<const T *>(Xn), xns[0], xns[1],
          static_cast<const T *>(Xm), xms[0], xms[1], static_cast<T *>(out), os[0], os[1], N, M, (int)D, chunk,
          m_tiles);
      return check_launch("chol_quad_form");
    });
  });
}

static int scatter_cov_launch(const char *what, int dtype, const void *rowptr, int rowptr_dtype, const void *col,
                              int col_dtype, const void *value, const void *Xn, const void *Xm, void *out, int64_t N,
                              int64_t M, int64_t D, void *nu_out, double nu0, void *stream) {
  clear_error();
  if (N < 0 || M < 0 || D < 1) {
    set_error("%s: invalid sizes (N=%lld, M=%lld, D=%lld)", what, (long long)N, (long long)M, (long long)D);
    return LAKDE_EINVAL;
  }
  if (N == 0) return LAKDE_OK;
  if (N > 0x7fffffffLL) {
    set_error("%s: N=%lld exceeds the grid limit", what, (long long)N);
    return LAKDE_EUNSUPPORTED;
  }
  if (!rowptr || !out || !Xn || (M > 0 && !Xm)) {
    set_error("%s: null pointer", what);
    return LAKDE_EINVAL;
  }
  if (int st = bind_device(what, {out, rowptr, col, value, Xn, Xm, nu_out})) return st;
  return dispatch_float(dtype, [&](auto t0) {
    using T = decltype(t0);
    return dispatch_index(rowptr_dtype, [&](auto r0) {
      using RP = decltype(r0);
      return dispatch_index(col_dtype, [&](auto c0) {
        using CI = decltype(c0);
        return dispatch_dp(D, [&](auto dp) {
          constexpr int DP = decltype(dp)::value;
          auto rp = static_cast<const RP *>(rowptr);
          auto cp = static_cast<const CI *>(col);
          auto vp = static_cast<const T *>(value);
          auto xn = static_cast<const T *>(Xn);
          auto xm = static_cast<const T *>(Xm);
          auto op = static_cast<T *>(out);
          if constexpr (DP <= 16) {
            const int64_t blocks = (N + 7) / 8;
            scatter_cov_warp<T, RP, CI, DP><<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(
                rp, cp, vp, xn, xm, op, N, M, (int)D, static_cast<T *>(nu_out), (T)nu0);
          } else if constexpr (sizeof(T) == 8) {
            scatter_cov_mma<RP, CI, DP><<<(unsigned)N, 32, 0, as_stream(stream)>>>(rp, cp, vp, xn, xm, op, M, (int)D,
                                                                                   static_cast<T *>(nu_out), (T)nu0);
          } else {
            using C = CtaScatterCfg<T, DP>;
            auto kern = scatter_cov_cta<T, RP, CI, DP>;
            int st = set_smem(kern, C::smem);
            if (st) return st;
            kern<<<(unsigned)N, C::THREADS, C::smem, as_stream(stream)>>>(rp, cp, vp, xn, xm, op, N, M, (int)D,
                                                                          static_cast<T *>(nu_out), (T)nu0);
          }
          return check_launch(what);
        });
      });
    });
  });
}

extern "C" int lakde_W_inv(int dtype, const void *rowptr, int rowptr_dtype, const void *col, int col_dtype,
                           const void *value, const void *Xn, const void *Xm, void *out, int64_t N, int64_t M,
                           int64_t D, void *stream) {
  return scatter_cov_launch("W_inv", dtype, rowptr, rowptr_dtype, col, col_dtype, value, Xn, Xm, out, N, M, D,
                            nullptr, 0.0, stream);
}

extern "C" int lakde_mstep(int dtype, int64_t N, int64_t D, int64_t npts, const void *rowptr, int rowptr_dtype,
                           const void *col, int col_dtype, const void *r, const void *X, int64_t kernel_offset,
                           double nu_0, void *S, void *nu, void *stream) {
  if (kernel_offset < 0 || kernel_offset + N > npts) {
    clear_error();
    set_error("mstep: kernel rows [%lld, %lld) outside the %lld points", (long long)kernel_offset,
              (long long)(kernel_offset + N), (long long)npts);
    return LAKDE_EINVAL;
  }
  const size_t es = dtype == LAKDE_F64 ? 8 : 4;
  const void *Xn = X ? static_cast<const char *>(X) + (size_t)kernel_offset * (size_t)D * es : nullptr;
  return scatter_cov_launch("mstep", dtype, rowptr, rowptr_dtype, col, col_dtype, r, Xn, X, S, N, npts, D, nu, nu_0,
                            stream);
}
