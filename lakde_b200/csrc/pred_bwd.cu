// Backward of the predictive log density (lakde/local_adaptive_kde.py:200-223).
//
// With d = y - x_n, z = W_triu_n^T d = L_n^-1 d, Q = |z|^2, h_n = (nu_n + 1)/2,
// lp_ny = log_coeff_n - h_n log1p(Q), out_y = -log N + logsumexp_n lp_ny and
// the softmax weight w_ny = exp(lp_ny - out_y - log N), an upstream gradient
// g_y gives
//   d out / d y   = sum_n w_ny (-2 h_n / (1 + Q)) W_triu_n z          (score)
//   d out / d L_n = -(sum_y g_y w_ny) diag(1 / L_ii)
//                   + 2 h_n W_triu_n (sum_y c_ny z z^T),  c_ny = g_y w_ny / (1 + Q)
// (lower triangle).  The pair pass recomputes every quad form instead of
// storing the pair x D differences: it writes c_ny [N, Nq], the per-CTA row
// sums of g_y w_ny and the score partials; a dense scatter pass forms
// S_c[n] = sum_y c_ny d d^T, from which the host finishes d/dL_n with D x D
// products (sum_y c_ny z z^T = W_triu^T S_c W_triu).
#include "common.cuh"
#include "sweep.cuh"

namespace lakde {

// The staged factor in the unrolled layout at every DP (the pass needs all of
// z at once); two queries a thread up to 32 dimensions in float32 (z and the
// score take 2 DP registers a query), else one.  A query's coordinates are
// read once per kernel, from a shared-memory column of the thread.
template <typename T, int DP>
struct BwdCfg : sweep::Cfg<T, DP, false> {
  using L = sweep::Cfg<T, DP, false>;
  static constexpr int P = sizeof(T) == 4 && DP <= 32 ? 2 : 1;
  static constexpr int TILE = sweep::THREADS * P;
  static constexpr int KT = DP <= 8 ? 16 : DP <= 32 ? 8 : 2;
  // CTAs an SM is asked for (float64 at 64 dimensions: 135 KB leave one)
  static constexpr int OCC = DP <= 32 && sizeof(T) == 4 ? 3 : 2;
  // two stages, the queries, the warps' sums of g w
  static constexpr size_t smem =
      (2 * (size_t)KT * L::KS + (size_t)DP * TILE + (size_t)KT * (sweep::THREADS / 32)) * sizeof(T);
};

// Chunks of kernels: three waves of the resident CTAs with the query tiles.
template <typename T, int DP>
static int64_t bwd_chunk(int64_t N, int64_t Nq) {
  using C = BwdCfg<T, DP>;
  const int64_t tiles = (Nq + C::TILE - 1) / C::TILE;
  int64_t nchunks = (int64_t)148 * 3 * C::OCC / tiles;
  if (nchunks < 1) nchunks = 1;
  const int64_t chunk = (N + nchunks - 1) / nchunks;
  return chunk < 4 ? 4 : chunk;
}

// Bound by the FMA pipe and the broadcast reads of U (twice per kernel: z =
// U^T d, then U z), with the accurate log1p / exp and one division a pair.
// 20,000 kernels x 4,096 queries at d = 21, float32: 10.2 -> 2.7 ms against one
// query per thread with element-wise reads of U in the second product.
template <typename T, int DP>
__global__ void __launch_bounds__(sweep::THREADS, BwdCfg<T, DP>::OCC) pred_bwd_pairs_kernel(
    const T *__restrict__ X, const T *__restrict__ W, const T *__restrict__ nu, const T *__restrict__ lcoef,
    const T *__restrict__ Y, const T *__restrict__ outp, const T *__restrict__ gout, T *__restrict__ cw,
    T *__restrict__ sw_part, T *__restrict__ score_part, int64_t N, int64_t Nq, int D, int64_t chunk, int64_t q_tiles,
    T log_n) {
  using C = BwdCfg<T, DP>;
  using L = typename C::L;
  constexpr int P = C::P, V = L::V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *st = reinterpret_cast<T *>(smem_raw);
  T *ys = st + 2 * C::KT * L::KS;
  T *sred = ys + DP * C::TILE;  // [KT][4] warp sums of g w
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t qt = blockIdx.x % q_tiles;
  const int64_t ch = blockIdx.x / q_tiles;
  const int64_t n_begin = ch * chunk;
  const int64_t n_end = (n_begin + chunk < N) ? n_begin + chunk : N;
  auto count = [&](int64_t n0) { return (int)((n_end - n0) < C::KT ? (n_end - n0) : C::KT); };
  auto stage = [&](int s, int64_t n0) {
    T *d = st + s * C::KT * L::KS;
    const int cnt = count(n0);
    sweep::stage_kernels<T, DP, L>(d, W, (int64_t)D * D, D, 1, X, D, 1, n0, cnt, D, tid);
    for (int k = tid; k < cnt; k += sweep::THREADS) {
      sweep::cp_async_elem(d + k * L::KS + L::S0, lcoef + n0 + k);
      sweep::cp_async_elem(d + k * L::KS + L::S0 + 1, nu + n0 + k);
    }
  };
  sweep::clear_stages<T, L, C::KT>(st, n_end - n_begin, tid);
  __syncthreads();
  stage(0, n_begin);
  sweep::cp_async_commit();

  T ly[P], g[P], score[P][DP];
  T *col = ys + tid * P;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const int64_t q = qt * C::TILE + tid + (int64_t)p * sweep::THREADS;
    const bool qv = q < Nq;
    ly[p] = qv ? outp[q] + log_n : T(0);
    g[p] = qv ? gout[q] : T(0);
#pragma unroll
    for (int d = 0; d < DP; ++d) {
      col[d * C::TILE + p] = (qv && d < D) ? Y[q * D + d] : T(0);
      score[p][d] = T(0);
    }
  }

  int b = 0;
  for (int64_t n0 = n_begin; n0 < n_end; n0 += C::KT, b ^= 1) {
    if (n0 + C::KT < n_end) stage(b ^ 1, n0 + C::KT);
    sweep::cp_async_commit();
    sweep::cp_async_wait<1>();
    __syncthreads();
    const int cnt = count(n0);
    for (int k = 0; k < cnt; ++k) {
      const T *sk = st + (b * C::KT + k) * L::KS;
      sweep::Pair<T> acc[P][(DP + 1) / 2];
      sweep::products<L, T, DP, P>(sk, [&](int p, int j) { return col[j * C::TILE + p]; }, acc);
      T q[P], f[P];
      sweep::squares<T, DP, P>(acc, q);
      const T lc = sk[L::S0], h = (sk[L::S0 + 1] + T(1)) / T(2);
      T gw = T(0);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const int64_t m = qt * C::TILE + tid + (int64_t)p * sweep::THREADS;
        const T lp = lc - h * log1p(q[p]);
        const T w = m < Nq ? exp(lp - ly[p]) : T(0);
        const T c = g[p] * w / (T(1) + q[p]);
        if (m < Nq) cw[(n0 + k) * Nq + m] = c;
        f[p] = T(-2) * h * c;
        gw += g[p] * w;
      }
      // score: g w (-2 h / (1 + Q)) U z = -2 h c U z, row j of U against z
#pragma unroll
      for (int j = 0; j < DP; ++j) {
        // the loads of two rows at a time (hoisting more of them spills)
        if ((j & 1) == 0) asm volatile("" ::: "memory");
        T uz[P];
#pragma unroll
        for (int p = 0; p < P; ++p) uz[p] = T(0);
#pragma unroll
        for (int i0 = V * (j / V); i0 < L::DPV; i0 += V) {
          T u[V];
          sweep::load_vec<T>(sk + L::at(j, i0), u);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const int i = i0 + v;
            if (i < j || i >= DP) continue;
#pragma unroll
            for (int p = 0; p < P; ++p) uz[p] = fma(u[v], (i & 1) ? acc[p][i / 2].hi() : acc[p][i / 2].lo(), uz[p]);
          }
        }
#pragma unroll
        for (int p = 0; p < P; ++p) score[p][j] = fma(f[p], uz[p], score[p][j]);
      }
      // sum over this CTA's queries of g w for kernel n
      gw = warp_sum(gw);
      if (lane == 0) sred[k * 4 + warp] = gw;
    }
    __syncthreads();  // the sums are written, the stage is free to refill
    for (int k = tid; k < cnt; k += sweep::THREADS) {
      const T s = sred[k * 4 + 0] + sred[k * 4 + 1] + sred[k * 4 + 2] + sred[k * 4 + 3];
      sw_part[qt * N + n0 + k] = s;
    }
    // (the next group's sums are written after its own barrier above)
  }
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const int64_t q = qt * C::TILE + tid + (int64_t)p * sweep::THREADS;
    if (q < Nq) {
#pragma unroll
      for (int d = 0; d < DP; ++d)
        if (d < D) score_part[(ch * Nq + q) * D + d] = score[p][d];
    }
  }
}

// out[i] = sum of parts[0 .. nparts - 1][i]: 32 sums a block, eight threads
// dealing a sum's parts between them (one thread walking all of them waited on
// its own loads: 20,000 kernels x 64 queries at d = 16, 1,332 parts, 57 -> 17 us).
template <typename T>
__global__ void __launch_bounds__(256) sum_parts_kernel(const T *__restrict__ parts, T *__restrict__ out, int64_t n,
                                                        int64_t nparts) {
  constexpr int G = 8;
  __shared__ T ss[G][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int64_t i = blockIdx.x * (int64_t)32 + lane;
  T s = T(0);
  if (i < n) {
#pragma unroll 4
    for (int64_t p = g; p < nparts; p += G) s += parts[p * n + i];
  }
  ss[g][lane] = s;
  __syncthreads();
  if (g != 0 || i >= n) return;
#pragma unroll
  for (int k = 1; k < G; ++k) s += ss[k][lane];
  out[i] = s;
}

// S_c[n] = sum_y c[n, y] (y - x_n)(y - x_n)^T over all queries.  A thread owns
// a 4 x 4 block of one kernel's lower triangle; a CTA takes G kernels packed
// densely into its threads and stages the raw queries 64 at a time for all of
// them (centred in registers), so the staging and its barriers are paid once
// per G kernels and the lanes are full.  One kernel per CTA left 11 of 32 lanes
// idle at 24 dimensions and waited on its own staging: 7.7 ms for 20,000
// kernels x 4,096 queries at d = 21, now 2.6 ms (issue 70 %).
template <typename T, int DP>
struct DenseScatterCfg {
  static constexpr int NB = DP < 4 ? 1 : DP / 4;
  static constexpr int NBLK = NB * (NB + 1) / 2;
  static constexpr int GMAX = NBLK >= 128 ? 2 : 256 / NBLK > 32 ? 32 : 256 / NBLK;  // kernels per CTA
  static constexpr int CH = 64;
  static constexpr int LD = (DP < 4 ? 4 : DP) + 4;
};

template <typename T, int DP>
__global__ void __launch_bounds__(320) dense_scatter_kernel(const T *__restrict__ cw, const T *__restrict__ X,
                                                            const T *__restrict__ Y, T *__restrict__ S, int64_t N,
                                                            int64_t Nq, int D, int G) {
  using C = DenseScatterCfg<T, DP>;
  constexpr int V = 16 / (int)sizeof(T);
  __shared__ __align__(16) T sd[C::CH][C::LD];
  __shared__ T sv[C::GMAX][C::CH];
  const int tid = threadIdx.x;
  const int64_t n0 = (int64_t)blockIdx.x * G;
  const int g = tid / C::NBLK, e = tid % C::NBLK;
  const int64_t n = n0 + g;
  const bool own = g < G && n < N;
  int bi = 0;
  while ((bi + 1) * (bi + 2) / 2 <= e) ++bi;
  const int bj = e - bi * (bi + 1) / 2;
  T xa[4], xb[4], acc[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    xa[p] = (own && 4 * bi + p < D) ? X[n * D + 4 * bi + p] : T(0);
    xb[p] = (own && 4 * bj + p < D) ? X[n * D + 4 * bj + p] : T(0);
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q] = T(0);
  }
  for (int64_t base = 0; base < Nq; base += C::CH) {
    const int cnt = (int)((Nq - base) < C::CH ? (Nq - base) : C::CH);
    __syncthreads();
    for (int f = tid; f < cnt * C::LD; f += blockDim.x) {
      const int pp = f / C::LD, d = f % C::LD;
      sd[pp][d] = d < D ? Y[(base + pp) * D + d] : T(0);
    }
    for (int f = tid; f < G * C::CH; f += blockDim.x) {
      const int k = f / C::CH, pp = f % C::CH;
      sv[k][pp] = (n0 + k < N && pp < cnt) ? cw[(n0 + k) * Nq + base + pp] : T(0);
    }
    __syncthreads();
    if (own) {
#pragma unroll 2
      for (int pp = 0; pp < cnt; ++pp) {
        const T v = sv[g][pp];
        T a[4], b[4];
#pragma unroll
        for (int p = 0; p < 4; p += V) {
          T u[V], w[V];
          sweep::load_vec<T>(&sd[pp][4 * bi + p], u);
          sweep::load_vec<T>(&sd[pp][4 * bj + p], w);
#pragma unroll
          for (int k = 0; k < V; ++k) {
            a[p + k] = u[k] - xa[p + k];
            b[p + k] = v * (w[k] - xb[p + k]);
          }
        }
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[p][q] = fma(b[q], a[p], acc[p][q]);
      }
    }
  }
  if (!own) return;
  T *o = S + n * (int64_t)D * D;
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = 4 * bi + p, j = 4 * bj + q;
      if (i >= D || j > i) continue;
      o[i * D + j] = acc[p][q];
      o[j * D + i] = acc[p][q];
    }
}

}  // namespace lakde

using namespace lakde;

extern "C" size_t lakde_log_pred_density_bwd_workspace(int dtype, int64_t N, int64_t Nq, int64_t D) {
  if (N <= 0 || Nq <= 0 || D < 1 || D > kMaxDim || (dtype != LAKDE_F32 && dtype != LAKDE_F64)) return 0;
  size_t bytes = 0;
  dispatch_float(dtype, [&](auto t0) {
    using T = decltype(t0);
    return dispatch_dp(D, [&](auto dp) {
      using C = BwdCfg<T, decltype(dp)::value>;
      const int64_t chunk = bwd_chunk<T, decltype(dp)::value>(N, Nq);
      const int64_t nchunks = (N + chunk - 1) / chunk;
      const int64_t q_tiles = (Nq + C::TILE - 1) / C::TILE;
      bytes = (size_t)(q_tiles * N + nchunks * Nq * D) * sizeof(T);
      return 0;
    });
  });
  return bytes;
}

extern "C" int lakde_log_pred_density_bwd(int dtype, int64_t N, int64_t Nq, int64_t D, const void *X,
                                          const void *W_triu, const void *nu, const void *log_coeff, const void *Y,
                                          const void *out, const void *grad_out, void *grad_Y, void *cw, void *sw,
                                          void *S_c, void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  if (N < 1 || Nq < 1 || D < 1) {
    set_error("log_pred_density_bwd: invalid sizes");
    return LAKDE_EINVAL;
  }
  const size_t need = lakde_log_pred_density_bwd_workspace(dtype, N, Nq, D);
  if (need == 0) {
    set_error("log_pred_density_bwd: unsupported dtype %d or D=%lld", dtype, (long long)D);
    return LAKDE_EUNSUPPORTED;
  }
  if (!workspace || workspace_bytes < need) {
    set_error("log_pred_density_bwd: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
    return LAKDE_EINVAL;
  }
  if (!X || !W_triu || !nu || !log_coeff || !Y || !out || !grad_out || !grad_Y || !cw || !sw || !S_c) {
    set_error("log_pred_density_bwd: null pointer");
    return LAKDE_EINVAL;
  }
  if (int st = bind_device("log_pred_density_bwd",
                           {grad_Y, X, W_triu, nu, log_coeff, Y, out, grad_out, cw, sw, S_c, workspace}))
    return st;
  return dispatch_float(dtype, [&](auto t0) {
    using T = decltype(t0);
    return dispatch_dp(D, [&](auto dp) {
      constexpr int DP = decltype(dp)::value;
      using C = BwdCfg<T, DP>;
      const int64_t chunk = bwd_chunk<T, DP>(N, Nq);
      const int64_t nchunks = (N + chunk - 1) / chunk;
      const int64_t q_tiles = (Nq + C::TILE - 1) / C::TILE;
      T *sw_part = static_cast<T *>(workspace);
      T *score_part = sw_part + q_tiles * N;
      auto kern = pred_bwd_pairs_kernel<T, DP>;
      if (C::smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem);
        if (e != cudaSuccess) {
          set_error("log_pred_density_bwd: %s", cudaGetErrorString(e));
          return (int)LAKDE_ECUDA;
        }
      }
      kern<<<(unsigned)(q_tiles * nchunks), sweep::THREADS, C::smem, as_stream(stream)>>>(
          static_cast<const T *>(X), static_cast<const T *>(W_triu), static_cast<const T *>(nu),
          static_cast<const T *>(log_coeff), static_cast<const T *>(Y), static_cast<const T *>(out),
          static_cast<const T *>(grad_out), static_cast<T *>(cw), sw_part, score_part, N, Nq, (int)D, chunk, q_tiles,
          (T)log((double)N));
      if (int st = check_launch("log_pred_density_bwd")) return st;
      sum_parts_kernel<T><<<(unsigned)((N + 31) / 32), 256, 0, as_stream(stream)>>>(sw_part, static_cast<T *>(sw),
                                                                                       N, q_tiles);
      if (int st = check_launch("log_pred_density_bwd_sw")) return st;
      sum_parts_kernel<T><<<(unsigned)((Nq * D + 31) / 32), 256, 0, as_stream(stream)>>>(
          score_part, static_cast<T *>(grad_Y), Nq * D, nchunks);
      if (int st = check_launch("log_pred_density_bwd_score")) return st;
      using SC = DenseScatterCfg<T, DP>;
      // as many kernels per CTA as fit, but at least about four CTAs an SM
      int64_t G = N / (148 * 4);
      G = G < 1 ? 1 : G > SC::GMAX ? SC::GMAX : G;
      // at least four warps, which share the staging where few threads compute:
      // 500 kernels x 10,000 queries at d = 2 1,565 -> 444 us against the one warp
      // that its block of the lower triangle needs
      unsigned threads = (unsigned)((G * SC::NBLK + 31) / 32) * 32;
      threads = threads < 128 ? 128 : threads;
      dense_scatter_kernel<T, DP><<<(unsigned)((N + G - 1) / G), threads, 0, as_stream(stream)>>>(
          static_cast<const T *>(cw), static_cast<const T *>(X), static_cast<const T *>(Y), static_cast<T *>(S_c), N,
          Nq, (int)D, (int)G);
      return check_launch("log_pred_density_bwd_scatter");
    });
  });
}
