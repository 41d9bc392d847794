// Predictive log density of the Student-t mixture (lakde/local_adaptive_kde.py:200-223):
// a dense kernels x queries sweep (sweep.cuh) fused with the Student-t transform
// and an online logsumexp.  The kernel axis is split into chunks so the grid
// fills the 148 SMs; each (query tile, chunk) CTA leaves a (max, sum) pair per
// query in a caller-provided workspace and a second pass folds the chunks.
#include <mutex>

#include "common.cuh"
#include "sweep.cuh"

namespace lakde {

// Kernels per CTA: as many chunks as make up to four full waves of the
// resident CTAs with the query tiles (a fifth, partial wave would cost up to a
// fifth of the time); every chunk costs two values per query of workspace.
template <typename T, int DP>
static int64_t pred_chunk_t(int64_t N, int64_t Nq) {
  using C = sweep::Cfg<T, DP>;
  const int64_t tiles = (Nq + C::TILE - 1) / C::TILE;
  int64_t nchunks = (int64_t)148 * 4 * C::OCC / tiles;
  if (nchunks < 1) nchunks = 1;
  const int64_t chunk = (N + nchunks - 1) / nchunks;
  return chunk < 8 ? 8 : chunk;
}

static int64_t pred_chunk(int dtype, int64_t D, int64_t N, int64_t Nq) {
  int64_t chunk = 1;
  dispatch_float(dtype, [&](auto t0) {
    using T = decltype(t0);
    return dispatch_dp(D, [&](auto dp) {
      chunk = pred_chunk_t<T, decltype(dp)::value>(N, Nq);
      return 0;
    });
  });
  return chunk;
}

// The per-(query, kernel) transcendentals of the predictive density: the
// hardware approximations for float32 (absolute error of log(1 + q) below
// 4e-7, relative error of exp a few ulp near 0; a few 1e-5 nats at most on
// the density after the (nu + 1) / 2 factor), the accurate functions for
// float64.
__device__ __forceinline__ float pred_log1p(float q) { return __logf(1.f + q); }
__device__ __forceinline__ double pred_log1p(double q) { return log1p(q); }
__device__ __forceinline__ float pred_exp(float x) { return __expf(x); }
__device__ __forceinline__ double pred_exp(double x) { return exp(x); }

// The kernels x points sweep of sweep.cuh with the Student-t transform and a
// running log-sum-exp per query in registers (one exponential per pair: the
// smaller of the running maximum and the new term moves to the larger).
// float32, 100,000 kernels x 20,000 queries at d = 8: 10.7 -> 5.3 ms (issue
// slots and FMA pipe both 70 % busy); 20,000 x 4,096 at d = 21: 3.06 -> 1.35 ms;
// 10,000 x 2,000 at d = 63: 6.4 -> 1.95 ms.
template <typename T, int DP>
__global__ void __launch_bounds__(sweep::THREADS, sweep::Cfg<T, DP>::OCC) pred_partial_kernel(
    const T *__restrict__ X, const T *__restrict__ W, const T *__restrict__ nu, const T *__restrict__ lcoef,
    const T *__restrict__ Y, T *__restrict__ ws_m, T *__restrict__ ws_s, int64_t N, int64_t Nq, int D, int64_t chunk,
    int64_t q_tiles) {
  using C = sweep::Cfg<T, DP>;
  constexpr int P = C::P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *st = reinterpret_cast<T *>(smem_raw);
  const int tid = threadIdx.x;
  const int64_t q0 = (blockIdx.x % q_tiles) * C::TILE;
  const int64_t ch = blockIdx.x / q_tiles;
  const int64_t n_begin = ch * chunk;
  const int64_t n_end = (n_begin + chunk < N) ? n_begin + chunk : N;
  auto count = [&](int64_t n0) { return (int)((n_end - n0) < C::KT ? (n_end - n0) : C::KT); };
  auto stage = [&](int s, int64_t n0) {
    T *d = st + s * C::KT * C::KS;
    const int cnt = count(n0);
    sweep::stage_kernels<T, DP>(d, W, (int64_t)D * D, D, 1, X, D, 1, n0, cnt, D, tid);
    for (int k = tid; k < cnt; k += sweep::THREADS) {
      sweep::cp_async_elem(d + k * C::KS + C::S0, lcoef + n0 + k);
      sweep::cp_async_elem(d + k * C::KS + C::S0 + 1, nu + n0 + k);
    }
  };
  sweep::clear_stages<T, C>(st, n_end - n_begin, tid);
  __syncthreads();
  stage(0, n_begin);
  sweep::cp_async_commit();
  sweep::Points<T, DP> pts;
  pts.load(Y, D, 1, q0, Nq, D, st + 2 * C::KT * C::KS, tid);
  T m[P], s[P];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    m[p] = neg_inf<T>();
    s[p] = T(0);
  }
  int b = 0;
  for (int64_t n0 = n_begin; n0 < n_end; n0 += C::KT, b ^= 1) {
    if (n0 + C::KT < n_end) stage(b ^ 1, n0 + C::KT);
    sweep::cp_async_commit();
    sweep::cp_async_wait<1>();
    __syncthreads();
    const int cnt = count(n0);
    for (int k = 0; k < cnt; ++k) {
      const T *sk = st + (b * C::KT + k) * C::KS;
      T q[P];
      pts.quad(sk, D, q);
      const T lc = sk[C::S0], h = (sk[C::S0 + 1] + T(1)) / T(2);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        const T lp = lc - h * pred_log1p(q[p]);
        if (lp != neg_inf<T>()) {
          const bool up = lp > m[p];
          const T e = pred_exp(up ? m[p] - lp : lp - m[p]);
          s[p] = up ? s[p] * e + T(1) : s[p] + e;
          m[p] = up ? lp : m[p];
        }
      }
    }
    __syncthreads();  // the stage is refilled in the next iteration
  }
#pragma unroll
  for (int p = 0; p < P; ++p) {
    const int64_t q = q0 + tid + (int64_t)p * sweep::THREADS;
    if (q < Nq) {
      ws_m[ch * Nq + q] = m[p];
      ws_s[ch * Nq + q] = s[p];
    }
  }
}

template <typename T>
__global__ void pred_coeff_kernel(const T *__restrict__ nu, const T *__restrict__ logdet, T *__restrict__ out,
                                  int64_t N, int D) {
  const int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (n >= N) return;
  const T a1 = (nu[n] + T(1)) / T(2);
  const T a2 = (nu[n] + T(1) - T(D)) / T(2);
  const T g1 = (T)lgamma((double)a1);
  const T g2 = (T)lgamma((double)a2);
  const double v = (double)g1 - (double)g2 + 0.5 * (double)logdet[n] - 0.5 * D * 1.14472988584940017414;
  out[n] = (T)v;
}

}  // namespace lakde

using namespace lakde;

extern "C" int lakde_pred_coeff(int dtype, int64_t N, int64_t D, const void *nu, const void *logdet_W,
                                void *log_coeff, void *stream) {
  clear_error();
  if (N < 0 || D < 1) {
    set_error("pred_coeff: invalid sizes");
    return LAKDE_EINVAL;
  }
  if (N == 0) return LAKDE_OK;
  if (int st = bind_device("pred_coeff", {log_coeff, nu, logdet_W})) return st;
  return dispatch_float(dtype, [&](auto t0) {
    using T = decltype(t0);
    pred_coeff_kernel<T><<<(unsigned)((N + 255) / 256), 256, 0, as_stream(stream)>>>(
        static_cast<const T *>(nu), static_cast<const T *>(logdet_W), static_cast<T *>(log_coeff), N, (int)D);
    return check_launch("pred_coeff");
  });
}

extern "C" size_t lakde_log_pred_density_workspace(int dtype, int64_t N, int64_t Nq, int64_t D) {
  if (N <= 0 || Nq <= 0 || D < 1 || D > kMaxDim || (dtype != LAKDE_F32 && dtype != LAKDE_F64)) return 0;
  const int64_t chunk = pred_chunk(dtype, D, N, Nq);
  const int64_t nchunks = (N + chunk - 1) / chunk;
  const size_t es = dtype == LAKDE_F32 ? 4 : 8;
  return (size_t)(2 * nchunks * Nq) * es;
}

// The partial and fold launches of the predictive density over the (max, sum)
// scratch `ws` (lakde_log_pred_density_workspace bytes), shared by the
// workspace and the allocation-free entry points.
static int launch_pred(const char *what, int dtype, int64_t N, int64_t Nq, int64_t D, const void *X,
                       const void *W_triu, const void *nu, const void *log_coeff, const void *Y, void *out, void *ws,
                       void *stream) {
  return dispatch_float(dtype, [&](auto t0) {
    using T = decltype(t0);
    return dispatch_dp(D, [&](auto dp) {
      constexpr int DP = decltype(dp)::value;
      using C = sweep::Cfg<T, DP>;
      const int64_t chunk = pred_chunk_t<T, DP>(N, Nq);
      const int64_t nchunks = (N + chunk - 1) / chunk;
      const int64_t q_tiles = (Nq + C::TILE - 1) / C::TILE;
      if (q_tiles * nchunks > 0x7fffffffLL) {
        set_error("%s: grid too large", what);
        return (int)LAKDE_EUNSUPPORTED;
      }
      auto kern = pred_partial_kernel<T, DP>;
      if (C::smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::smem);
        if (e != cudaSuccess) {
          set_error("%s: %s", what, cudaGetErrorString(e));
          return (int)LAKDE_ECUDA;
        }
      }
      T *ws_m = static_cast<T *>(ws);
      T *ws_s = ws_m + nchunks * Nq;
      kern<<<(unsigned)(q_tiles * nchunks), sweep::THREADS, C::smem, as_stream(stream)>>>(
          static_cast<const T *>(X), static_cast<const T *>(W_triu), static_cast<const T *>(nu),
          static_cast<const T *>(log_coeff), static_cast<const T *>(Y), ws_m, ws_s, N, Nq, (int)D, chunk, q_tiles);
      if (int st = check_launch(what)) return st;
      sweep::fold_kernel<T><<<(unsigned)((Nq + 31) / 32), 256, 0, as_stream(stream)>>>(
          ws_m, ws_s, static_cast<T *>(out), Nq, nchunks, (T)log((double)N));
      return check_launch(what);
    });
  });
}

extern "C" int lakde_log_pred_density(int dtype, int64_t N, int64_t Nq, int64_t D, const void *X, const void *W_triu,
                                      const void *nu, const void *log_coeff, const void *Y, void *out,
                                      void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  if (N < 1 || Nq < 0 || D < 1) {
    set_error("log_pred_density: invalid sizes (N=%lld, Nq=%lld, D=%lld)", (long long)N, (long long)Nq,
              (long long)D);
    return LAKDE_EINVAL;
  }
  if (Nq == 0) return LAKDE_OK;
  const size_t need = lakde_log_pred_density_workspace(dtype, N, Nq, D);
  if (need == 0) {
    set_error("log_pred_density: unsupported dtype %d or D=%lld", dtype, (long long)D);
    return LAKDE_EUNSUPPORTED;
  }
  if (!workspace || workspace_bytes < need) {
    set_error("log_pred_density: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
    return LAKDE_EINVAL;
  }
  if (!X || !W_triu || !nu || !log_coeff || !Y || !out) {
    set_error("log_pred_density: null pointer");
    return LAKDE_EINVAL;
  }
  if (int st = bind_device("log_pred_density", {out, X, W_triu, nu, log_coeff, Y, workspace})) return st;
  return launch_pred("log_pred_density", dtype, N, Nq, D, X, W_triu, nu, log_coeff, Y, out, workspace, stream);
}

// ---------------------------------------------------------------------------
// Allocation-free variant.  Some callers cannot call cudaMalloc: hosts that own
// all device memory themselves (a framework's caching allocator, a plugin
// sandbox) or that forbid device allocation once they are running.  For them
// the (max, sum) partials live in this file-scope device array instead of a
// caller workspace.  It is 16 MiB; every GPU that loads the library holds it
// until the process exits.  All calls share it, and it keeps the contents of the
// last call: every slot a call reads is written earlier in that same call, so
// nothing needs clearing, but calls that overlap on the GPU (concurrent
// streams, or several host threads) race on it.
// ---------------------------------------------------------------------------
namespace lakde {

constexpr size_t kNoAllocScratchBytes = 16u << 20;
static __device__ __align__(256) unsigned char g_pred_scratch[kNoAllocScratchBytes];

// Device address of g_pred_scratch per device, resolved on the first call that
// runs on that device (with the device current) and kept for the life of the
// process.  A cudaDeviceReset destroys the array with the context, so the
// address is not valid across one (nor is any other device pointer).
constexpr int kMaxDevices = 128;
static void *g_pred_scratch_ptr[kMaxDevices];
static std::mutex g_pred_scratch_mu;

static int pred_scratch_address(void **out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    set_error("log_pred_density_noalloc: cudaGetDevice failed: %s", cudaGetErrorString(e));
    return LAKDE_ECUDA;
  }
  if (dev < 0 || dev >= kMaxDevices) {
    set_error("log_pred_density_noalloc: device index %d is beyond the %d devices this entry point serves", dev,
              kMaxDevices);
    return LAKDE_EUNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_pred_scratch_mu);
  if (!g_pred_scratch_ptr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_pred_scratch);
    if (e != cudaSuccess || !p) {
      set_error("log_pred_density_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return LAKDE_ECUDA;
    }
    g_pred_scratch_ptr[dev] = p;
  }
  *out = g_pred_scratch_ptr[dev];
  return LAKDE_OK;
}

}  // namespace lakde

extern "C" int lakde_log_pred_density_noalloc(int dtype, int64_t N, int64_t Nq, int64_t D, const void *X,
                                              const void *W_triu, const void *nu, const void *log_coeff,
                                              const void *Y, void *out, void *stream) {
  clear_error();
  if (N < 1 || Nq < 0 || D < 1) {
    set_error("log_pred_density_noalloc: invalid sizes (N=%lld, Nq=%lld, D=%lld)", (long long)N, (long long)Nq,
              (long long)D);
    return LAKDE_EINVAL;
  }
  if (Nq == 0) return LAKDE_OK;
  const size_t need = lakde_log_pred_density_workspace(dtype, N, Nq, D);
  if (need == 0) {
    set_error("log_pred_density_noalloc: unsupported dtype %d or D=%lld", dtype, (long long)D);
    return LAKDE_EUNSUPPORTED;
  }
  if (need > kNoAllocScratchBytes) {
    set_error("log_pred_density_noalloc: %lld queries x %lld kernels need %zu bytes of scratch, more than the "
              "built-in %zu bytes; split the queries into smaller batches",
              (long long)Nq, (long long)N, need, kNoAllocScratchBytes);
    return LAKDE_EINVAL;
  }
  if (!X || !W_triu || !nu || !log_coeff || !Y || !out) {
    set_error("log_pred_density_noalloc: null pointer");
    return LAKDE_EINVAL;
  }
  if (int st = bind_device("log_pred_density_noalloc", {out, X, W_triu, nu, log_coeff, Y})) return st;
  void *scratch = nullptr;
  if (int st = pred_scratch_address(&scratch)) return st;
  return launch_pred("log_pred_density_noalloc", dtype, N, Nq, D, X, W_triu, nu, log_coeff, Y, out, scratch, stream);
}
