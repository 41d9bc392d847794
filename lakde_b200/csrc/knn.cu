// Selection half of the exact kNN graph (lakde/utils.py:77-116, which ranks
// torch.cdist distances with topk).  The caller computes a block of float64
// squared distances |a|^2 + |b|^2 - 2ab with one library GEMM; this kernel
// turns each row of the block into that point's k nearest neighbours, nearest
// first, equal distances ordered by index:
//
//   1. one CTA (small k and many rows: one warp) per row streams the row once,
//      keeping every value below a running threshold in a shared-memory buffer;
//      when the next chunk could overflow the buffer it is sorted (bitonic, by
//      value then index) and cut to its kc = k + 8 smallest, whose largest becomes
//      the threshold;
//   2. the kc candidates are re-ranked by exact float64 differences
//      sum_d (x_c - x_r)^2 (the GEMM form cancels for close points) and the
//      first k by (exact distance, index) are written.
//
// The point itself is excluded unless include_self (lakde/utils.py:104-105).
// Values that are not finite are no distances (a row of a point with an infinite
// coordinate holds -inf and +inf): such a row has neighbours -1.
#include "common.cuh"

namespace lakde {

// 256 threads per row, or 1,024 when the candidate buffer holds 4,096 or
// more entries (large k: the buffer's sorts dominate, so more threads share
// them; two such CTAs still fit an SM)
constexpr int kKnnThreads = 256, kKnnThreadsLarge = 1024;
constexpr int kKnnChunk = 1024;  // values a CTA scans between buffer checks

// Ascending bitonic sort of n (a power of two) (key, index) pairs in shared
// memory, ties by index; every thread of the CTA takes part.
__device__ __forceinline__ void bitonic_sort(double *key, int32_t *idx, int n) {
  for (int size = 2; size <= n; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      __syncthreads();
      for (int t = threadIdx.x; t < n / 2; t += blockDim.x) {
        const int lo = 2 * t - (t & (stride - 1));
        const int hi = lo + stride;
        const bool up = (lo & size) == 0;
        const double ka = key[lo], kb = key[hi];
        const int32_t ia = idx[lo], ib = idx[hi];
        const bool a_gt_b = ka > kb || (ka == kb && ia > ib);
        if (a_gt_b == up) {
          key[lo] = kb;
          key[hi] = ka;
          idx[lo] = ib;
          idx[hi] = ia;
        }
      }
    }
  }
  __syncthreads();
}

template <typename I, typename O>
__global__ void __launch_bounds__(kKnnThreadsLarge) knn_select_kernel(const double *__restrict__ dist, int64_t N,
                                                                 int64_t row0, const double *__restrict__ X, int D,
                                                                 int include_self, int k, int kc, int cap,
                                                                 I *__restrict__ out_idx, O *__restrict__ out_dist) {
  extern __shared__ double knn_smem[];
  double *key = knn_smem;
  int32_t *idx = reinterpret_cast<int32_t *>(knn_smem + cap);
  __shared__ int cnt;
  __shared__ double thr;
  const int64_t r = blockIdx.x;
  const int64_t self = row0 + r;
  const double *drow = dist + r * N;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  if (threadIdx.x == 0) {
    cnt = 0;
    thr = inf;
  }
  __syncthreads();

  // 1. threshold scan
  for (int64_t base = 0; base < N; base += kKnnChunk) {
    // every thread reads the count before any thread adds to it again
    const int c = cnt;
    __syncthreads();
    if (c + kKnnChunk > cap) {
      // pad, sort, keep the kc smallest
      for (int t = c + threadIdx.x; t < cap; t += blockDim.x) {
        key[t] = inf;
        idx[t] = 0x7fffffff;
      }
      bitonic_sort(key, idx, cap);
      if (threadIdx.x == 0) {
        cnt = c < kc ? c : kc;
        thr = c < kc ? inf : key[kc - 1];
      }
      __syncthreads();
    }
    const double t_now = thr;
    for (int u = threadIdx.x; u < kKnnChunk; u += blockDim.x) {
      const int64_t j = base + u;
      if (j < N) {
        double v = drow[j];
        if (v != v || (!include_self && j == self)) v = inf;
        if (v < t_now && v > -inf) {
          const int p = atomicAdd(&cnt, 1);
          key[p] = v;
          idx[p] = (int32_t)j;
        }
      }
    }
    __syncthreads();
  }
  {
    const int c = cnt;
    for (int t = c + threadIdx.x; t < cap; t += blockDim.x) {
      key[t] = inf;
      idx[t] = 0x7fffffff;
    }
    bitonic_sort(key, idx, cap);
  }

  // 2. exact re-ranking of the kc candidates (the rest padded as +inf)
  int n2 = 1;
  while (n2 < kc) n2 <<= 1;
  const double *xr = X + self * D;
  for (int t = threadIdx.x; t < n2; t += blockDim.x) {
    double e = inf;
    int32_t c = 0x7fffffff;
    if (t < kc) {
      c = idx[t];
      if (c >= 0 && c < N && (include_self || c != self)) {
        const double *xc = X + (int64_t)c * D;
        double s = 0.0;
        for (int d = 0; d < D; ++d) {
          const double df = xc[d] - xr[d];
          s = fma(df, df, s);
        }
        e = s;
      } else if (!(c >= 0 && c < N)) {
        c = 0x7fffffff;
      }
    }
    key[t] = e;
    idx[t] = c;
  }
  bitonic_sort(key, idx, n2);
  for (int t = threadIdx.x; t < k; t += blockDim.x) {
    const int32_t c = idx[t];
    out_idx[r * k + t] = (I)(c == 0x7fffffff ? -1 : c);
    if (out_dist) out_dist[r * k + t] = (O)sqrt(key[t]);
  }
}

// ------------------------------------------------- a warp per row (small k)
// The same selection with one warp per row and no block barrier: the warp
// streams 256 values at a time (four 16-byte loads per lane in flight) and
// appends those below its threshold by ballot.  When the next 256 could overflow
// its buffer it cuts it by bisection on the value to between kc and 3/2 kc
// entries (about ten counting passes over 512 entries, 1k instructions; a
// bitonic sort of them takes 7k, and four warps per row with a quarter each, so
// four times the sorts, were slower than one), and sorts only what is left at
// the end.  Whole graph of 50,000 points at d = 21, k = 64: selection 24.4 -> 5.0
// ms (one pass over the 20 GB of distances is 3.1), with the GEMM 49.0 -> 12.9;
// 100,003 points at d = 63, k = 100: 169 -> 65 ms.
constexpr int kWarpRows = 8;    // warps (rows) per block
constexpr int kWarpStep = 256;  // values a warp scans between buffer checks

__device__ __forceinline__ void warp_bitonic_sort(double *key, int32_t *idx, int n, int lane) {
  for (int size = 2; size <= n; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      __syncwarp();
      for (int t = lane; t < n / 2; t += 32) {
        const int lo = 2 * t - (t & (stride - 1));
        const int hi = lo + stride;
        const bool up = (lo & size) == 0;
        const double ka = key[lo], kb = key[hi];
        const int32_t ia = idx[lo], ib = idx[hi];
        const bool a_gt_b = ka > kb || (ka == kb && ia > ib);
        if (a_gt_b == up) {
          key[lo] = kb;
          key[hi] = ka;
          idx[lo] = ib;
          idx[hi] = ia;
        }
      }
    }
  }
  __syncwarp();
}

template <typename I, typename O, int CAP>
__global__ void __launch_bounds__(32 * kWarpRows) knn_select_warp_kernel(const double *__restrict__ dist, int64_t nb,
                                                                         int64_t N, int64_t row0,
                                                                         const double *__restrict__ X, int D,
                                                                         int include_self, int k, int kc,
                                                                         I *__restrict__ out_idx,
                                                                         O *__restrict__ out_dist) {
  extern __shared__ double knn_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  double *key = knn_smem + warp * CAP;
  int32_t *idx = reinterpret_cast<int32_t *>(knn_smem + kWarpRows * CAP) + warp * CAP;
  const int64_t r = (int64_t)blockIdx.x * kWarpRows + warp;
  if (r >= nb) return;
  const int64_t self = row0 + r;
  const double *drow = dist + r * N;
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  int cnt = 0;
  double thr = inf;  // later values at or above it are not among the kc smallest

  // sorts the cnt entries (padded with +inf) and keeps the kc smallest
  const auto sort_cut = [&]() {
    int n = 32;
    while (n < cnt) n <<= 1;
    for (int t = cnt + lane; t < n; t += 32) {
      key[t] = inf;
      idx[t] = 0x7fffffff;
    }
    warp_bitonic_sort(key, idx, n, lane);
    if (cnt >= kc) {
      cnt = kc;
      thr = key[kc - 1];
    }
  };
  // keeps the entries up to a pivot with kc to 3/2 kc of them: every later value
  // that is not below the pivot has kc predecessors.  Sorts when no such pivot is
  // found in 40 halvings (many equal values).
  const auto cut = [&]() {
    if (cnt < kc) return;
    __syncwarp();
    double lo = inf, hi = -inf;
    for (int t = lane; t < cnt; t += 32) {
      lo = fmin(lo, key[t]);
      hi = fmax(hi, key[t]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const int most = kc + kc / 2;
    int c = cnt;
    double pivot = hi;
    for (int it = 0; it < 40 && c > most; ++it) {
      const double mid = lo + 0.5 * (hi - lo);
      int m = 0;
      for (int t = lane; t < cnt; t += 32) m += key[t] <= mid;
      m = __reduce_add_sync(0xffffffffu, m);
      if (m < kc) {
        lo = mid;
      } else {
        hi = pivot = mid;
        c = m;
      }
    }
    if (c > most) {
      sort_cut();
      return;
    }
    // entries up to the pivot move forward, in order; a batch is read before
    // any of it is overwritten
    int kept = 0;
    for (int t0 = 0; t0 < cnt; t0 += 32) {
      const int t = t0 + lane;
      const double v = t < cnt ? key[t] : inf;
      const int32_t i = t < cnt ? idx[t] : 0;
      const bool keep = t < cnt && v <= pivot;
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const int p = kept + __popc(m & below);
        key[p] = v;
        idx[p] = i;
      }
      kept += __popc(m);
      __syncwarp();
    }
    cnt = kept;
    thr = pivot;
  };

  // 1. threshold scan
  const bool vec = (reinterpret_cast<uintptr_t>(drow) & 15u) == 0;
  for (int64_t base = 0; base < N; base += kWarpStep) {
    if (cnt + kWarpStep > CAP) cut();
    double v[kWarpStep / 32];
    // value e of this lane is column base + 64 (e / 2) + 2 lane + e % 2
    if (vec && base + kWarpStep <= N) {
#pragma unroll
      for (int e = 0; e < kWarpStep / 32; e += 2) {
        const double2 d2 = __ldcs(reinterpret_cast<const double2 *>(drow + base + 32 * e + 2 * lane));
        v[e] = d2.x;
        v[e + 1] = d2.y;
      }
    } else {
#pragma unroll
      for (int e = 0; e < kWarpStep / 32; ++e) {
        const int64_t j = base + 64 * (e / 2) + 2 * lane + (e & 1);
        v[e] = j < N ? drow[j] : inf;
      }
    }
#pragma unroll
    for (int e = 0; e < kWarpStep / 32; ++e) {
      const int64_t j = base + 64 * (e / 2) + 2 * lane + (e & 1);
      bool in = v[e] < thr && (include_self || j != self);  // false for NaN
      if (!__any_sync(0xffffffffu, in)) continue;
      in = in && v[e] > -inf;
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in) {
        const int p = cnt + __popc(m & below);
        key[p] = v[e];
        idx[p] = (int32_t)j;
      }
      cnt += __popc(m);
    }
  }
  cut();
  sort_cut();

  // 2. exact re-ranking of the kc candidates
  int n2 = 32;
  while (n2 < kc) n2 <<= 1;
  const double *xr = X + self * D;
  for (int t = lane; t < n2; t += 32) {
    double e = inf;
    int32_t c = 0x7fffffff;
    if (t < cnt) {
      c = idx[t];
      const double *xc = X + (int64_t)c * D;
      double s = 0.0;
#pragma unroll 4
      for (int d = 0; d < D; ++d) {
        const double df = xc[d] - xr[d];
        s = fma(df, df, s);
      }
      e = s;
    }
    key[t] = e;
    idx[t] = c;
  }
  warp_bitonic_sort(key, idx, n2, lane);
  for (int t = lane; t < k; t += 32) {
    const int32_t c = idx[t];
    out_idx[r * k + t] = (I)(c == 0x7fffffff ? -1 : c);
    if (out_dist) out_dist[r * k + t] = (O)sqrt(key[t]);
  }
}

}  // namespace lakde

using namespace lakde;

extern "C" int lakde_knn_select(const void *dist, int64_t nb, int64_t N, int64_t row0, const void *X, int64_t D,
                                int include_self, int64_t k, int idx_dtype, void *out_idx, int dist_dtype,
                                void *out_dist, void *stream) {
  clear_error();
  if (nb < 0 || N < 1 || D < 1 || row0 < 0 || row0 + nb > N || k < 1 || N > 0x7ffffffeLL) {
    set_error("knn_select: invalid sizes (nb=%lld, N=%lld, D=%lld, row0=%lld, k=%lld)", (long long)nb, (long long)N,
              (long long)D, (long long)row0, (long long)k);
    return LAKDE_EINVAL;
  }
  const int64_t avail = include_self ? N : N - 1;
  if (k > avail) {
    set_error("knn_select: k=%lld exceeds the %lld candidate points", (long long)k, (long long)avail);
    return LAKDE_EINVAL;
  }
  if (nb == 0) return LAKDE_OK;
  if (!dist || !X || !out_idx || (idx_dtype != LAKDE_I32 && idx_dtype != LAKDE_I64) ||
      (out_dist && dist_dtype != LAKDE_F32 && dist_dtype != LAKDE_F64)) {
    set_error("knn_select: null pointer or unsupported dtype");
    return LAKDE_EINVAL;
  }
  const int64_t kc = (k + 8 < avail) ? k + 8 : avail;
  int64_t cap = 2048;
  while (cap < kc + kKnnChunk) cap <<= 1;
  const size_t smem = (size_t)cap * (sizeof(double) + sizeof(int32_t));
  if (smem > 200 * 1024) {
    set_error("knn_select: k=%lld needs %zu bytes of shared memory for its candidates", (long long)k, smem);
    return LAKDE_EUNSUPPORTED;
  }
  if (int st = bind_device("knn_select", {dist, X, out_idx, out_dist})) return st;
  cudaStream_t s = as_stream(stream);
  auto launch_warps = [&](auto ti, auto to, auto tc) {
    using I = decltype(ti);
    using O = decltype(to);
    constexpr int CAP = decltype(tc)::value;
    auto kern = knn_select_warp_kernel<I, O, CAP>;
    constexpr size_t bytes = (size_t)kWarpRows * CAP * (sizeof(double) + sizeof(int32_t));
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) {
      set_error("knn_select: cannot reserve %zu bytes of shared memory", bytes);
      return (int)LAKDE_ECUDA;
    }
    kern<<<(unsigned)((nb + kWarpRows - 1) / kWarpRows), 32 * kWarpRows, bytes, s>>>(
        static_cast<const double *>(dist), nb, N, row0, static_cast<const double *>(X), (int)D, include_self, (int)k,
        (int)kc, static_cast<I *>(out_idx), static_cast<O *>(out_dist));
    return check_launch("knn_select");
  };
  auto launch = [&](auto ti, auto to) {
    using I = decltype(ti);
    using O = decltype(to);
    // a warp per row while 3/2 of its candidates and a step fit its buffer: 6 KB
    // up to 160 candidates (32 rows an SM in flight), 12 KB up to 500; beyond, a
    // block per row, whose barriers cost less than a lone warp's sorts.  And only
    // with rows enough: below 8 warps an SM (1,184 rows) a launch takes as long as
    // one warp over its row, 3.0 us per 1,000 values, while a block's threads share
    // theirs; but a block also sorts its whole buffer, which short rows do not
    // repay.  Block / warp, us, at 148, 592 and 1,024 rows: k = 5, 1,000,000 points
    // 2245 / 3040, 2397 / 3074, 2655 / 3142; 400,000 points 955 / 1234, 1085 / 1248,
    // 1240 / 1275; 100,000 points 305 / 327, 412 / 330, 505 / 336; 30,000 points 89 /
    // 91, 215 / 111, 315 / 113; k = 490, 3,000 points 68 / 141, 193 / 141, 326 / 141;
    // 400,000 points 1137 / 1441, 1490 / 1454, 2029 / 1480.
    const bool many = nb > 8 * 148;
    if (kc <= 160 && (many || N <= 32768 || (N <= 131072 && nb >= 256)))
      return launch_warps(ti, to, std::integral_constant<int, 512>{});
    if (kc > 160 && kc <= 500 && (many || (N <= 262144 && nb >= 600)))
      return launch_warps(ti, to, std::integral_constant<int, 1024>{});
    auto kern = knn_select_kernel<I, O>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      set_error("knn_select: cannot reserve %zu bytes of shared memory", smem);
      return (int)LAKDE_ECUDA;
    }
    const int threads = cap >= 4096 ? kKnnThreadsLarge : kKnnThreads;
    kern<<<(unsigned)nb, threads, smem, s>>>(static_cast<const double *>(dist), N, row0,
                                                 static_cast<const double *>(X), (int)D, include_self, (int)k,
                                                 (int)kc, (int)cap, static_cast<I *>(out_idx),
                                                 static_cast<O *>(out_dist));
    return check_launch("knn_select");
  };
  if (idx_dtype == LAKDE_I32) {
    if (out_dist && dist_dtype == LAKDE_F32) return launch(int32_t(0), float(0));
    return launch(int32_t(0), double(0));
  }
  if (out_dist && dist_dtype == LAKDE_F32) return launch(int64_t(0), float(0));
  return launch(int64_t(0), double(0));
}
