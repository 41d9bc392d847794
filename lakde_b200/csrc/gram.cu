// Weighted Gram sum of the hierarchical model's shared-precision update in
// FP64 (lakde/local_hierarchical_kde.py:293-297):
//   out = sum_n w_n W_triu_n W_triu_n^T        (D x D, symmetric)
// straight from the float32 (or float64) factors, without a float64 copy of
// all of them, on the FP64 tensor cores: each warp walks every (blocks x
// warps)-th kernel with the lower 8 x 8 tiles of the sum in registers.  A step
// takes four columns j of W_n: lane l holds W[8 I + l / 4][j + l % 4] of each row
// block I, which is the A fragment of rows I (scaled by w_n) and, the product
// being with W^T, the B fragment of columns I; the next eight columns' loads
// are in flight under a block's products.  Rows below the diagonal block are
// zero and not loaded.  The warps' sums are added in a fixed order, per block
// and then over the blocks, so the result does not depend on scheduling.
//
// Bound by the FP64 tensor pipe: NT (NT + 1) (NT + 2) / 3 MMAs of 16 cycles per
// kernel.  20,000 kernels at d = 43, both launches: 414 -> 72 us (scalar FMAs on 4 x 4
// register blocks staged through shared memory, and one thread walking all
// partials of an element, before).
#include "common.cuh"
#include "factor_dmma.cuh"

namespace lakde {

constexpr int kGramBlocks = 592;  // partials the workspace has room for
constexpr int kGramWarps = 4;

template <typename T, int NT>
__device__ __forceinline__ void gram_load(const T *__restrict__ Wn, int J, int D, int lane, T (&f)[NT][2]) {
  const int r = lane >> 2, c = 8 * J + (lane & 3);
#pragma unroll
  for (int I = 0; I < NT; ++I) {
    if (I > J) continue;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int i = 8 * I + r, j = c + 4 * s;
      f[I][s] = (i <= j && j < D) ? Wn[(int64_t)i * D + j] : T(0);
    }
  }
}

template <typename T, int NT>
__global__ void __launch_bounds__(32 * kGramWarps) gram_partial_kernel(const T *__restrict__ W, const T *__restrict__ w,
                                                                      int64_t N, int D,
                                                                      double *__restrict__ partials) {
  constexpr int NTILE = NT * (NT + 1) / 2;
  __shared__ double red[NTILE * 64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double acc[NTILE][2];
#pragma unroll
  for (int t = 0; t < NTILE; ++t) acc[t][0] = acc[t][1] = 0.0;
  const int64_t stride = (int64_t)gridDim.x * kGramWarps, DD = (int64_t)D * D;
  int64_t n = (int64_t)blockIdx.x * kGramWarps + warp;
  T f[2][NT][2];
  T wn = T(0);
  if (n < N) {
    gram_load<T, NT>(W + n * DD, 0, D, lane, f[0]);
    wn = w[n];
  }
  bool left = false;
  while (n < N) {
    const int64_t nn = n + stride;
    const double wd = (double)wn;
    // a kernel of infinite weight is left for the end: times the zeros of a
    // fragment its weight would make the whole sum NaN
    const bool take = !isinf(wd);
    left = left || !take;
#pragma unroll
    for (int J = 0; J < NT; ++J) {
      // block J is in f[J % 2] (NT even: the next kernel's block 0 in f[0])
      if (J + 1 < NT) {
        gram_load<T, NT>(W + n * DD, J + 1, D, lane, f[(J + 1) & 1]);
      } else if (NT % 2 == 0 && nn < N) {
        gram_load<T, NT>(W + nn * DD, 0, D, lane, f[0]);
        wn = w[nn];
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!take) break;
        double b[NT];
#pragma unroll
        for (int I = 0; I < NT; ++I)
          if (I <= J) b[I] = (double)f[J & 1][I][s];
#pragma unroll
        for (int I = 0; I < NT; ++I) {
          if (I > J) continue;
          const double a = wd * b[I];
#pragma unroll
          for (int k = 0; k <= I; ++k) dmma::mma(acc[I * (I + 1) / 2 + k][0], acc[I * (I + 1) / 2 + k][1], a, b[k]);
        }
      }
    }
    if (NT % 2 == 1 && nn < N) {
      gram_load<T, NT>(W + nn * DD, 0, D, lane, f[0]);
      wn = w[nn];
    }
    n = nn;
  }
  // the warps' sums in turn
  for (int v = 0; v < kGramWarps; ++v) {
    if (warp == v) {
#pragma unroll
      for (int t = 0; t < NTILE; ++t) {
        double *r = red + t * 64 + (lane >> 2) * 8 + 2 * (lane & 3);
        r[0] = (v ? r[0] : 0.0) + acc[t][0];
        r[1] = (v ? r[1] : 0.0) + acc[t][1];
      }
    }
    __syncthreads();
  }
  const int tri = D * (D + 1) / 2;
  const bool infinite = __syncthreads_or(left);
  for (int e = threadIdx.x; e < NTILE * 64; e += 32 * kGramWarps) {
    int I = 0;
    const int t = e >> 6;
    while ((I + 1) * (I + 2) / 2 <= t) ++I;
    const int i = 8 * I + ((e >> 3) & 7), k = 8 * (t - I * (I + 1) / 2) + (e & 7);
    if (i >= D || k > i) continue;
    double sum = red[e];
    if (infinite) {
      // w times the finished element of W W^T
#pragma unroll 1
      for (int64_t m0 = (int64_t)blockIdx.x * kGramWarps; m0 < N; m0 += stride)
#pragma unroll 1
        for (int64_t m = m0; m < m0 + kGramWarps && m < N; ++m) {
          if (!isinf((double)w[m])) continue;
          double el = 0.0;
#pragma unroll 1
          for (int j = i; j < D; ++j) el = fma((double)W[m * DD + i * D + j], (double)W[m * DD + k * D + j], el);
          sum = fma((double)w[m], el, sum);
        }
    }
    partials[(int64_t)blockIdx.x * tri + i * (i + 1) / 2 + k] = sum;
  }
}

// One warp per element, its lanes over the partials (fixed order).
__global__ void __launch_bounds__(256) gram_final_kernel(const double *__restrict__ partials, int nparts, int D,
                                                         double *__restrict__ out) {
  const int tri = D * (D + 1) / 2, lane = threadIdx.x & 31;
  const int e = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (e >= tri) return;
  double s = 0.0;
#pragma unroll 4
  for (int p = lane; p < nparts; p += 32) s += partials[(int64_t)p * tri + e];
  s = warp_sum(s);
  if (lane == 0) {
    int i = 0;
    while ((i + 1) * (i + 2) / 2 <= e) ++i;
    const int k = e - i * (i + 1) / 2;
    out[i * D + k] = s;
    out[k * D + i] = s;
  }
}

}  // namespace lakde

using namespace lakde;

extern "C" size_t lakde_weighted_gram_workspace(int64_t D) {
  if (D < 1 || D > kMaxDim) return 0;
  return (size_t)kGramBlocks * (size_t)(D * (D + 1) / 2) * sizeof(double);
}

extern "C" int lakde_weighted_gram(int dtype, int64_t N, int64_t D, const void *W_triu, const void *w, double *out,
                                   void *workspace, size_t workspace_bytes, void *stream) {
  clear_error();
  if (N < 0 || D < 1 || D > kMaxDim) {
    set_error("weighted_gram: invalid sizes (N=%lld, D=%lld)", (long long)N, (long long)D);
    return D > kMaxDim ? LAKDE_EUNSUPPORTED : LAKDE_EINVAL;
  }
  if (!out || !workspace || (N > 0 && (!W_triu || !w))) {
    set_error("weighted_gram: null pointer");
    return LAKDE_EINVAL;
  }
  if (workspace_bytes < lakde_weighted_gram_workspace(D)) {
    set_error("weighted_gram: workspace of %zu bytes needed, %zu given", lakde_weighted_gram_workspace(D),
              workspace_bytes);
    return LAKDE_EINVAL;
  }
  if (int st = bind_device("weighted_gram", {out, W_triu, w, workspace})) return st;
  return dispatch_float(dtype, [&](auto t0) {
    using T = decltype(t0);
    double *part = static_cast<double *>(workspace);
    return dispatch_dp(D, [&](auto dp) {
      constexpr int NT = (decltype(dp)::value + 7) / 8;
      // three blocks an SM (two at 64 dimensions: the sum's tiles in registers)
      int64_t blocks = (N + kGramWarps - 1) / kGramWarps;
      const int64_t most = 148 * (NT >= 8 ? 2 : 3);
      blocks = blocks < 1 ? 1 : blocks > most ? most : blocks;
      gram_partial_kernel<T, NT><<<(unsigned)blocks, 32 * kGramWarps, 0, as_stream(stream)>>>(
          static_cast<const T *>(W_triu), static_cast<const T *>(w), N, (int)D, part);
      if (int st = check_launch("weighted_gram")) return st;
      const int tri = (int)(D * (D + 1) / 2);
      gram_final_kernel<<<(unsigned)((tri + 7) / 8), 256, 0, as_stream(stream)>>>(part, (int)blocks, (int)D, out);
      return check_launch("weighted_gram_final");
    });
  });
}
