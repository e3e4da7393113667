// Column-statistics kernels shared by the centring paths (generic dense O and the RBM
// Obar writer). Each translation unit that includes this header gets its own copy.
#pragma once

#include "qgx_common.cuh"

namespace qgx {
namespace {

// Sums over chunks of partial sums laid out [chunk][column], by CTAs of 32 columns x 8 groups of chunks:
// the compensated FP64 additions (about seven instructions of 64 clocks of a sub-core each) bound
// them, and one thread per column in CTAs of 256 left most SMs idle (33 chunks of 1056 columns: 39 us
// for two sums; 6 now for the one that unweighted samples need).
constexpr int kRedCols = 32, kRedGroups = 8, kRedThreads = kRedCols * kRedGroups;
inline unsigned reduce_blocks(int64_t cols) { return (unsigned)((cols + kRedCols - 1) / kRedCols); }

// the sum of column col (this thread's: blockIdx.x 32 + lane), in the first warp of the CTA
__device__ inline double reduce_column(const double* __restrict__ part, int64_t nchunk, int64_t cols, int64_t col) {
  __shared__ double2 sh[kRedGroups][kRedCols];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  KahanD k;
  if (col < cols)
    for (int64_t c = g; c < nchunk; c += kRedGroups) k.add(part[c * cols + col]);
  __syncthreads();
  sh[g][lane] = make_double2(k.s, k.c);
  __syncthreads();
  KahanD sum;
  if (g == 0) {
#pragma unroll
    for (int q = 0; q < kRedGroups; ++q) {
      sum.add(sh[q][lane].x);
      sum.c += sh[q][lane].y;
    }
  }
  return sum.value();
}

// mean_u[col] = sum_k part_u[k, col] / ns, omean[col] = sum_k part_w[k, col] / ns (part_w NULL: no
// weights, the same as mean_u), mean_f = float copy of mean_u (each output may be NULL).
__global__ void __launch_bounds__(kRedThreads)
    col_reduce_kernel(const double* __restrict__ part_u, const double* __restrict__ part_w, int64_t nchunk, int64_t np,
                      int64_t ns, double* __restrict__ mean_u, double* __restrict__ omean, float* __restrict__ mean_f) {
  const int64_t col = blockIdx.x * (int64_t)kRedCols + (threadIdx.x & 31);
  const double su = reduce_column(part_u, nchunk, np, col);
  const double sw = part_w ? reduce_column(part_w, nchunk, np, col) : su;
  if (threadIdx.x >= 32 || col >= np) return;
  const double mu = su / (double)ns;
  if (mean_u) mean_u[col] = mu;
  if (mean_f) mean_f[col] = (float)mu;
  if (omean) omean[col] = part_w ? sw / (double)ns : mu;
}

// x[col] = sum_k part[k, col]
__global__ void __launch_bounds__(kRedThreads)
    sum_partials_kernel(const double* __restrict__ part, int64_t nchunk, int64_t cols, double* __restrict__ x) {
  const int64_t col = blockIdx.x * (int64_t)kRedCols + (threadIdx.x & 31);
  const double s = reduce_column(part, nchunk, cols, col);
  if (threadIdx.x < 32 && col < cols) x[col] = s;
}

}  // namespace
}  // namespace qgx
