// Gram matrices of the SR / MinSR solve (quantax/optimizer/solver.py:139 T = A A^T and
// :157 S = A^T A), FP32 operands, written as FP64 for the solver.
//
// This file holds the SIMT paths: QGX_GRAM_FP32 (FP32 accumulation) and QGX_GRAM_FP64, the
// Gram of the FP32 matrix to about 48 bits: every product is formed exactly as a float pair
// (TwoProd by FMA) and summed into a float-pair accumulator (TwoSum). FP64 arithmetic runs at
// a small fraction of the FP32 rate on this GPU, and this keeps the work on the FP32 pipe.
// Output tiles of register micro-tiles, K staged through shared memory in chunks of 16 with a
// register prefetch of the next chunk. Only tiles on or below the diagonal are computed; each
// element below it is written twice (itself and its mirror). The tensor-core paths (TF32 / BF16 /
// split TF32) live in gram_tc.cu.
#include <algorithm>

#include "qgx_common.cuh"

namespace qgx {

int gram_tc(const float* A, int64_t rows, int64_t k, int64_t lda, double* T, int64_t ldt, int mode, cudaStream_t st);

namespace {

constexpr int BK = 16;
constexpr int PAD = 4;

// Four consecutive elements for shared memory, zeros outside the matrix.
// TRANS = false: vectors are rows of A (T = A A^T, vector length klen, nvec of them): elements
// kk .. kk + 3 of vector v. TRANS = true: vectors are columns of A (S = A^T A): element kk of
// vectors v .. v + 3. One 16-byte load where vec (A and its rows start on 16 bytes) and all four exist.
template <bool TRANS>
__device__ inline float4 load_quad(const float* __restrict__ A, int64_t lda, int64_t v, int64_t kk, int64_t nvec,
                                   int64_t klen, bool vec) {
  float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (v >= nvec || kk >= klen) return q;
  const float* p = A + (TRANS ? kk * lda + v : v * lda + kk);
  const int64_t left = TRANS ? nvec - v : klen - kk;
  if (vec && left >= 4) return __ldg(reinterpret_cast<const float4*>(p));
  q.x = __ldg(p);
  if (left > 1) q.y = __ldg(p + 1);
  if (left > 2) q.z = __ldg(p + 2);
  if (left > 3) q.w = __ldg(p + 3);
  return q;
}

// (c.x, c.y) += (a b.x, a b.y) in one instruction, each rounded as fmaf
__device__ inline void fma_pair(float2& c, float a, float2 b) {
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %2};\n\tmov.b64 b, {%3, %4};\n\tmov.b64 c, {%0, %1};\n\t"
      "fma.rn.f32x2 c, a, b, c;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "+f"(c.x), "+f"(c.y)
      : "f"(a), "f"(b.x), "f"(b.y));
}

// (h, l) += a * b exactly rounded to a float pair; the _rn intrinsics are never contracted
__device__ inline void ds_fma(float a, float b, float& h, float& l) {
  const float p = __fmul_rn(a, b);
  const float e = fmaf(a, b, -p);
  const float t = __fadd_rn(h, p);
  const float z = __fsub_rn(t, h);
  l = __fadd_rn(l, __fadd_rn(__fadd_rn(__fsub_rn(h, __fsub_rn(t, z)), __fsub_rn(p, z)), e));
  h = t;
}

// TB x TB output tiles, TM x TM outputs per thread. Every output is one chain of operations over k
// in order whatever the tile, so the tile never changes a result. FP32 sums run as packed pairs of
// columns (fma.rn.f32x2: the same two roundings in half the issue slots).
// FP32, bound by the multiply-adds and, with 4 x 4, as much by the shared-memory reads:
// - 128 x 128, 8 x 8 per thread: 10.95 ms for 8192 x 8192 (13.99 with scalar multiply-adds).
// - 32 x 32, 4 x 4, 64 threads, for sizes whose 128 x 128 tiles do not fill the SMs: 144 us for S of
//   4099 x 1056 (45 tiles of 128 x 128: 394; 450 with scalar multiply-adds).
// FP64 sums (float pairs, ten dependent operations per product, bound by issue and latency): 64 x 64,
// 4 x 4, 256 threads: 11.3 ms for 4096 x 4096, 1.54 ms for 1056 x 4099. 128 x 128 with 8 x 8 per thread,
// 255 registers and one CTA per SM: 32.8 and 8.26 ms.
template <bool TRANS, bool DS, int TB, int TM>
__global__ void __launch_bounds__((TB / TM) * (TB / TM), 1)
    gram_simt_kernel(const float* __restrict__ A, int64_t nvec, int64_t klen, int64_t lda, double* __restrict__ T,
                     int64_t ldt, bool vec) {
  constexpr int NT = (TB / TM) * (TB / TM);
  constexpr int Q = TB * BK / 4 / NT;  // quads of an operand per thread and chunk
  static_assert((TM == 4 || TM == 8) && TB * BK / 4 % NT == 0, "whole quads");
  __shared__ __align__(16) float As[2][BK][TB + PAD];
  __shared__ __align__(16) float Bs[2][BK][TB + PAD];

  // lower-triangular tile index -> (bi, bj), bi >= bj
  const int64_t tile = blockIdx.x;
  int64_t bi = (int64_t)((sqrtf(8.0f * (float)tile + 1.0f) - 1.0f) * 0.5f);
  while ((bi + 1) * (bi + 2) / 2 <= tile) ++bi;
  while (bi * (bi + 1) / 2 > tile) --bi;
  const int64_t bj = tile - bi * (bi + 1) / 2;
  const int64_t row0 = bi * TB, col0 = bj * TB;

  const int tid = threadIdx.x;
  const int tx = tid % (TB / TM), ty = tid / (TB / TM);

  float4 ra[Q], rb[Q];
  // quad e of an operand chunk: along the vectors (TRANS) or along k
  auto vec_of = [](int e) { return TRANS ? 4 * (e % (TB / 4)) : e / (BK / 4); };
  auto k_of = [](int e) { return TRANS ? e / (TB / 4) : 4 * (e % (BK / 4)); };
  auto gload = [&](int64_t k0) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int e = tid + q * NT;
      ra[q] = load_quad<TRANS>(A, lda, row0 + vec_of(e), k0 + k_of(e), nvec, klen, vec);
      rb[q] = load_quad<TRANS>(A, lda, col0 + vec_of(e), k0 + k_of(e), nvec, klen, vec);
    }
  };
  auto put = [](float (&s)[BK][TB + PAD], int v, int kk, const float4& x) {
    if (TRANS) {
      *reinterpret_cast<float4*>(&s[kk][v]) = x;
    } else {
      s[kk][v] = x.x;
      s[kk + 1][v] = x.y;
      s[kk + 2][v] = x.z;
      s[kk + 3][v] = x.w;
    }
  };
  auto sstore = [&](int buf) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int e = tid + q * NT;
      put(As[buf], vec_of(e), k_of(e), ra[q]);
      put(Bs[buf], vec_of(e), k_of(e), rb[q]);
    }
  };

  float2 acc[TM][TM / 2], accl[DS ? TM : 1][DS ? TM / 2 : 1];  // columns (2 h, 2 h + 1)
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int h = 0; h < TM / 2; ++h) acc[i][h] = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < (DS ? TM : 1); ++i)
#pragma unroll
    for (int h = 0; h < (DS ? TM / 2 : 1); ++h) accl[i][h] = make_float2(0.0f, 0.0f);

  const int64_t nk = (klen + BK - 1) / BK;
  gload(0);
  sstore(0);
  __syncthreads();
  for (int64_t kc = 0; kc < nk; ++kc) {
    const int buf = (int)(kc & 1);
    if (kc + 1 < nk) gload((kc + 1) * BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM];
      float2 b[TM / 2];
#pragma unroll
      for (int u = 0; u < TM / 4; ++u) {
        const float4 x = *reinterpret_cast<const float4*>(&As[buf][kk][u * (TB * 4 / TM) + ty * 4]);
        const float4 y = *reinterpret_cast<const float4*>(&Bs[buf][kk][u * (TB * 4 / TM) + tx * 4]);
        a[4 * u] = x.x;
        a[4 * u + 1] = x.y;
        a[4 * u + 2] = x.z;
        a[4 * u + 3] = x.w;
        b[2 * u] = make_float2(y.x, y.y);
        b[2 * u + 1] = make_float2(y.z, y.w);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int h = 0; h < TM / 2; ++h) {
          if constexpr (DS) {
            ds_fma(a[i], b[h].x, acc[i][h].x, accl[i][h].x);
            ds_fma(a[i], b[h].y, acc[i][h].y, accl[i][h].y);
          } else {
            fma_pair(acc[i][h], a[i], b[h]);
          }
        }
    }
    if constexpr (DS) {
      // renormalise each pair (FastTwoSum, |h| >= |l|) once per chunk: the low word stays
      // below half an ulp of the high word, which keeps its own rounding negligible (about
      // 1e-13 relative at K = 8192, against 3e-12 without)
      auto renorm = [](float& h, float& l) {
        const float t = __fadd_rn(h, l);
        l = __fsub_rn(l, __fsub_rn(t, h));
        h = t;
      };
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int h = 0; h < TM / 2; ++h) {
          renorm(acc[i][h].x, accl[i][h].x);
          renorm(acc[i][h].y, accl[i][h].y);
        }
    }
    if (kc + 1 < nk) sstore(buf ^ 1);
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int64_t r = row0 + (i / 4) * (TB * 4 / TM) + ty * 4 + i % 4;
#pragma unroll
    for (int j = 0; j < TM; ++j) {
      const int64_t c = col0 + (j / 4) * (TB * 4 / TM) + tx * 4 + j % 4;
      if (r < nvec && c <= r) {
        double v = (double)(j & 1 ? acc[i][j / 2].y : acc[i][j / 2].x);
        if constexpr (DS) v += (double)(j & 1 ? accl[i][j / 2].y : accl[i][j / 2].x);
        T[r * ldt + c] = v;
        if (c < r) T[c * ldt + r] = v;
      }
    }
  }
}

template <bool TRANS, bool DS, int TB, int TM>
int launch_tile(const float* A, int64_t nvec, int64_t klen, int64_t lda, double* T, int64_t ldt, cudaStream_t st) {
  const int64_t nb = (nvec + TB - 1) / TB;
  const int64_t tiles = nb * (nb + 1) / 2;
  if (tiles > 0x7fffffff) return QGX_ERR_UNSUPPORTED;
  const bool vec = lda % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
  gram_simt_kernel<TRANS, DS, TB, TM>
      <<<(unsigned)tiles, (TB / TM) * (TB / TM), 0, st>>>(A, nvec, klen, lda, T, ldt, vec);
  return launch_status();
}

template <bool TRANS, bool DS = false>
int launch_gram_simt(const float* A, int64_t nvec, int64_t klen, int64_t lda, double* T, int64_t ldt, cudaStream_t st) {
  if constexpr (DS) {
    return launch_tile<TRANS, DS, 64, 4>(A, nvec, klen, lda, T, ldt, st);
  } else {
    // the tile with the shorter fullest SM; per output 32 x 32 tiles take 1.4 (S = A^T A) to 1.66
    // (T = A A^T) times as long as 128 x 128 ones where both fill the SMs (4096: 1.87 against 1.53 ms
    // and 2.31 against 1.61 ms)
    const int64_t sms = device_sm_count();
    auto fullest = [&](int64_t b) {
      const int64_t nb = (nvec + b - 1) / b;
      return (nb * (nb + 1) / 2 + sms - 1) / sms * b * b;
    };
    return 3 * fullest(32) < 2 * fullest(128) ? launch_tile<TRANS, DS, 32, 4>(A, nvec, klen, lda, T, ldt, st)
                                              : launch_tile<TRANS, DS, 128, 8>(A, nvec, klen, lda, T, ldt, st);
  }
}

}  // namespace
}  // namespace qgx

using namespace qgx;

extern "C" {

int qgx_gram(const float* A, int64_t rows, int64_t k, int64_t lda, double* T, int64_t ldt, int32_t mode,
             qgx_stream_t stream) {
  QGX_CHECK_ARG(rows >= 0 && k >= 0 && lda >= k && ldt >= rows);
  if (rows == 0) return QGX_OK;
  QGX_CHECK_ARG(A && T);
  if (mode == QGX_GRAM_FP32) return launch_gram_simt<false>(A, rows, k, lda, T, ldt, as_cuda(stream));
  if (mode == QGX_GRAM_FP64) return launch_gram_simt<false, true>(A, rows, k, lda, T, ldt, as_cuda(stream));
  if (mode == QGX_GRAM_TF32 || mode == QGX_GRAM_BF16 || mode == QGX_GRAM_3XTF32)
    return gram_tc(A, rows, k, lda, T, ldt, mode, as_cuda(stream));
  return QGX_ERR_ARG;
}

int qgx_gram_t(const float* A, int64_t rows, int64_t k, int64_t lda, double* S, int64_t lds, qgx_stream_t stream) {
  QGX_CHECK_ARG(rows >= 0 && k >= 0 && lda >= k && lds >= k);
  if (k == 0) return QGX_OK;
  QGX_CHECK_ARG(A && S);
  return launch_gram_simt<true>(A, k, rows, lda, S, lds, as_cuda(stream));
}

}  // extern "C"
