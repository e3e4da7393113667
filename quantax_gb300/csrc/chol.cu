// FP64 Cholesky factorisation A = L L^T for the diagonal-shifted MinSR / SR solves
// (quantax/optimizer/solver.py:50-62: jax.scipy.linalg.solve(T + shift, b, assume_a="pos")).
//
// A is n x n, symmetric, row-major with leading dimension lda. L overwrites the lower triangle
// (L[i][j] at A[i lda + j], i >= j); the strict upper triangle is not touched, so it still
// holds the matrix by symmetry. Read as column-major, the factor is the upper triangle
// U = L^T with A = U^T U.
//
// FP64 arithmetic runs at about two FMAs per clock per SM on GB300 and every FP64 instruction
// takes 64 clocks, so nothing here runs on the FP64 pipe but the last step of an update (and the panels
// of a matrix whose rows hardly interact, see weak_coupling_kernel): right-looking, 256-column panels, each factored as four 64-column blocks (potrf of the 64 x 64
// diagonal block and the 64-wide triangular solve of every row below it) in 60-bit fixed point
// on the integer pipe (qgx_fixed.cuh). Every update of the form C -= P P^T runs on the tensor cores
// as an exact integer product (the Ozaki scheme: Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix multiplication and
// its applications", Numer. Algorithms 59, 2012):
//   * each row r of the panel P (K <= 256 columns) is scaled by 2^-e_r, e_r the exponent with
//     max_k |P_rk| < 2^e_r, and rounded to the integer F = round(P 2^(56 - e_r)), |F| <= 2^56;
//   * F is written as 8 balanced base-128 digits S_0 .. S_7 (|S_0| <= 128, S_t in [-64, 64)
//     for t >= 1), each exact in BF16; P_rk = 2^e_r sum_t S_t[r][k] 2^(-7(t+1)) up to 2^(e_r-57);
//   * for each level l = t + u <= 7 the tensor core accumulates I_l = sum_(t+u=l) S_t S_u^T
//     over K in FP32: every product is an integer below 2^14 in magnitude and every partial
//     sum an integer below 2^24 (at most 8 pairs, K <= 256), so the FP32 accumulation is exact;
//   * the epilogue forms V = sum_l I_l 2^(38 - 7 l) exactly in int64 (levels 6 and 7 rounded
//     to 2^-38), converts once to FP64 and subtracts 2^(e_i + e_j - 52) V from C_ij.
// The products with t + u >= 8 are dropped: with the digits' own truncation the update's error
// is a few 2^-56 K 2^(e_i + e_j), below FP64's own rounding of a K-term dot product.
//
// The tensor-core kernel (ozaki_syrk_kernel) takes 128 x 64 tiles of C, one CTA per SM and a few
// tiles per CTA; the digits are stored as the shared-memory image of its operands.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "qgx_common.cuh"
#include "qgx_fixed.cuh"
#include "qgx_tc.cuh"

namespace qgx {
namespace {

constexpr int kPanel = 256;                     // columns of one tensor-core trailing update
constexpr int kBlk = 64;                        // columns of one diagonal block
constexpr int kSlices = 8;                      // BF16 digits per element
constexpr int kFixBits = 56;                    // kSlices * 7 fraction bits of the sliced rows
constexpr int kOzM = 128, kOzN = 64, kOzKB = 32;  // tile rows, tile columns, K per stage
constexpr int kOzStages = 2;
constexpr int kOzRowBytes = kOzKB * 2;                         // one operand row of a stage
constexpr int kOzABytes = kSlices * kOzM * kOzRowBytes;        // 64 KB
constexpr int kOzBBytes = kSlices * kOzN * kOzRowBytes;        // 32 KB
constexpr int kOzStageBytes = kOzABytes + kOzBBytes;
constexpr int kOzEpiWarps = 8;                                 // epilogue warps; then producer, MMA issuer
constexpr int kOzThreads = 32 * (kOzEpiWarps + 2);
constexpr int kOzTurn = 8, kOzTurnLd = kOzTurn + 1;            // columns per turn through the transpose buffers
constexpr int kOzTurnBytes = kOzEpiWarps * 32 * kOzTurnLd * 8;
constexpr size_t kOzSmem = 1024 + (size_t)kOzStages * kOzStageBytes + kOzTurnBytes + 256;
constexpr uint32_t kOzTmemCols = kSlices * kOzN;               // eight 64-column FP32 level accumulators
constexpr int kOzGroup = 8;                                    // row tiles per rasterisation group

// Digit slices are stored as the operand images of the update's stages: [128-row block][32-column
// block][slice][row][64 bytes], the 16-byte chunks of a row swizzled as the 64-byte swizzle of the
// MMA descriptors has them, so that a stage's A operand is one contiguous 64 KB copy and its B
// operand (a 64-row half) eight of 4 KB.
inline int64_t slice_rows(int64_t n) { return (n + kOzM - 1) / kOzM * kOzM; }

inline int64_t al256(int64_t b) { return (b + 255) / 256 * 256; }

// ---- fixed-point panel ----------------------------------------------------------------------
// Row r's scale comes from an upper bound on its diagonal entry at the start of the panel,
// a_rr <= f 2^E (f > 0): set from the matrix, then lowered by each panel's squares.
struct RowBound {
  float* f;
  int* E;
};

// smallest e with 2^(2e) >= 2 f 2^E: the row's entries of L are below 2^e sqrt(1/2)
__device__ inline int row_exponent(const RowBound& b, int64_t r) {
  const float f = fmaxf(b.f[r], 8.6736174e-19f);  // 2^-60: a bound that rounding took to zero
  const int E = ((__float_as_int(f) >> 23) & 255) - 126 + b.E[r];
  return (E + 2) >> 1;
}

// *info: the smallest order of a leading minor found not positive definite (0: none)
__device__ inline void record_info(int* info, int64_t order) {
  if (atomicCAS(info, 0, (int)order) != 0) atomicMin(info, (int)order);
}

__device__ inline double quiet_nan() { return __longlong_as_double(0x7FF8000000000000LL); }

// How far the chain kernels of a factorisation have come (column groups published, CTAs started) and
// the arithmetic of its panel: FP64 if the tickets' top bit is set (choose_panel_kernel). A CTA has it
// with its ticket, and a load of its own would be half a microsecond of every block.
struct ChainState {
  int groups;
  unsigned tickets;
};
constexpr unsigned kPanelFp64 = 1u << 31;

__global__ void diag_bound_kernel(const double* __restrict__ A, int64_t lda, int64_t n, RowBound bound,
                                  ChainState* __restrict__ chain, int* __restrict__ score, int* __restrict__ info) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r == 0) *chain = ChainState{0, 0u};
  if (r >= n) return;
  score[r] = 0;
  const double a = A[r * lda + r];
  float f = 0.0f;
  int E = 0;
  if (a > 0.0 && dbl_finite(a))
    f = (float)frexp(a, &E);
  else
    record_info(info, r + 1);
  bound.f[r] = f;
  bound.E[r] = E;
}

// Which arithmetic the panel takes. Fixed point keeps an entry of L to 2^-61 of its row's scale 2^e_r,
// FP64 to 2^-53 of itself: the first is the better where the entries of A are not far below sqrt(a_rr
// a_kk) (the errors of FP64's sums are those of the large products), the second where rows hardly
// interact. So the entries of A below the diagonal are counted: a weak one is not zero and below 2^-12
// 2^(e_r + e_k) (2^-9 to 2^-11 of sqrt(a_rr a_kk)), and if of any row and its column more than a quarter
// of the entries that are not zero are weak, the panel is factored in FP64. Random couplings of size c
// beside the diagonal, n = 64, median relative error of an entry of L, FP64 and fixed point: 1.1e-16 and
// 4.5e-17 at c = 2^-4, 7.9e-17 and 1.2e-16 at 2^-7 (a tenth of the entries weak), 7.7e-17 and 2.4e-16 at
// 2^-8 (a fifth, of some row more than a quarter), 7.5e-17 and 9.7e-13 at 2^-20. Of a Gram of RBM or
// ResConv samples 1 to 5% are weak (13% in a row of 6000 samples of 65536 parameters).
// One pass over the lower triangle, bound by the latency of its loads: a CTA walks along a row of tiles
// and loads the next one beside the count (n = 1056: 5 us, 8192: 53 us; 101 with a CTA per tile).
constexpr int kWeakBits = 12, kWeakTile = 64, kWeakThreads = 256;
__global__ void __launch_bounds__(kWeakThreads)
    weak_coupling_kernel(const double* __restrict__ A, int64_t lda, int64_t n, RowBound bound, int per_cta,
                         int* __restrict__ score) {
  // row tile blockIdx.y, per_cta column tiles from blockIdx.x per_cta on
  const int64_t first = blockIdx.x * (int64_t)per_cta, last = min(first + per_cta, (int64_t)blockIdx.y + 1);
  if (first >= last) return;
  __shared__ int er[kWeakTile], ec[2][kWeakTile], col_score[2][kWeakTile];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int64_t r0 = blockIdx.y * (int64_t)kWeakTile;
  constexpr int kWarps = kWeakThreads / 32, kRows = kWeakTile / kWarps;  // rows per warp
  double v[kRows][2];
  int e = 0;  // exponent of column t
  auto load = [&](int64_t tile) {
    const int64_t c0 = tile * kWeakTile;
#pragma unroll
    for (int k = 0; k < kRows; ++k)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int64_t r = r0 + warp + k * kWarps, j = c0 + 32 * q + lane;
        v[k][q] = r < n && j < r ? A[r * lda + j] : 0.0;
      }
    if (t < kWeakTile && c0 + t < n) e = row_exponent(bound, c0 + t);
  };
  load(first);
  if (t < kWeakTile) {
    er[t] = r0 + t < n ? row_exponent(bound, r0 + t) : 0;
    col_score[0][t] = col_score[1][t] = 0;
  }
  int rs[kRows] = {};  // scores: 3 for a weak entry, -1 for another that is not zero
  for (int64_t tile = first; tile < last; ++tile) {
    const int buf = (int)(tile & 1);
    uint32_t hi[kRows][2];  // exponent and leading bits, the sign out; 1 for a value that only later bits hold
#pragma unroll
    for (int k = 0; k < kRows; ++k)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint64_t b = dbl_bits(v[k][q]) << 1;
        hi[k][q] = (uint32_t)(b >> 33) | (b << 31 != 0);
      }
    if (t < kWeakTile) ec[buf][t] = e;
    if (tile + 1 < last) load(tile + 1);
    __syncthreads();
    const int limit[2] = {ec[buf][lane] - kWeakBits + 1022, ec[buf][32 + lane] - kWeakBits + 1022};
    int cs[2] = {};
#pragma unroll
    for (int k = 0; k < kRows; ++k)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        // |a| < 2^(exponent field - 1022)
        const int s = hi[k][q] == 0 ? 0 : (int)(hi[k][q] >> 20) <= er[warp + k * kWarps] + limit[q] ? 3 : -1;
        rs[k] += s;
        cs[q] += s;
      }
#pragma unroll
    for (int q = 0; q < 2; ++q) atomicAdd(&col_score[buf][32 * q + lane], cs[q]);
    __syncthreads();
    if (t < kWeakTile) {
      const int64_t c = tile * kWeakTile + t;
      if (col_score[buf][t] != 0) atomicAdd(score + c, col_score[buf][t]);
      col_score[buf][t] = 0;  // used again two tiles on
    }
  }
#pragma unroll
  for (int k = 0; k < kRows; ++k) {
    const int s = __reduce_add_sync(0xffffffffu, rs[k]);
    if (lane == 0 && s != 0) atomicAdd(score + r0 + warp + k * kWarps, s);
  }
}

constexpr int kChooseThreads = 1024;
__global__ void __launch_bounds__(kChooseThreads) choose_panel_kernel(const int* __restrict__ score, int64_t n,
                                                                      ChainState* __restrict__ chain) {
  int any = 0;
  for (int64_t r = threadIdx.x; r < n; r += kChooseThreads) any |= score[r] > 0;
  if (__syncthreads_or(any) && threadIdx.x == 0) chain->tickets = kPanelFp64;
}

// the block's factor in fixed point, as the triangular solve reads it
struct __align__(16) BlockFactor {
  Fx l[kBlk][kBlk];   // l[k][i] = L_ik 2^-e_i, i > k
  FxPivot piv[kBlk];  // m = 0: column k is not a number (a pivot at or before it failed)
};

constexpr float kFullRow = 0.52f;  // a row's squares sum to at most 1/2 (1 + rounding of its bound)
constexpr float kFxHigh = 4.656612873077393e-10f;  // 2^-31: the unit of Fx::h
// Work layout of the 64-column chain, potrf_block and trsm_block: the columns go in
// groups of four; lanes are rows, and a warp holds its 32 rows' entries of one group's columns
// (trsm: of two, w and w + 8). A group's owner scales its four columns one after the other in
// registers and publishes them in shared memory; after one barrier every warp takes the group's
// update of its later columns, the next owner first of all. A dead group costs nothing, so the
// executed multiply-adds are those of the triangle.

// A group of four columns as an update takes it: x, the entries of the lane's row (negated), and
// y, the rows of the columns that are updated
struct GroupUpdate {
  Fx x[4], y[4][4];
  // x: entry of the lane's row in the group's first column (stride ldx); y: the updated group's
  // first row of it (stride ldy)
  __device__ inline GroupUpdate(const Fx* __restrict__ xp, int ldx, const Fx* __restrict__ yp, int ldy) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = xp[k * ldx];
      x[k].h = -x[k].h;
      x[k].l = -x[k].l;
      const int4 a = *reinterpret_cast<const int4*>(yp + k * ldy), b = *reinterpret_cast<const int4*>(yp + k * ldy + 2);
      y[k][0] = Fx{a.x, a.y};
      y[k][1] = Fx{a.z, a.w};
      y[k][2] = Fx{b.x, b.y};
      y[k][3] = Fx{b.z, b.w};
    }
  }
  __device__ inline void column(int e, int64_t* s1, int64_t* s2) const {
#pragma unroll
    for (int k = 0; k < 4; ++k) fx_mad(s1[e], s2[e], x[k], y[k][e]);
  }
};

// s[e] -= sum over the group's columns k of x_k y_k[e], e the four columns of the warp's group
__device__ inline void apply_group(const Fx* __restrict__ x, int ldx, const Fx* __restrict__ y, int ldy, int64_t* s1,
                                   int64_t* s2) {
  const GroupUpdate u(x, ldx, y, ldy);
#pragma unroll
  for (int e = 0; e < 4; ++e) u.column(e, s1, s2);
}

constexpr int kPotrfThreads = 512;
constexpr int kPotrfLd = kBlk + 2;  // 16-byte rows
struct PotrfShared {
  union {
    double a[kBlk][kBlk + 1];               // the block as read, [row][column]
    __align__(16) Fx l[kBlk][kPotrfLd];     // the factor, [column][row]
  };
  FxPivot piv[kBlk];
  uint64_t u[kBlk];      // normalised pivots
  float squares[kBlk];   // of the row's entries so far
  int e[kBlk];
  int bad[kBlk];         // row cannot belong to a positive definite matrix
  int kfail;             // first column whose pivot failed
  double root[2];        // FP64: the pivot's square root and its inverse
};

// the warp's 32 rows (from row0) of the columns k0 .. k0 + 3, scaled and published; all updates are
// taken but the previous group's, which is taken here (its share of column k0 first: the chain
// waits for nothing else). PIVOT: the columns' pivots are among these rows and are inverted here
// (by every lane alike); else they were, a barrier ago.
template <bool PIVOT>
__device__ inline void solve_group(PotrfShared& sh, int k0, int row0, int lane, int64_t* s1, int64_t* s2) {
  const int i = row0 + lane;
  float squares = sh.squares[i];
  bool bad = sh.bad[i] != 0;
  int kfail = sh.kfail;
  // the first group has no previous one: any finite operand times zero
  GroupUpdate prev(&sh.l[k0 > 0 ? k0 - 4 : 0][i], kPotrfLd, &sh.l[k0 > 0 ? k0 - 4 : 0][k0], kPotrfLd);
  if (k0 == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) prev.x[k] = Fx{0, 0};
  }
  prev.column(0, s1, s2);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int k = k0 + e, src = k - row0;
    int64_t X;
    bool in_range, positive;
    if (PIVOT) {
      const int64_t p1 = __shfl_sync(0xffffffffu, bad ? 0 : s1[e], src), p2 = __shfl_sync(0xffffffffu, s2[e], src);
      const FxInverse inv = fx_inverse(kfail < kBlk ? 0 : p1, p2);
      positive = inv.Y != 0;
      in_range = fx_in_range(s1[e], inv.t);
      X = fx_scale(s1[e], s2[e], inv, in_range);
      if (!positive) kfail = min(kfail, k);
      if (lane == 0) {
        sh.piv[k] = fx_pivot(inv);
        sh.u[k] = inv.u;
      }
    } else {
      const FxPivot piv = sh.piv[k];
      positive = piv.m != 0;
      in_range = fx_in_range(s1[e], piv.t);
      X = fx_scale(s1[e], s2[e], piv, in_range);
    }
    Fx x = fx_split(X);
    if (e == 0) {
#pragma unroll
      for (int f = 1; f < 4; ++f) prev.column(f, s1, s2);
    }
    const float xv = (float)x.h * kFxHigh;
    const float sq = fmaf(xv, xv, squares);
    const bool below = i > k && positive;
    bad |= below && (!in_range || !fx_is_entry(X) || sq > kFullRow);
    if (below && !bad)
      squares = sq;
    else
      x = Fx{0, 0};
    Fx y[4];
#pragma unroll
    for (int f = e + 1; f < 4; ++f) {
      if (PIVOT) {
        y[f].h = __shfl_sync(0xffffffffu, x.h, k0 + f - row0);
        y[f].l = __shfl_sync(0xffffffffu, x.l, k0 + f - row0);
      } else {
        y[f] = sh.l[k][k0 + f];
      }
    }
    sh.l[k][i] = x;
    x.h = -x.h;
    x.l = -x.l;
#pragma unroll
    for (int f = e + 1; f < 4; ++f) fx_mad(s1[f], s2[f], x, y[f]);
  }
  sh.squares[i] = squares;
  if (bad) sh.bad[i] = 1;
  if (PIVOT && lane == 0) sh.kfail = kfail;
}

// The diagonal block's factorisation in FP64, for matrices whose rows hardly interact
// (choose_panel_kernel), from sh.a: bound by FP64 instructions (64 clocks of a sub-core each). 512
// threads as a 32 x 16 grid over the trailing block; the pivot's inverse square root scales its column.
// *groups becomes groups0 + 16 once the block can be read from A.
__device__ __noinline__ void potrf_block_fp64(PotrfShared& sh, double* __restrict__ A, int64_t lda, int64_t c, int nb,
                                        int* __restrict__ groups, int groups0, int* __restrict__ info) {
  const int t = threadIdx.x, ti = t >> 4, tj = t & 15;
  constexpr int kRows = kPotrfThreads / 16;
  for (int k = 0; k < nb; ++k) {
    if (t == 0) {
      double d = sh.a[k][k];
      if (!(d > 0.0)) {
        record_info(info, c + k + 1);
        d = quiet_nan();
      }
      const double r = rsqrt(d);
      sh.root[0] = d * r;  // sqrt(d)
      sh.root[1] = r;
    }
    __syncthreads();
    const double r = sh.root[1];
    if (t == 0) sh.a[k][k] = sh.root[0];
    for (int i = k + 1 + t; i < nb; i += kPotrfThreads) sh.a[i][k] *= r;
    __syncthreads();
    for (int i = k + 1 + ti; i < nb; i += kRows) {
      const double aik = sh.a[i][k];
      for (int j = k + 1 + tj; j <= i; j += 16) sh.a[i][j] = fma(-aik, sh.a[j][k], sh.a[i][j]);
    }
    __syncthreads();
  }
  for (int i = ti; i < nb; i += kRows)
    for (int j = tj; j <= i; j += 16) A[(c + i) * lda + c + j] = sh.a[i][j];
  __threadfence();
  __syncthreads();
  if (t == 0)
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(groups), "r"(groups0 + kBlk / 4) : "memory");
}

// Cholesky of the nb x nb (nb <= 64) diagonal block at (c, c), in place, in fixed point. The
// first pivot that is not positive makes the remaining columns NaN and is recorded in *info as
// c + k + 1 (the order of the failing leading minor, as LAPACK and cuSOLVER report it). Eight warps
// hold rows 0 .. 31, one column group each, and eight rows 32 .. 63, two groups each; the lower
// rows follow the upper ones by one group. The chain of 64 pivots bounds it (one CTA), so
// the lower rows' multiply-adds and the stores are kept off the sub-cores that the chain runs on.
// Measured: 30 us a block (62 us in FP64), about 780 clocks a column, of which the inverse square
// root and the scaling take 500. Complete groups are published in `out` for the triangular solve:
// *groups becomes groups0 + g + 1 once group g can be read.
__device__ inline void potrf_block(PotrfShared& sh, bool fp64, double* __restrict__ A, int64_t lda, int64_t c, int nb,
                                   RowBound bound, BlockFactor* __restrict__ out, int* __restrict__ groups, int groups0,
                                   int* __restrict__ info) {
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  if (t < kBlk) {
    sh.e[t] = t < nb ? row_exponent(bound, c + t) : 0;
    sh.bad[t] = 0;
    sh.squares[t] = 0.0f;
  }
  if (t == 0) sh.kfail = kBlk;
#pragma unroll
  for (int q = 0; q < kBlk * kBlk / kPotrfThreads; ++q) {
    const int r = (t >> 6) + q * (kPotrfThreads / kBlk), j = t & 63;
    sh.a[r][j] = r < nb && j <= r ? A[(c + r) * lda + c + j] : 0.0;
  }
  __syncthreads();
  if (fp64) {
    potrf_block_fp64(sh, A, lda, c, nb, groups, groups0, info);
    return;
  }
  // warps 0, 1 (mod 4): the upper rows, on two of the SM's four sub-cores; 2, 3: the lower ones
  const bool lower = (w & 2) != 0;
  const int g0 = (w >> 2) * 2 + (w & 1), row0 = lower ? 32 : 0, i = row0 + lane;
  int64_t s1[8], s2[8];  // columns 4 g0 .. and, in the lower rows, 32 + 4 g0 ..
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    s1[q] = s2[q] = 0;
    if (q >= 4 && !lower) continue;
    const int j = 4 * g0 + (q & 3) + (q >> 2) * 32;
    const double a = sh.a[i][j];
    if (!dbl_finite(a)) sh.bad[i] = 1;
    // rows past the matrix: a diagonal of 1/4
    s1[q] = i == j && i >= nb ? 1LL << 60 : fx_from_double(a, sh.e[i] + sh.e[j], 62);
  }
  __syncthreads();
  // column k of 32 rows (of half h) to the matrix
  auto store_column = [&](int k, int h) {
    const int r = 32 * h + lane;
    const Fx x = sh.l[k][r];
    if (r >= nb || r < k) return;
    double v;
    if (k >= sh.kfail)
      v = quiet_nan();
    else if (r == k)
      v = fx_to_double(fx_sqrt(sh.u[k], sh.piv[k]), sh.e[k] - sh.piv[k].t - 61);
    else
      v = fx_to_double(fx_join(x), sh.e[r] - kFxBits);
    A[(c + r) * lda + c + k] = v;
  };
  auto store_group = [&](int g, int h) {
#pragma unroll 1
    for (int e = 0; e < 4; ++e) store_column(4 * g + e, h);
  };
  // group g, complete in both halves, to the triangular solve (one warp)
  auto publish = [&](int g) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = 4 * g + e;
      if (g < 8) out->l[k][lane] = sh.l[k][lane];
      out->l[k][32 + lane] = sh.l[k][32 + lane];
    }
    if (lane < 4) out->piv[4 * g + lane] = sh.piv[4 * g + lane];
    __threadfence();
    __syncwarp();
    if (lane == 0)
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(groups), "r"(groups0 + g + 1) : "memory");
  };
#pragma unroll 1
  for (int step = 0; step < 9; ++step) {
    const int g = lower ? step - 1 : step;  // the group these rows solve
    if (g >= 0 && g < 8) {
      const int k0 = 4 * (g - 1);  // the previous group's first column
      if (g0 == g) {
        if (lower)
          solve_group<false>(sh, 4 * g, row0, lane, s1, s2);
        else
          solve_group<true>(sh, 4 * g, row0, lane, s1, s2);
      } else if (g0 > g && g > 0) {
        apply_group(&sh.l[k0][i], kPotrfLd, &sh.l[k0][4 * g0], kPotrfLd, s1, s2);
      }
      if (lower && g > 0) apply_group(&sh.l[k0][i], kPotrfLd, &sh.l[k0][32 + 4 * g0], kPotrfLd, s1 + 4, s2 + 4);
    }
    if (!lower && g0 == step - 2) publish(g0);
    __syncthreads();
  }
#pragma unroll 1
  for (int g = 8; g < 16; ++g) {
    const int k0 = 4 * (g - 1);
    if (lower) {
      if (g0 == g - 8)
        solve_group<true>(sh, 4 * g, row0, lane, s1 + 4, s2 + 4);
      else if (g0 > g - 8)
        apply_group(&sh.l[k0][i], kPotrfLd, &sh.l[k0][32 + 4 * g0], kPotrfLd, s1 + 4, s2 + 4);
    } else if (g0 == g - 8) {
      store_group(g0, 0);
    } else if (g0 == ((g - 7) & 7)) {
      store_group(g0, 1);
    } else if (g > 8 && g0 == ((g - 6) & 7)) {
      store_group(g - 1, 1);
    } else if (g0 == ((g - 5) & 7)) {
      publish(g - 1);
    }
    __syncthreads();
  }
  if (!lower && g0 == 4) publish(15);
  if (!lower && g0 < 4) store_column(60 + g0, 1);
  if (t == 0 && sh.kfail < nb) record_info(info, c + sh.kfail + 1);
}

// The 8 digits of F0 and F1 (|F| <= 2^56), columns k and k + 1 (k even) of slice row r, into the
// slices of kblocks 32-column blocks. With 64 added at each of the seven lower places the balanced
// digits are the 7-bit fields minus 64, the top one the remaining signed part.
__device__ inline void store_digits(uint8_t* S, int kblocks, int64_t r, int k, int64_t F0, int64_t F1) {
  const int row = (int)(r & (kOzM - 1)), chunk = ((k >> 3) & 3) ^ ((row >> 1) & 3);
  uint8_t* s = S + ((r / kOzM) * kblocks + (k >> 5)) * (int64_t)kOzABytes + row * kOzRowBytes + chunk * 16 + (k & 7) * 2;
  const uint64_t F[2] = {(uint64_t)F0 + 0x1020408102040ULL, (uint64_t)F1 + 0x1020408102040ULL};
#pragma unroll
  for (int t = 0; t < kSlices; ++t) {
    uint32_t w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int d = t == 0 ? (int)((int64_t)F[h] >> 49) : (int)((uint32_t)(F[h] >> (7 * (7 - t))) & 127) - 64;
      w[h] = __float_as_uint(__int_as_float(0x4B400000 + d) - 12582912.0f);  // (float)d
    }
    // the high halves: exact in BF16
    *reinterpret_cast<uint32_t*>(s + t * (kOzM * kOzRowBytes)) = __byte_perm(w[0], w[1], 0x7632);
  }
}

// Rows first .. first + 32 TILES - 1 of the 64 columns at c: x L_cc^T = a with L_cc the diagonal
// block's factor, in place, and, for the update of the panel's later columns, the rows' digit slices S
// (slice row r - r0) with exponents ex (S may be NULL). Eight warps per tile of 32 rows. Bound by the
// integer pipe at many rows (2016 multiply-adds of three instructions per row), by the chain of 64
// scalings at few. A row whose squares exceed its bound cannot be completed to a positive definite
// matrix: its order is recorded and it becomes NaN. FOLLOW: the factorisation may still run; a warp
// more copies its column groups to shared memory as they are published (*groups reaches groups0 + g +
// 1), and the solve goes on with each as it comes. Else the whole factor is there.
constexpr int kTileWarps = 8, kTileRows = 32;
struct TrsmTile {
  union {
    double a[kTileRows][kBlk + 1];  // the rows as read
    Fx x[kBlk][kTileRows + 1];      // the solution, [column][row]
  };
  float squares[kTileRows];
  int bad[kTileRows], nan_row[kTileRows], er[kTileRows];
};
template <int TILES>
struct TrsmShared {
  BlockFactor f;
  TrsmTile tile[TILES];
  int e[kBlk];
  uint64_t full[kBlk / 4];  // FOLLOW: column group copied
  int fail;                 // a wait ran out
};

__device__ inline void trsm_group(const BlockFactor& f, TrsmTile& sh, int k0, int lane, int64_t* s1, int64_t* s2) {
  float squares = sh.squares[lane];
  bool bad = sh.bad[lane] != 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int k = k0 + e;
    const FxPivot piv = f.piv[k];
    const bool in_range = fx_in_range(s1[e], piv.t);
    const int64_t X = fx_scale(s1[e], s2[e], piv, in_range);
    Fx x = fx_split(X);
    const float xv = (float)x.h * kFxHigh;
    squares = fmaf(xv, xv, squares);
    bad |= !in_range || !fx_is_entry(X) || squares > kFullRow;
    if (bad) x = Fx{0, 0};
    sh.x[k][lane] = x;
    x.h = -x.h;
    x.l = -x.l;
#pragma unroll
    for (int q = e + 1; q < 4; ++q) fx_mad(s1[q], s2[q], x, f.l[k][k0 + q]);
  }
  sh.squares[lane] = squares;
  if (bad) sh.bad[lane] = 1;
}

template <int TILES, bool FOLLOW>
__device__ inline void trsm_block(TrsmShared<TILES>& sh, double* __restrict__ A, int64_t lda, int64_t c, int64_t r0,
                                  int64_t first, int64_t n, RowBound bound, const BlockFactor* __restrict__ factor,
                                  const int* __restrict__ groups, int groups0, uint8_t* __restrict__ S,
                                  int* __restrict__ ex, int* __restrict__ info, int32_t* __restrict__ status) {
  constexpr int kSolvers = 32 * kTileWarps * TILES;  // threads
  const int t = threadIdx.x, lane = t & 31;
  if (t >= kSolvers + (FOLLOW ? 32 : 0)) return;
  static_assert(sizeof(BlockFactor) % 16 == 0 && sizeof(FxPivot) == 16 && sizeof(Fx) == 8, "copied in 16-byte words");
  if (!FOLLOW) {
#pragma unroll
    for (int e = t; e < (int)(sizeof(BlockFactor) / 16); e += kSolvers)
      reinterpret_cast<int4*>(&sh.f)[e] = reinterpret_cast<const int4*>(factor)[e];
  }
  if (t == 0) {
    if (FOLLOW)
      for (int g = 0; g < kBlk / 4; ++g) mbar_init(&sh.full[g], 1);
    sh.fail = 0;
  }
  if (t < kBlk) sh.e[t] = row_exponent(bound, c + t);
  if (t < TILES * kTileRows) {
    TrsmTile& tl = sh.tile[t / kTileRows];
    const int r = t % kTileRows;
    tl.er[r] = first + t < n ? row_exponent(bound, first + t) : 0;
    tl.squares[r] = 0.0f;
    tl.bad[r] = 0;
    tl.nan_row[r] = 0;
  }
  if (t < kSolvers) {
#pragma unroll
    for (int e = t; e < TILES * kTileRows * kBlk; e += kSolvers) {
      const int r = e >> 6, j = e & 63;
      // rows past the matrix solve zeros
      sh.tile[r / kTileRows].a[r % kTileRows][j] = first + r < n ? A[(first + r) * lda + c + j] : 0.0;
    }
  }
  __syncthreads();
  if (FOLLOW && t >= kSolvers) {  // the copying warp
    int seen = groups0;
    bool ok = true;
    for (int g = 0; g < kBlk / 4; ++g) {
      const uint64_t t0 = global_timer();
      while (ok && seen - groups0 <= g) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(groups) : "memory");
        if (seen - groups0 <= g && global_timer() - t0 > kWaitLimitNs) ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        sh.fail = 1;  // the rows become NaN; the missing pivots count as failed
        if (lane < 4) sh.f.piv[4 * g + lane] = FxPivot{0, 0};
      } else {
        const int4* src = reinterpret_cast<const int4*>(&factor->l[4 * g][0]);
        int4* dst = reinterpret_cast<int4*>(&sh.f.l[4 * g][0]);
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[lane + 32 * q] = __ldcg(src + lane + 32 * q);
        if (lane < 4)
          reinterpret_cast<int4*>(sh.f.piv)[4 * g + lane] = __ldcg(reinterpret_cast<const int4*>(factor->piv) + 4 * g + lane);
      }
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&sh.full[g])) : "memory");
    }
    return;
  }
  const int tile = t / (32 * kTileWarps), w = (t >> 5) % kTileWarps;
  TrsmTile& tl = sh.tile[tile];
  auto tile_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + tile), "r"(32 * kTileWarps) : "memory"); };
  auto wait_group = [&](int g) {
    if (FOLLOW && !mbar_wait(&sh.full[g], 0)) sh.fail = 1;
  };
  int64_t s1[8], s2[8];  // columns 4 w .. 4 w + 3 and 32 + 4 w ..
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int j = 4 * w + (q & 3) + (q >> 2) * 32;
    const double a = tl.a[lane][j];
    if (!dbl_finite(a)) tl.nan_row[lane] = 1;
    s1[q] = fx_from_double(a, tl.er[lane] + sh.e[j], 62);
    s2[q] = 0;
  }
  tile_sync();
#pragma unroll 1
  for (int g = 0; g < 8; ++g) {
    const int k0 = 4 * (g - 1);
    if (g > 0) wait_group(g - 1);
    if (w >= g) {
      if (g > 0) apply_group(&tl.x[k0][lane], kTileRows + 1, &sh.f.l[k0][4 * w], kBlk, s1, s2);
      if (w == g) {
        wait_group(g);
        trsm_group(sh.f, tl, 4 * g, lane, s1, s2);
      }
    }
    // the owner publishes before it goes on to its second group
    if (w == g) tile_sync();
    if (g > 0) apply_group(&tl.x[k0][lane], kTileRows + 1, &sh.f.l[k0][32 + 4 * w], kBlk, s1 + 4, s2 + 4);
    if (w != g) tile_sync();
  }
#pragma unroll 1
  for (int g = 8; g < 16; ++g) {
    const int k0 = 4 * (g - 1);
    wait_group(g - 1);
    if (w >= g - 8) {
      apply_group(&tl.x[k0][lane], kTileRows + 1, &sh.f.l[k0][32 + 4 * w], kBlk, s1 + 4, s2 + 4);
      if (w == g - 8) {
        wait_group(g);
        trsm_group(sh.f, tl, 4 * g, lane, s1 + 4, s2 + 4);
      }
    }
    tile_sync();
  }
  wait_group(15);
  const bool fail = *reinterpret_cast<volatile int*>(&sh.fail) != 0;
  if (fail && status && lane == 0) atomicExch(status, QGX_ERR_TIMEOUT);
  // four rows per warp, two neighbouring columns per lane
  const bool pivots0 = sh.f.piv[2 * lane].m != 0, pivots1 = sh.f.piv[2 * lane + 1].m != 0;
#pragma unroll 1
  for (int rl = w; rl < kTileRows; rl += kTileWarps) {
    const int64_t rr = first + tile * kTileRows + rl;
    if (rr >= n) break;
    const bool bad = tl.bad[rl] != 0, nans = bad || fail || tl.nan_row[rl] != 0;
    const int e = tl.er[rl];
    if (bad && lane == 0) record_info(info, rr + 1);
    const int64_t X0 = fx_join(tl.x[2 * lane][rl]), X1 = fx_join(tl.x[2 * lane + 1][rl]);
    double* out = A + rr * lda + c + 2 * lane;
    out[0] = nans || !pivots0 ? quiet_nan() : fx_to_double(X0, e - kFxBits);
    out[1] = nans || !pivots1 ? quiet_nan() : fx_to_double(X1, e - kFxBits);
    if (S == nullptr) continue;
    // every |X| < 2^bits: exponent e + bits - 60, F = X 2^(56 - bits)
    const uint64_t a0 = X0 < 0 ? 0ULL - (uint64_t)X0 : (uint64_t)X0, a1 = X1 < 0 ? 0ULL - (uint64_t)X1 : (uint64_t)X1;
    const int bits = __reduce_max_sync(0xffffffffu, 64 - clz64(a0 | a1));
    const int up = 56 - bits;
    const int64_t F0 = up >= 0 ? (int64_t)((uint64_t)X0 << up) : (X0 + (1LL << (-up - 1))) >> -up;
    const int64_t F1 = up >= 0 ? (int64_t)((uint64_t)X1 << up) : (X1 + (1LL << (-up - 1))) >> -up;
    const int64_t sr = rr - r0;
    if (lane == 0) ex[sr] = bits == 0 ? 0 : e + bits - kFxBits;
    store_digits(S, kBlk / kOzKB, sr, 2 * lane, F0, F1);
  }
}

// The same in FP64, for matrices whose rows hardly interact (choose_panel_kernel), from the diagonal
// block in A (FOLLOW: once it is published whole). Eight lanes per row, lane l holding columns l, l + 8,
// ..., l + 56: the owner of column k scales it and hands it to the others, which update their later
// columns. Bound by FP64 instructions.
struct TrsmFp64Shared {
  double l[kBlk][kBlk + 1];
  double rec[kBlk];  // 1 / l_kk
  int fail;          // the wait ran out
};
template <int TILES, bool FOLLOW>
__device__ inline void trsm_block_fp64(TrsmFp64Shared& sh, double* __restrict__ A, int64_t lda, int64_t c, int64_t r0,
                                       int64_t first, int64_t n, const int* __restrict__ groups, int groups0,
                                       uint8_t* __restrict__ S, int* __restrict__ ex, int32_t* __restrict__ status) {
  constexpr int kSolvers = 32 * kTileWarps * TILES;  // threads, eight per row
  const int t = threadIdx.x;
  if (t >= kSolvers) return;
  if (t == 0) {
    int seen = groups0 + kBlk / 4;
    if (FOLLOW) {
      const uint64_t t0 = global_timer();
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(groups) : "memory");
      } while (seen - groups0 < kBlk / 4 && global_timer() - t0 <= kWaitLimitNs);
    }
    sh.fail = seen - groups0 < kBlk / 4;
    if (sh.fail && status) atomicExch(status, QGX_ERR_TIMEOUT);
  }
  __syncthreads();
  for (int e = t; e < kBlk * kBlk; e += kSolvers) {
    const int i = e / kBlk, j = e % kBlk;
    sh.l[i][j] = j <= i ? __ldcg(A + (c + i) * lda + c + j) : 0.0;
  }
  __syncthreads();
  if (t < kBlk) sh.rec[t] = 1.0 / sh.l[t][t];
  __syncthreads();
  const int sub = t & 7;
  const int64_t r = first + (t >> 3);
  const bool live = r < n;  // eight lanes share a row; those past the matrix solve zeros
  double* row = A + (live ? r : r0) * lda + c;
  double x[kBlk / 8];
#pragma unroll
  for (int q = 0; q < kBlk / 8; ++q) x[q] = live ? row[8 * q + sub] : 0.0;
#pragma unroll
  for (int k = 0; k < kBlk; ++k) {
    const int qk = k >> 3;
    double xk = 0.0;
    if (sub == (k & 7)) {
      x[qk] *= sh.rec[k];
      xk = x[qk];
    }
    xk = __shfl_sync(0xffffffffu, xk, k & 7, 8);
#pragma unroll
    for (int q = 0; q < kBlk / 8; ++q)
      if (8 * q + sub > k) x[q] = fma(-xk, sh.l[8 * q + sub][k], x[q]);
  }
  uint64_t mx = 0;
#pragma unroll
  for (int q = 0; q < kBlk / 8; ++q) {
    if (sh.fail) x[q] = quiet_nan();
    if (live) row[8 * q + sub] = x[q];
    const uint64_t b = dbl_bits(x[q]) & 0x7FFFFFFFFFFFFFFFULL;
    mx = b < 0x7FF0000000000000ULL && b > mx ? b : mx;  // NaN and infinities slice as zero
  }
  if (S == nullptr) return;
  // the row's exponent and digits, as slice_rows_kernel takes them
  int top = mx == 0 ? -1 : max((int)(mx >> 52), 1);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
  const int e = top < 0 ? 0 : top - 1022;
  if (live && sub == 0) ex[r - r0] = e;
#pragma unroll
  for (int q = 0; q < kBlk / 8; ++q) {
    const int64_t F = fx_from_double(x[q], e, kFixBits);
    const int64_t next = __shfl_down_sync(0xffffffffu, F, 1);
    if (live && (sub & 1) == 0) store_digits(S, kBlk / kOzKB, r - r0, 8 * q + sub, F, next);
  }
}

template <int TILES>
union ChainShared {
  PotrfShared potrf;
  TrsmShared<TILES> trsm;
  TrsmFp64Shared trsm_fp64;
};
constexpr int chain_threads(int tiles) { return std::max(kPotrfThreads, 32 * (kTileWarps * tiles + 1)); }

// One 64-column block of the panel chain in one launch: the diagonal block's factorisation (role 0) and
// the triangular solve of the rows below (32 TILES rows per further role), which follows it a few column
// groups behind and ends a few microseconds after it. A CTA's role is the order in which the CTAs
// start: the factorisation is running before any CTA waits for it. The waiting CTAs keep their SMs from
// the trailing update that runs beside, so this is for rows that leave it some; one tile per CTA, with
// no other tile's integer work beside the chain, where there are few. About 50 us a block with the
// update of the next columns (62 as two launches): n = 1056: 1.06 -> 0.87 ms, 4096: 4.36 -> 3.63, 8192:
// 11.5 -> 10.5. Jobs on other streams do not pay for it: eight served together run at 96.4 steps/s, 94.6
// with two launches.
template <int TILES>
__global__ void __launch_bounds__(chain_threads(TILES), 1)
    chain_block_kernel(double* __restrict__ A, int64_t lda, int64_t c, int nb, int64_t n, RowBound bound,
                       BlockFactor* __restrict__ factor, uint8_t* __restrict__ S, int* __restrict__ ex,
                       ChainState* __restrict__ chain, int groups0, unsigned tickets0, int* __restrict__ info,
                       int32_t* __restrict__ status) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  ChainShared<TILES>& sh = *reinterpret_cast<ChainShared<TILES>*>(smem_raw);
  __shared__ unsigned role_slot;
  if (threadIdx.x == 0) role_slot = atomicAdd(&chain->tickets, 1u) - tickets0;
  __syncthreads();
  const bool fp64 = (role_slot & kPanelFp64) != 0;
  const unsigned role = role_slot & ~kPanelFp64;
  if (role == 0) {
    if (threadIdx.x < kPotrfThreads)
      potrf_block(sh.potrf, fp64, A, lda, c, nb, bound, factor, &chain->groups, groups0, info);
  } else {
    const int64_t r0 = c + kBlk, first = r0 + (int64_t)(role - 1) * TILES * kTileRows;
    if (fp64) {
      trsm_block_fp64<TILES, true>(sh.trsm_fp64, A, lda, c, r0, first, n, &chain->groups, groups0, S, ex, status);
      return;
    }
    trsm_block<TILES, true>(sh.trsm, A, lda, c, r0, first, n, bound, factor, &chain->groups, groups0, S, ex, info,
                            status);
  }
}

// the same as two launches
__global__ void __launch_bounds__(kPotrfThreads) potrf_block_kernel(double* __restrict__ A, int64_t lda, int64_t c,
                                                                    int nb, RowBound bound,
                                                                    BlockFactor* __restrict__ factor,
                                                                    ChainState* __restrict__ chain, int groups0,
                                                                    int* __restrict__ info) {
  __shared__ PotrfShared sh;
  potrf_block(sh, (__ldcg(&chain->tickets) & kPanelFp64) != 0, A, lda, c, nb, bound, factor, &chain->groups, groups0, info);
}

__global__ void __launch_bounds__(32 * kTileWarps) trsm_block_kernel(double* __restrict__ A, int64_t lda, int64_t c,
                                                                     int64_t n, RowBound bound,
                                                                     const BlockFactor* __restrict__ factor,
                                                                     const ChainState* __restrict__ chain,
                                                                     uint8_t* __restrict__ S, int* __restrict__ ex,
                                                                     int* __restrict__ info) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int64_t r0 = c + kBlk, first = r0 + (int64_t)blockIdx.x * kTileRows;
  if ((__ldcg(&chain->tickets) & kPanelFp64) != 0) {
    trsm_block_fp64<1, false>(*reinterpret_cast<TrsmFp64Shared*>(smem_raw), A, lda, c, r0, first, n, nullptr, 0, S, ex,
                              nullptr);
    return;
  }
  trsm_block<1, false>(*reinterpret_cast<TrsmShared<1>*>(smem_raw), A, lda, c, r0, first, n, bound, factor, nullptr, 0, S,
                       ex, info, nullptr);
}

// ---- digit slices ---------------------------------------------------------------------------
// Rows [0, m) of a 256-column panel (row r at A + (row0 + r) lda + col0): exponent e_r and the
// 8 BF16 digit slices S, and the rows' bounds lowered by the panel's squares. One warp per row, two
// neighbouring columns per lane and step, integer arithmetic throughout (an FP64 compare or conversion
// costs 64 clocks per warp): 12 us for 8000 rows, 49 MB read and written (61 us with FP64 arithmetic
// and two-byte stores).
__global__ void slice_rows_kernel(const double* __restrict__ A, int64_t lda, int64_t row0, int64_t col0, int64_t m,
                                  uint8_t* __restrict__ S, int* __restrict__ ex, RowBound bound) {
  const int64_t r = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= m) return;  // whole warps
  const double* a = A + (row0 + r) * lda + col0;
  constexpr int kSteps = kPanel / 64;
  double v[kSteps][2];
  uint64_t mx = 0;
#pragma unroll
  for (int i = 0; i < kSteps; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      v[i][h] = a[64 * i + 2 * lane + h];
      const uint64_t b = dbl_bits(v[i][h]) & 0x7FFFFFFFFFFFFFFFULL;
      mx = b < 0x7FF0000000000000ULL && b > mx ? b : mx;  // NaN and infinities slice as zero
    }
  // the exponent with every |a_k| < 2^e; 0 for a zero row
  const int top = __reduce_max_sync(0xffffffffu, mx == 0 ? -1 : max((int)(mx >> 52), 1));
  const int e = top < 0 ? 0 : top - 1022;
  if (lane == 0) ex[r] = e;
  float squares = 0.0f;
#pragma unroll
  for (int i = 0; i < kSteps; ++i) {
    int64_t F[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      F[h] = fx_from_double(v[i][h], e, kFixBits);                // |F| <= 2^56
      const float x = (float)(int)(F[h] >> 26) * 9.3132257e-10f;  // 2^-30
      squares = fmaf(x, x, squares);
    }
    store_digits(S, kPanel / kOzKB, r, 64 * i + 2 * lane, F[0], F[1]);
  }
  squares = warp_sum(squares);
  // the squares are taken 2^-10 short, far more than the rounding of the float sums: the bound
  // stays one
  if (lane == 0) bound.f[row0 + r] -= 0.999f * ldexpf(squares, 2 * e - bound.E[row0 + r]);
}

// ---- tensor-core update C -= P P^T (lower part) ----------------------------------------------
// K-major BF16 operand rows of 64 bytes, 64-byte swizzle: 8-row groups 512 bytes apart
__device__ inline uint64_t desc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);  // start address
  d |= (uint64_t)1 << 16;                   // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(512 >> 4) << 32;          // stride byte offset: 8 rows x 64 bytes
  d |= (uint64_t)1 << 46;                   // descriptor version of tcgen05
  d |= (uint64_t)4 << 61;                   // 64-byte swizzle
  return d;
}

// BF16 x BF16 -> FP32, K-major A and B, M = 128, N = n (a multiple of 16, at most 256)
constexpr uint32_t oz_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kOzM >> 4) << 24);
}

__device__ inline void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

// bulk copy of bytes (a multiple of 16) from global to shared memory, both 16-byte aligned
__device__ inline void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// 16 columns of this warp's 32 TMEM lanes into registers, without waiting (tmem_wait_ld makes
// them usable): several loads can be in flight behind one wait
__device__ inline void tmem_ld_16cols_nowait(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__device__ inline void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Tile `index` of the lower part of an m x ncols region whose diagonal starts at its corner, in
// groups of kOzGroup row tiles, column by column inside a group, so that the tiles in flight share
// operand blocks in L2. False for the enumeration's tiles above the diagonal (among a group's last
// columns), which the caller skips.
__device__ inline bool oz_tile(int64_t index, int64_t m, int64_t ncols, int64_t* bi, int64_t* bj) {
  const int64_t nr = (m + kOzM - 1) / kOzM, nc = (ncols + kOzN - 1) / kOzN;
  for (int64_t g = 0; g * kOzGroup < nr; ++g) {
    const int64_t rows = min((int64_t)kOzGroup, nr - g * kOzGroup);
    const int64_t cols = min(nc, 2 * (g * kOzGroup + rows));
    if (index < rows * cols) {
      *bi = g * kOzGroup + index % rows;
      *bj = index / rows;
      return *bj <= 2 * *bi + 1;
    }
    index -= rows * cols;
  }
  return false;
}

// C[i][j] -= sum_k P[i][k] P[j][k] for i >= j in the m x ncols region at C (ldc), slice row
// off + i (off a multiple of 128) being P's row i; kblocks 32-column blocks of P.
//
// Warps 0-7: epilogue; warp 8: the producer; warp 9: the MMA issuer. Per 16-element K step the
// issuer multiplies each A slice t (M 128) with the B slices u = 0 .. 7 - t, which lie side by side
// in shared memory, so D's 64-column block u is S_t S_u^T and lands in the accumulator of level
// t + u: levels t .. 7 are one contiguous range of N = 64 (8 - t) columns, taken in instructions of
// at most 256. Every level sum stays an integer below 2^24, so the FP32 accumulation is exact in
// any order. The eight accumulators fill the tensor memory; the epilogue warps (warp w: TMEM lanes
// 32 (w mod 4) .., columns 32 (w / 4) ..) first fold all levels into registers, which frees it for
// the next tile's MMAs, and update C beside those, through transpose buffers of eight columns.
//
// Why 128 x 64: the MMAs of a K step take 1152 clocks at the tensor cores' rate and its operands are
// 48 KB, 42 bytes a clock and SM out of L2 (71 for 128 x 32 tiles). Why a few tiles per CTA and not
// a persistent grid: the panel chain of the look-ahead runs beside this kernel and gets an SM only
// when a CTA ends. Measured: 1.67 ms for the 15872-row update of a 16384 factorisation, tensor pipe
// 59% (31.5% for 128 x 32 tiles, two CTAs per SM, single 80 KB stages, 36 products of N = 32 ..
// 256); L2 runs at a quarter of its rate, so the rest is most likely the drain of the accumulators between
// tiles and the first and last tile of a CTA. The factorisation at n = 32768: 343 ms, 617 before.
__global__ void __launch_bounds__(kOzThreads, 1)
    ozaki_syrk_kernel(const uint8_t* __restrict__ S, const int* __restrict__ ex, int kblocks, int off, int64_t m,
                      int64_t ncols, double* __restrict__ C, int64_t ldc, int64_t tiles, int per_cta,
                      int32_t* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  double* turn = reinterpret_cast<double*>(smem + kOzStages * kOzStageBytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kOzStages * kOzStageBytes + kOzTurnBytes);
  uint64_t* empty = full + kOzStages;
  uint64_t* acc_full = empty + kOzStages;
  uint64_t* acc_empty = acc_full + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
  volatile int* fail = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kOzStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, kOzEpiWarps);
    *fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(kOzTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int64_t first = blockIdx.x * (int64_t)per_cta, last = min(tiles, first + per_cta);
  int64_t bi = 0, bj = 0;

  if (warp == kOzEpiWarps) {
    if (lane == 0) {
      int it = 0;  // stage loads issued
      for (int64_t tile = first; tile < last && !*fail; ++tile) {
        if (!oz_tile(tile, m, ncols, &bi, &bj)) continue;
        const uint8_t* a = S + (off / kOzM + bi) * kblocks * (int64_t)kOzABytes;
        const int64_t br = off / kOzN + bj;  // 64-row half blocks
        const uint8_t* b = S + (br >> 1) * kblocks * (int64_t)kOzABytes + (br & 1) * (kOzN * kOzRowBytes);
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % kOzStages;
          if (!mbar_wait(&empty[s], (uint32_t)((it / kOzStages) & 1) ^ 1u)) {
            *fail = 1;
            break;
          }
          uint8_t* dst = smem + s * kOzStageBytes;
          mbar_expect_tx(&full[s], kOzStageBytes);
          bulk_load(dst, a + kb * (int64_t)kOzABytes, kOzABytes, &full[s]);
#pragma unroll
          for (int t = 0; t < kSlices; ++t)
            bulk_load(dst + kOzABytes + t * (kOzN * kOzRowBytes),
                      b + kb * (int64_t)kOzABytes + t * (kOzM * kOzRowBytes), kOzN * kOzRowBytes, &full[s]);
        }
      }
      if (*fail)  // no copy may land in shared memory after the CTA has left: wait (bounded)
        for (int k = max(0, it - kOzStages); k < it; ++k)
          mbar_wait(&full[k % kOzStages], (uint32_t)((k / kOzStages) & 1));
    }
  } else if (warp == kOzEpiWarps + 1) {
    if (lane == 0) {
      int it = 0, done = 0;  // stages consumed, tiles issued
      for (int64_t tile = first; tile < last && !*fail; ++tile) {
        if (!oz_tile(tile, m, ncols, &bi, &bj)) continue;
        if (done > 0 && !mbar_wait(acc_empty, (uint32_t)(done - 1) & 1u)) {
          *fail = 1;
          break;
        }
        tc_fence_after();
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % kOzStages;
          if (!mbar_wait(&full[s], (uint32_t)((it / kOzStages) & 1))) {
            *fail = 1;
            break;
          }
          tc_fence_after();
          const uint32_t base = smem_u32(smem + s * kOzStageBytes);
#pragma unroll 1
          for (int kk = 0; kk < kOzKB / 16; ++kk) {  // 32 bytes of K per instruction
#pragma unroll
            for (int t = 0; t < kSlices; ++t) {
              const uint64_t da = desc_sw64(base + t * (kOzM * kOzRowBytes) + kk * 32);
#pragma unroll
              for (int u = 0; u < kSlices - t; u += 4) {
                const int n = kOzN * (kSlices - t - u < 4 ? kSlices - t - u : 4);
                const uint64_t db = desc_sw64(base + kOzABytes + u * (kOzN * kOzRowBytes) + kk * 32);
                mma_bf16(tmem + (uint32_t)(kOzN * (t + u)), da, db, oz_idesc(n), (kb == 0 && kk == 0 && t == 0) ? 0u : 1u);
              }
            }
          }
          mma_commit(&empty[s]);
        }
        mma_commit(acc_full);  // also after a failed wait: tracks every MMA issued so far
        if (*fail) mbar_wait(acc_full, (uint32_t)done & 1u);
        ++done;
      }
    }
  } else {
    const int q = warp & 3, cols0 = 32 * (warp >> 2);
    double* tr = turn + warp * 32 * kOzTurnLd;
    int done = 0;
    for (int64_t tile = first; tile < last && !*fail; ++tile) {
      if (!oz_tile(tile, m, ncols, &bi, &bj)) continue;
      const int64_t row0 = bi * kOzM + 32 * q, col0 = bj * kOzN + cols0;
      const int64_t i = row0 + lane;
      const int ei = i < m ? ex[off + i] : 0;
      const int ej = col0 + lane < ncols ? ex[off + col0 + lane] : 0;
      // while the MMAs run: this warp's part of C into L2 (lane: one row, two lines)
      if (i < m) {
        if (col0 < ncols) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + i * ldc + col0));
        if (col0 + 16 < ncols) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + i * ldc + col0 + 16));
      }
      if (!mbar_wait(acc_full, (uint32_t)done & 1u) || *fail) {
        *fail = 1;
        break;
      }
      ++done;
      tc_fence_after();
      int64_t v[32];
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const uint32_t addr = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(cols0 + 16 * g);
        // two neighbouring levels fit 32 bits: |I_l| < 2^23.4, so |128 I_l + I_(l+1)| < 2^31
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t r[4][16];
#pragma unroll
          for (int l = 0; l < 4; ++l) tmem_ld_16cols_nowait(addr + (uint32_t)(kOzN * (4 * half + l)), r[l]);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            auto level = [&](int l) { return __float2int_rn(__uint_as_float(r[l][j])); };
            const int hi = 128 * level(0) + level(1), lo = 128 * level(2) + level(3);
            // V = sum_l I_l 2^(38 - 7 l), levels 6 and 7 rounded to 2^-38 together
            if (half == 0)
              v[16 * g + j] = ((int64_t)hi << 31) + ((int64_t)lo << 17);
            else
              v[16 * g + j] += ((int64_t)hi << 3) + ((lo + 1024) >> 11);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(acc_empty)) : "memory");
      // C[i][j] -= 2^(e_i + e_j - 52) V_ij, eight columns a turn: lane = row into the buffer, then
      // four rows of 64 bytes per access
      const int rr = lane >> 3, cc = lane & 7;
#pragma unroll
      for (int c = 0; c < 32; c += kOzTurn) {
#pragma unroll
        for (int j = 0; j < kOzTurn; ++j)
          tr[lane * kOzTurnLd + j] = fx_to_double(v[c + j], ei + __shfl_sync(0xffffffffu, ej, c + j) - 52);
        __syncwarp();
        double cv[8];
        const int64_t j = col0 + c + cc;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int64_t r = row0 + 4 * k + rr;
          cv[k] = r < m && j < ncols && j <= r ? C[r * ldc + j] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int64_t r = row0 + 4 * k + rr;
          if (r < m && j < ncols && j <= r) C[r * ldc + j] = cv[k] - tr[(4 * k + rr) * kOzTurnLd + cc];
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*fail && threadIdx.x == 0 && status) atomicExch(status, QGX_ERR_TIMEOUT);
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kOzTmemCols) : "memory");
  }
}

struct CholWs {
  uint8_t* s_panel[2];        // digits of a trailing panel's 256 columns (two panels in flight)
  int* e_panel[2];            // n row exponents each
  uint8_t* s_block;           // digits of the 64 columns below a diagonal block
  int* e_block;               // n row exponents
  BlockFactor* factor;        // the current diagonal block's
  ChainState* chain;
  RowBound bound;             // n row bounds
};

int64_t chol_layout(int64_t n, void* base, CholWs* ws) {
  int64_t off = 0;
  auto take = [&](int64_t b) {
    const int64_t o = off;
    off += al256(b);
    return o;
  };
  const int64_t nr = slice_rows(n);
  const int64_t o_sp0 = take(kSlices * nr * kPanel * 2), o_sp1 = take(kSlices * nr * kPanel * 2);
  const int64_t o_ep0 = take(n * 4), o_ep1 = take(n * 4);
  const int64_t o_sb = take(kSlices * nr * kBlk * 2), o_eb = take(n * 4), o_bf = take(sizeof(BlockFactor));
  const int64_t o_rf = take(n * 4), o_re = take(n * 4), o_cs = take(sizeof(ChainState));
  if (base && ws) {
    char* b = static_cast<char*>(base);
    ws->s_panel[0] = reinterpret_cast<uint8_t*>(b + o_sp0);
    ws->s_panel[1] = reinterpret_cast<uint8_t*>(b + o_sp1);
    ws->e_panel[0] = reinterpret_cast<int*>(b + o_ep0);
    ws->e_panel[1] = reinterpret_cast<int*>(b + o_ep1);
    ws->s_block = reinterpret_cast<uint8_t*>(b + o_sb);
    ws->e_block = reinterpret_cast<int*>(b + o_eb);
    ws->factor = reinterpret_cast<BlockFactor*>(b + o_bf);
    ws->chain = reinterpret_cast<ChainState*>(b + o_cs);
    ws->bound.f = reinterpret_cast<float*>(b + o_rf);
    ws->bound.E = reinterpret_cast<int*>(b + o_re);
  }
  return off;
}

// C -= P P^T on and below the diagonal of the region of rows [r0, r0 + m) x columns
// [r0, r0 + ncols) of A, P the K-column panel sliced into S (slice row r = matrix row s0 + r)
int ozaki_region(double* A, int64_t lda, const uint8_t* S, const int* ex, int64_t s0, int K, int64_t r0, int64_t m,
                 int64_t ncols, int32_t* status, cudaStream_t st, int64_t* kernels) {
  if (m <= 0 || ncols <= 0) return QGX_OK;
  int64_t tiles = 0;  // as oz_tile enumerates them
  const int64_t nr = (m + kOzM - 1) / kOzM, nc = (ncols + kOzN - 1) / kOzN;
  for (int64_t g = 0; g * kOzGroup < nr; ++g) {
    const int64_t rows = std::min<int64_t>(kOzGroup, nr - g * kOzGroup);
    tiles += rows * std::min<int64_t>(nc, 2 * (g * kOzGroup + rows));
  }
  // several tiles per CTA hide the next tile's first loads behind the epilogue; fewer where the
  // tiles would not fill the SMs four times over
  const int64_t sms = device_sm_count();
  const int per_cta = tiles >= 16 * sms ? 4 : tiles >= 4 * sms ? 2 : 1;
  if (m > 0x7fffffffLL || tiles > 0x7fffffffLL) return QGX_ERR_UNSUPPORTED;
  QGX_CHECK_CUDA(cudaFuncSetAttribute(ozaki_syrk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOzSmem));
  ozaki_syrk_kernel<<<(unsigned)((tiles + per_cta - 1) / per_cta), kOzThreads, kOzSmem, st>>>(
      S, ex, K / kOzKB, (int)(r0 - s0), m, ncols, A + r0 * lda + r0, lda, tiles, per_cta, status);
  ++*kernels;
  return launch_status();
}

// Per device: the look-ahead stream (highest priority) and the events that order it against the
// caller's stream. One factorisation at a time per device (the mutex is held while enqueueing).
struct LookAhead {
  std::mutex mu;
  cudaStream_t aux = nullptr;
  cudaEvent_t start = nullptr, end = nullptr, strip_done[2] = {}, rest_done[2] = {};
};
constexpr int kMaxCholDevices = 64;
LookAhead g_look[kMaxCholDevices];
std::mutex g_look_init;

int look_ahead_for_current_device(LookAhead** out) {
  int dev = 0;
  QGX_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxCholDevices) return QGX_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_look_init);
  LookAhead& la = g_look[dev];
  if (!la.aux) {
    int lo = 0, hi = 0;
    QGX_CHECK_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    QGX_CHECK_CUDA(cudaStreamCreateWithPriority(&la.aux, cudaStreamNonBlocking, hi));
    cudaEvent_t* evs[6] = {&la.start, &la.end, &la.strip_done[0], &la.strip_done[1], &la.rest_done[0],
                           &la.rest_done[1]};
    for (cudaEvent_t* e : evs) QGX_CHECK_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  }
  *out = &la;
  return QGX_OK;
}

}  // namespace

int64_t chol_f64_workspace_bytes(int64_t n) { return n > 0 ? chol_layout(n, nullptr, nullptr) : 0; }

// A = L L^T in place (see the file comment). info: 0, or the order of the first leading minor
// that is not positive definite. status (may be NULL): QGX_ERR_TIMEOUT if a wait ran out, a tensor
// core's or the chain's. Adds the number of kernels launched to *kernels.
//
// Look-ahead: panel k's trailing update is split into the next panel's 256 columns (the strip)
// and the rest. The panel chain (diagonal blocks, triangular solves, the in-panel updates), the
// panel's slicing and the strip run on a high-priority internal stream; the rest runs on the
// caller's stream, so the next panel's chain overlaps the large tensor-core update. Panel
// k's chain waits for the rest update of panel k - 2, and panel k's strip for the rest update of
// panel k - 1: every update of a column block is ordered after the previous one (the strip and
// the previous panel's rest both update the next panel's columns below its diagonal). Two slice
// buffers alternate between panels. The caller's stream waits for the internal one at the end,
// so the factor is complete in stream order.
int chol_f64(double* A, int64_t n, int64_t lda, int* info, int32_t* status, void* work, cudaStream_t st,
             int64_t* kernels) {
  if ((reinterpret_cast<uintptr_t>(work) & 255) != 0) return QGX_ERR_ARG;
  LookAhead* la = nullptr;
  int rc = look_ahead_for_current_device(&la);
  if (rc != QGX_OK) return rc;
  std::lock_guard<std::mutex> lock(la->mu);
  CholWs ws;
  chol_layout(n, work, &ws);
  cudaStream_t aux = la->aux;
  QGX_CHECK_CUDA(cudaMemsetAsync(info, 0, sizeof(int), st));
  if (status) QGX_CHECK_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), st));
  QGX_CHECK_CUDA(cudaEventRecord(la->start, st));
  QGX_CHECK_CUDA(cudaStreamWaitEvent(aux, la->start, 0));
  QGX_CHECK_CUDA(cudaFuncSetAttribute(chain_block_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(ChainShared<1>)));
  QGX_CHECK_CUDA(cudaFuncSetAttribute(chain_block_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(ChainShared<2>)));
  QGX_CHECK_CUDA(cudaFuncSetAttribute(trsm_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(TrsmShared<1>)));
  int* score = ws.e_panel[1];  // free until the second panel is sliced
  diag_bound_kernel<<<(unsigned)((n + 255) / 256), 256, 0, aux>>>(A, lda, n, ws.bound, ws.chain, score, info);
  // column tiles per CTA: one where that leaves SMs idle, else up to eight, whose loads overlap
  const int64_t scans = (n + kWeakTile - 1) / kWeakTile, sms = device_sm_count();
  const int scan_per = (int)std::max<int64_t>(1, std::min<int64_t>(8, scans * (scans + 1) / 2 / (4 * sms)));
  if (scans > 65535) return QGX_ERR_UNSUPPORTED;
  weak_coupling_kernel<<<dim3((unsigned)((scans + scan_per - 1) / scan_per), (unsigned)scans), kWeakThreads, 0, aux>>>(
      A, lda, n, ws.bound, scan_per, score);
  choose_panel_kernel<<<1, kChooseThreads, 0, aux>>>(score, n, ws.chain);
  *kernels += 3;
  int64_t k = 0;
  unsigned tickets = 0;  // drawn by the launches so far
  for (int64_t c0 = 0; c0 < n; c0 += kPanel, ++k) {
    const int64_t pe = std::min<int64_t>(c0 + kPanel, n);
    if (k >= 2) QGX_CHECK_CUDA(cudaStreamWaitEvent(aux, la->rest_done[k & 1], 0));
    // the panel chain
    for (int64_t cj = c0; cj < pe; cj += kBlk) {
      const int nb = (int)std::min<int64_t>(kBlk, n - cj);
      const int64_t rb = cj + kBlk;  // first row below the block
      const int64_t rows = std::max<int64_t>(0, n - rb);
      const int groups0 = (int)(cj / kBlk) * (kBlk / 4);
      uint8_t* S = rb < pe ? ws.s_block : nullptr;
      // the rows' tiles of 32 per CTA where the factorisation and the solve share a launch; 0: they do
      // not. One on up to half of the SMs, two on up to three quarters (n = 8192: 10.5 ms; 10.6 with one
      // on all SMs, 11.5 without), so that the trailing update keeps some (n = 16384: 50.9 ms; 51.2 with
      // two on all SMs, 52.8 with sharing at any size, 51.4 without).
      const int64_t tiles = (rows + kTileRows - 1) / kTileRows;
      const int per_cta = rows == 0 ? 0 : 2 * tiles < sms ? 1 : 2 * tiles < 3 * sms ? 2 : 0;
      if (per_cta > 0) {
        const unsigned grid = 1 + (unsigned)((tiles + per_cta - 1) / per_cta);
        if (per_cta == 1)
          chain_block_kernel<1><<<grid, chain_threads(1), sizeof(ChainShared<1>), aux>>>(
              A, lda, cj, nb, n, ws.bound, ws.factor, S, ws.e_block, ws.chain, groups0, tickets, info, status);
        else
          chain_block_kernel<2><<<grid, chain_threads(2), sizeof(ChainShared<2>), aux>>>(
              A, lda, cj, nb, n, ws.bound, ws.factor, S, ws.e_block, ws.chain, groups0, tickets, info, status);
        tickets += grid;
        ++*kernels;
      } else {
        potrf_block_kernel<<<1, kPotrfThreads, 0, aux>>>(A, lda, cj, nb, ws.bound, ws.factor, ws.chain, groups0, info);
        ++*kernels;
        if (rb >= n) break;
        trsm_block_kernel<<<(unsigned)tiles, 32 * kTileWarps, sizeof(TrsmShared<1>), aux>>>(
            A, lda, cj, n, ws.bound, ws.factor, ws.chain, S, ws.e_block, info);
        ++*kernels;
      }
      if ((rc = launch_status()) != QGX_OK) return rc;
      // the block's columns update the rest of the panel (K = 64)
      if (rb < pe && (rc = ozaki_region(A, lda, ws.s_block, ws.e_block, rb, kBlk, rb, n - rb, pe - rb, status, aux,
                                        kernels)) != QGX_OK)
        return rc;
    }
    if (pe >= n) break;
    // the panel's trailing update (K = 256): the strip on the internal stream, the rest on st
    const int b = (int)(k & 1);
    const int64_t ms = n - pe, pe2 = std::min<int64_t>(pe + kPanel, n);
    slice_rows_kernel<<<(unsigned)((ms + 7) / 8), 256, 0, aux>>>(A, lda, pe, c0, ms, ws.s_panel[b], ws.e_panel[b],
                                                                ws.bound);
    ++*kernels;
    if ((rc = launch_status()) != QGX_OK) return rc;
    // the strip updates the next panel's columns, which the previous panel's rest update (on st)
    // also updates: both read-modify-write the same entries, so the strip waits for it
    if (k >= 1) QGX_CHECK_CUDA(cudaStreamWaitEvent(aux, la->rest_done[(k - 1) & 1], 0));
    if ((rc = ozaki_region(A, lda, ws.s_panel[b], ws.e_panel[b], pe, kPanel, pe, ms, pe2 - pe, status, aux,
                           kernels)) != QGX_OK)
      return rc;
    if (pe2 < n) {
      QGX_CHECK_CUDA(cudaEventRecord(la->strip_done[b], aux));
      QGX_CHECK_CUDA(cudaStreamWaitEvent(st, la->strip_done[b], 0));
      if ((rc = ozaki_region(A, lda, ws.s_panel[b], ws.e_panel[b], pe, kPanel, pe2, n - pe2, n - pe2, status, st,
                             kernels)) != QGX_OK)
        return rc;
      QGX_CHECK_CUDA(cudaEventRecord(la->rest_done[b], st));
    }
  }
  QGX_CHECK_CUDA(cudaEventRecord(la->end, aux));
  QGX_CHECK_CUDA(cudaStreamWaitEvent(st, la->end, 0));
  return launch_status();
}

// ---- factorisation graphs ------------------------------------------------------------
// A factorisation is a long launch sequence (about 2000 kernels and event operations at
// n = 32768). Enqueued one by one it fills the device's queue of pending launches, after which
// every further launch waits for the GPU: the caller's thread is held for the whole
// factorisation, and callers on other streams (the jobs of a serving loop) cannot get their
// work queued meanwhile. The sequence is therefore captured once per set of buffers into a
// CUDA graph (on a private stream, relaxed capture mode; the look-ahead stream joins the capture
// through its events, which become edges of the graph) and replayed with one launch. Two
// replays share no stream or event, so factorisations on different streams can overlap.
namespace {

struct CholKey {
  double* A;
  int64_t n, lda;
  int* info;
  int32_t* status;
  void* work;
  int device;
  bool operator==(const CholKey& o) const {
    return A == o.A && n == o.n && lda == o.lda && info == o.info && status == o.status && work == o.work &&
           device == o.device;
  }
};

struct CholGraph {
  CholKey key;
  cudaGraphExec_t exec;
  int64_t kernels;
  uint64_t last_use;
};

constexpr int kMaxCholGraphs = 16;
std::mutex g_chol_graph_mutex;
std::vector<CholGraph> g_chol_graphs;
uint64_t g_chol_clock = 0;
cudaStream_t g_chol_capture[kMaxCholDevices] = {};

}  // namespace

int chol_f64_graph(double* A, int64_t n, int64_t lda, int* info, int32_t* status, void* work, cudaStream_t st,
                   int64_t* kernels) {
  int dev = 0;
  QGX_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxCholDevices) return QGX_ERR_UNSUPPORTED;
  const CholKey key{A, n, lda, info, status, work, dev};
  std::lock_guard<std::mutex> lock(g_chol_graph_mutex);
  CholGraph* hit = nullptr;
  for (auto& e : g_chol_graphs)
    if (e.key == key) hit = &e;
  if (!hit) {
    if (!g_chol_capture[dev]) QGX_CHECK_CUDA(cudaStreamCreateWithFlags(&g_chol_capture[dev], cudaStreamNonBlocking));
    cudaStream_t cs = g_chol_capture[dev];
    QGX_CHECK_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeRelaxed));
    int64_t count = 0;
    const int rc = chol_f64(A, n, lda, info, status, work, cs, &count);
    cudaGraph_t graph = nullptr;
    const cudaError_t ce = cudaStreamEndCapture(cs, &graph);
    if (rc != QGX_OK) {
      if (graph) cudaGraphDestroy(graph);
      cudaGetLastError();
      return rc;
    }
    QGX_CHECK_CUDA(ce);
    cudaGraphExec_t exec = nullptr;
    // the look-ahead chain keeps the priority of the stream it was captured from
    const cudaError_t ie = cudaGraphInstantiateWithFlags(&exec, graph, cudaGraphInstantiateFlagUseNodePriority);
    cudaGraphDestroy(graph);
    QGX_CHECK_CUDA(ie);
    if ((int)g_chol_graphs.size() >= kMaxCholGraphs) {  // evict the least recently used (an
      // executable graph still running is freed when it completes)
      auto lru = std::min_element(g_chol_graphs.begin(), g_chol_graphs.end(),
                                  [](const CholGraph& a, const CholGraph& b) { return a.last_use < b.last_use; });
      cudaGraphExecDestroy(lru->exec);
      g_chol_graphs.erase(lru);
    }
    g_chol_graphs.push_back(CholGraph{key, exec, count, 0});
    hit = &g_chol_graphs.back();
  }
  hit->last_use = ++g_chol_clock;
  QGX_CHECK_CUDA(cudaGraphLaunch(hit->exec, st));
  *kernels += hit->kernels;
  return QGX_OK;
}

}  // namespace qgx

using namespace qgx;

extern "C" {

int64_t qgx_cholesky_workspace_bytes(int64_t n) { return chol_f64_workspace_bytes(n); }

int qgx_cholesky(double* A, int64_t n, int64_t lda, int32_t* info, int32_t* status, void* workspace,
                 int64_t workspace_bytes, qgx_stream_t stream) {
  QGX_CHECK_ARG(n > 0 && lda >= n && A && info && workspace);
  QGX_CHECK_ARG(workspace_bytes >= chol_f64_workspace_bytes(n));
  QGX_CHECK_ARG((reinterpret_cast<uintptr_t>(workspace) & 255) == 0);
  int64_t kernels = 0;
  return chol_f64_graph(A, n, lda, info, status, workspace, as_cuda(stream), &kernels);
}

}  // extern "C"
