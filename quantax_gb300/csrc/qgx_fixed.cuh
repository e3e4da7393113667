// Fixed-point arithmetic of the FP64 Cholesky's panel (chol.cu): FP64-class products on the
// integer pipe.
//
// An FP64 instruction occupies a GB300 SM sub-core's FP64 pipe for 64 clocks per warp whatever
// the number of active lanes (measured: 1.67 FMA per clock per SM), a 32 x 32 -> 64 bit
// multiply-add with 64-bit accumulation for five (measured: 25 per clock per SM). A Cholesky
// factor's rows are bounded a priori, |L_rk| <= sqrt(a_rr), so with a power of two
// 2^e_r >= sqrt(2 a_rr) per row every quantity of the factorisation is a fixed-point number of
// known range:
//   x  = L_rk 2^-e_r, sum_k x^2 <= 1/2, held as h 2^-31 + l 2^-60 (|l| <= 2^28), and
//   v  = C_rk 2^-(e_r + e_k), |v| <= 1/2, held as s1 2^-62 + s2 2^-91,
// and v -= x y takes three multiply-adds: s1 -= xh yh, s2 -= xh yl, s2 -= xl yh (the dropped
// xl yl is below 2^-64; over 64 columns the sums stay below 2^63 by Cauchy-Schwarz). Against
// FP64, whose roundings are relative to each value: x is kept to 2^-61 of 2^e_r <= 2.9
// sqrt(a_rr), the FP64 spacing of an entry of 2^-7 sqrt(a_rr), which is the typical size in a
// row of 16384 columns. Entries far below that are held in fewer bits than FP64 has, so matrices with
// many of them are not factored this way (chol.cu, weak_coupling_kernel).
#pragma once

#include <stdint.h>

#include <cmath>
#include <cstring>

namespace qgx {
namespace {

constexpr int kFxBits = 60;  // fraction bits of x

struct Fx {  // h 2^-31 + l 2^-60
  int h, l;
};

__host__ __device__ inline int clz64(uint64_t v) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}

__host__ __device__ inline uint64_t dbl_bits(double a) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(a);
#else
  uint64_t b;
  memcpy(&b, &a, 8);
  return b;
#endif
}

__host__ __device__ inline double bits_dbl(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double a;
  memcpy(&a, &b, 8);
  return a;
#endif
}

__host__ __device__ inline bool dbl_finite(double a) { return ((dbl_bits(a) >> 52) & 0x7FF) != 0x7FF; }

// a 2^(bits - E) rounded to the nearest integer, saturating at +-2^62; a not finite gives 0
__host__ __device__ inline int64_t fx_from_double(double a, int E, int bits) {
  const uint64_t b = dbl_bits(a);
  const int ex = (int)((b >> 52) & 0x7FF);
  const uint64_t frac = b & 0xFFFFFFFFFFFFFULL;
  if (ex == 0x7FF) return 0;
  const uint64_t mant = ex ? frac | (1ULL << 52) : frac;
  const int p = (ex ? ex : 1) - 1075 - E + bits;  // the value is mant 2^p
  int64_t v;
  if (p >= 0) {
    v = mant == 0 ? 0 : p > 9 && p > clz64(mant) - 2 ? (int64_t)(1LL << 62) : (int64_t)(mant << p);
  } else {
    const int s = p < -55 ? 55 : -p;
    v = (int64_t)((mant + (1ULL << (s - 1))) >> s);
  }
  return (b >> 63) ? -v : v;
}

// v 2^p rounded to the nearest double, on the integer pipe
__host__ __device__ inline double fx_to_double(int64_t v, int p) {
  if (v == 0) return 0.0;
  const uint64_t a = v < 0 ? 0ULL - (uint64_t)v : (uint64_t)v;
  const int lz = clz64(a);
  const uint64_t n = a << lz, r = n + 0x400;
  const bool carry = r < n;  // rounded up to the next power of two
  const int ex = 63 - lz + p + 1023 + (carry ? 1 : 0);
  if (ex < 1 || ex > 2046) return ldexp((double)v, p);
  const uint64_t frac = carry ? 0 : (r >> 11) & 0xFFFFFFFFFFFFFULL;
  return bits_dbl(((uint64_t)(v < 0) << 63) | ((uint64_t)ex << 52) | frac);
}

// s += a b
__host__ __device__ inline void mad_wide(int64_t& s, int a, int b) {
#ifdef __CUDA_ARCH__
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s) : "r"(a), "r"(b));
#else
  s += (int64_t)a * b;
#endif
}

// v -= x y; the caller passes x negated
__host__ __device__ inline void fx_mad(int64_t& s1, int64_t& s2, const Fx& nx, const Fx& y) {
  mad_wide(s1, nx.h, y.h);
  mad_wide(s2, nx.h, y.l);
  mad_wide(s2, nx.l, y.h);
}

// (s1 2^-62 + s2 2^-91) 2^t in units of 2^-62, 0 <= t <= 29; modulo 2^64, exact whenever the
// result fits
__host__ __device__ inline int64_t fx_combine(int64_t s1, int64_t s2, int t) {
  return (int64_t)(((uint64_t)s1 << t) + (uint64_t)(s2 >> (29 - t)));
}

// floor of a b / 2^64 up to 2 units below, a and b at most 2^63, or a < 2^63 and b < 2^63 + 2^32: the two
// cross products have to stay below 2^64 together
__host__ __device__ inline uint64_t fx_mulhi(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  const uint64_t mid = (uint64_t)ah * bl + (uint64_t)al * bh;
  return (uint64_t)ah * bh + (mid >> 32);
}

// a row's value split for fx_mad: X in units of 2^-60
__host__ __device__ inline Fx fx_split(int64_t X) {
  Fx r;
  r.h = (int)((X + (1LL << 28)) >> 29);
  r.l = (int)(X - ((int64_t)r.h << 29));
  return r;
}
__host__ __device__ inline int64_t fx_join(const Fx& x) { return ((int64_t)x.h << 29) + x.l; }

// Inverse square root of a pivot v, 2^-58 <= v <= 1/2 (below that the pivot counts as not
// positive: it is noise of its row): 1 / sqrt(v) = Y 2^-23 (1 + c 2^-60) 2^t from a float estimate
// Y 2^-23 in [1, 2] for the normalised pivot u in [1/4, 1) and one third-order step
// c = h/2 + 3 h^2/8 with h = 1 - u y0^2 (|h| < 2^-20.5; error 5 h^3 / 16).
struct FxInverse {
  uint32_t Y;  // 0: the pivot is not positive
  int t;
  int64_t c;
  uint64_t u;  // units of 2^-62
};
__host__ __device__ inline FxInverse fx_inverse(int64_t s1, int64_t s2) {
  const int64_t v0 = fx_combine(s1, s2, 0);
  const bool pos = v0 >= 16;
  const int t2 = (clz64((uint64_t)(pos ? v0 : 1LL << 60)) - 2) & ~1;
  FxInverse r;
  r.u = (uint64_t)(pos ? v0 : 1LL << 60) << t2;  // in [2^60, 2^62)
  const float f = (float)(uint32_t)(r.u >> 32);  // 2^30 u; its inverse root's bits less those of
  uint32_t Y;                                    // 2^-16 are y0 2^23
#ifdef __CUDA_ARCH__
  float y0;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(f));
  Y = (uint32_t)__float_as_int(y0) - 0x37800000u;
#else
  const float y0 = 1.0f / std::sqrt(f);
  memcpy(&Y, &y0, 4);
  Y -= 0x37800000u;
#endif
  const int64_t h = (1LL << 60) - (int64_t)fx_mulhi(r.u << 1, ((uint64_t)Y * Y) << 15);  // 2^-60
  const int hh = (int)(h >> 11);                                                         // 2^-49
  r.c = (h >> 1) + (((int64_t)(3 * hh) * hh) >> 41);
  r.Y = pos ? Y : 0;
  r.t = t2 >> 1;
  return r;
}

// the same as one factor: 1 / sqrt(v) = m 2^-62 2^t
struct FxPivot {
  uint64_t m;  // 0: the pivot is not positive
  int t;
};
__host__ __device__ inline FxPivot fx_pivot(const FxInverse& p) {
  FxPivot r;
  r.m = ((uint64_t)p.Y << 39) + (uint64_t)((p.c * (int64_t)p.Y) >> 21);
  r.t = p.t;
  return r;
}

// sqrt(v) of the pivot in units of 2^-(61 + t)
__host__ __device__ inline int64_t fx_sqrt(uint64_t u, const FxPivot& p) { return (int64_t)fx_mulhi(u << 1, p.m); }

// whether |v| 2^t is below 3/4, so that fx_scale's products fit: every row of a positive definite
// matrix passes (|x| <= sqrt(1/2) and the mantissa of 1 / sqrt(v) is at least 1), but so do others, whose
// x reaches 1.5: fx_is_entry looks at the scaled value
__host__ __device__ inline bool fx_in_range(int64_t s1, int t) {
  const int top = (int)(s1 >> 32);
  return (top < 0 ? -top : top) <= ((3 << 28) >> t);
}

// whether X, in units of 2^-60, is below 3/4 (up to 2^-28): every entry of a positive definite matrix's
// factor is, and fx_split holds it (its high part has 32 bits: |x| < 1)
__host__ __device__ inline bool fx_is_entry(int64_t X) {
  const int top = (int)(X >> 32);
  return (top < 0 ? -top : top) <= (3 << 26);
}

// x = v 2^t m 2^-62 in units of 2^-60 (0 unless in range)
__host__ __device__ inline int64_t fx_scale(int64_t s1, int64_t s2, const FxPivot& piv, bool in_range) {
  const int64_t w = fx_combine(s1, s2, piv.t);
  const uint64_t a = in_range ? (w < 0 ? 0ULL - (uint64_t)w : (uint64_t)w) : 0;
  const int64_t X = (int64_t)((fx_mulhi(a << 1, piv.m) + 1) >> 1);
  return w < 0 ? -X : X;
}

// the same from the inverse's parts: v y0 does not wait for c, so the chain from a pivot to its
// column is the shorter by one multiplication
__host__ __device__ inline int64_t fx_scale(int64_t s1, int64_t s2, const FxInverse& inv, bool in_range) {
  const int64_t w = fx_combine(s1, s2, inv.t);
  const uint64_t a = in_range ? (w < 0 ? 0ULL - (uint64_t)w : (uint64_t)w) : 0;
  const uint64_t T = fx_mulhi(a << 1, (uint64_t)inv.Y << 39);  // 2^-61, below 2^62
  const uint64_t c = (uint64_t)(inv.c < 0 ? -inv.c : inv.c) << 23;  // 2^-83, below 2^63
  const uint64_t d = fx_mulhi(T << 1, c) >> 20;  // (2^-62 2^-83 2^64) 2^20: 2^-61
  const int64_t X = (int64_t)((inv.c < 0 ? T - d : T + d) + 1) >> 1;
  return w < 0 ? -X : X;
}

}  // namespace
}  // namespace qgx
