"""The fixed-point arithmetic of the Cholesky panel (csrc/qgx_fixed.cuh, which compiles for the host
too), run on the CPU: the steps of a diagonal block's columns, as csrc/chol.cu takes them."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "quantax_gb300" / "csrc"

HOST = r"""
#define __host__
#define __device__
#define __align__(n) alignas(n)
#include "qgx_fixed.cuh"
using namespace qgx;

// smallest e with 2^(2e) >= 2 a
static int exponent(double a) {
  int E;
  const double f = frexp(a, &E);
  return ((f == 1.0 ? 1 : 0) + E + 2) >> 1;
}

extern "C" uint64_t pivot(int64_t v) { return fx_pivot(fx_inverse(v, 0)).m; }
extern "C" uint64_t mulhi(uint64_t a, uint64_t b) { return fx_mulhi(a, b); }

// n x n (n <= 64) lower factor of A (row-major, in place); the order of the first failing minor, or 0
extern "C" int factor(double* A, int n) {
  static Fx l[64][64];  // [column][row]
  int e[64], info = 0, kfail = n;
  bool bad[64];
  float squares[64];
  static int64_t s1[64][64], s2[64][64];
  for (int i = 0; i < n; ++i) {
    e[i] = exponent(A[i * n + i]);
    bad[i] = false;
    squares[i] = 0.0f;
  }
  for (int i = 0; i < n; ++i)
    for (int j = 0; j <= i; ++j) {
      s1[i][j] = fx_from_double(A[i * n + j], e[i] + e[j], 62);
      s2[i][j] = 0;
    }
  for (int k = 0; k < n; ++k) {
    const FxInverse inv = fx_inverse(kfail < n || bad[k] ? 0 : s1[k][k], s2[k][k]);
    if (inv.Y == 0 && kfail == n) kfail = k;
    if (kfail < n) {
      info = info ? info : kfail + 1;
      break;
    }
    A[k * n + k] = fx_to_double(fx_sqrt(inv.u, fx_pivot(inv)), e[k] - inv.t - 61);
    for (int i = k + 1; i < n; ++i) {
      const bool in_range = fx_in_range(s1[i][k], inv.t);
      const int64_t X = fx_scale(s1[i][k], s2[i][k], inv, in_range);
      Fx x = fx_split(X);
      const float xv = (float)x.h * 4.656612873077393e-10f;
      const float sq = xv * xv + squares[i];
      bad[i] |= !in_range || !fx_is_entry(X) || sq > 0.52f;
      if (bad[i])
        x = Fx{0, 0};
      else
        squares[i] = sq;
      l[k][i] = x;
      A[i * n + k] = fx_to_double(fx_join(x), e[i] - kFxBits);
    }
    for (int i = k + 1; i < n; ++i)
      for (int j = k + 1; j <= i; ++j) fx_mad(s1[i][j], s2[i][j], Fx{-l[k][i].h, -l[k][i].l}, l[k][j]);
  }
  return info;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    (d / "host.cpp").write_text(HOST)
    gxx = shutil.which("g++")
    assert gxx, "g++ builds the library's host code"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(CSRC), "-o",
                    str(d / "host.so"), str(d / "host.cpp")], check=True)
    lib = C.CDLL(str(d / "host.so"))
    lib.mulhi.restype = C.c_uint64
    lib.mulhi.argtypes = [C.c_uint64, C.c_uint64]
    lib.pivot.restype = C.c_uint64
    lib.pivot.argtypes = [C.c_int64]
    return lib


def factor(host, A):
    A = np.ascontiguousarray(A, dtype=np.float64).copy()
    info = host.factor(A.ctypes.data_as(C.POINTER(C.c_double)), A.shape[0])
    return np.tril(A), info


def test_two_by_two_matrices_are_told_apart(host):
    """|a_10| against sqrt(a_00 a_11) from 1/4 to 5 on diagonals that reach every part of the row scale:
    indefinite matrices fail in their second minor, the others give the factor. (An entry whose scaled
    value lies between 1 and 3/2 must not come back as a small one of the other sign.)"""
    ratios = [r for r in np.arange(0.25, 5.0, 0.02) if abs(r - 1.0) > 1e-9]
    for d0 in np.exp2(np.arange(0.0, 2.0, 0.12)):
        for d1 in np.exp2(np.arange(-2.0, 2.0, 0.12)):
            for r in ratios:
                for sign in (1.0, -1.0):
                    a = sign * r * np.sqrt(d0 * d1)
                    L, info = factor(host, [[d0, a], [a, d1]])
                    assert info == (2 if r > 1.0 else 0), (d0, d1, a)
                    if r < 1.0:
                        assert abs(L[1, 0] * L[0, 0] - a) <= 2.0 ** -51 * np.sqrt(d0 * d1)
                        assert abs(L[1] @ L[1] - d1) <= 2.0 ** -51 * d1


def test_high_products_at_the_ends_of_their_range(host):
    """fx_mulhi against whole products: at most 2 below the floor for factors up to 2^63, and for one
    below 2^63 with one below 2^63 + 2^32 (the mantissa of an inverse square root may round past 2)."""
    rng = np.random.default_rng(0)
    ends = [0, 1, 2 ** 32 - 1, 2 ** 32, 2 ** 62, 2 ** 63 - 2 ** 32, 2 ** 63 - 1, 2 ** 63]
    some = [int(v) for v in rng.integers(0, 2 ** 63, 2000)]
    past = [2 ** 63 + 1, 2 ** 63 + 2 ** 31, 2 ** 63 + 2 ** 32 - 1]
    pairs = [(a, b) for a in ends + some[:50] for b in ends + some[:50]] + list(zip(some, some[::-1]))
    pairs += [(a, b) for a in ends[:-1] + some for b in past]
    for a, b in pairs:
        exact = a * b >> 64
        for got in (host.mulhi(a, b), host.mulhi(b, a)):
            assert exact - 2 <= got <= exact, (a, b)


def test_every_inverse_square_root_fits_the_products(host):
    """The factors that fx_inverse, fx_sqrt and fx_scale multiply: pivots beside the powers of two and
    over the whole range, whose mantissas m 2^-62 of 1 / sqrt(v) lie in [1, 2] up to the estimate."""
    rng = np.random.default_rng(1)
    ends = [m + d for k in range(4, 62) for m in (2 ** k,) for d in (-1, 0, 1) if 16 <= m + d <= 2 ** 61]
    for v in ends + [int(x) for x in np.exp2(rng.uniform(4, 61, 4000))]:
        m = host.pivot(v)
        assert 2 ** 62 - 2 ** 8 <= m < 2 ** 63 + 2 ** 32, v
