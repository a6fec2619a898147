"""Fixed-point arithmetic of the tridiagonalisation (tridiag_fixed.cuh) on the host, no GPU.

The header's functions compile for the host; here they are held against exact integers and, put
together to a Householder reduction, against LAPACK's eigenvalues.  Bounds: a product is off by its
rounding (half a unit) and by what the cut low limbs drop (below a unit in all); the square root and
the reciprocal are Newton steps to 2^-60, the few units of their last multiplications included.
"""
import ctypes
import math
import random
import shutil
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA_INCLUDE = Path("/usr/local/cuda/include")
FA, FV = 60, 58

HARNESS = r"""
#include "tridiag_fixed.cuh"
#include <vector>
using namespace tb::trifx;
typedef long long i64;
typedef unsigned long long u64;
extern "C" {
i64 t_fixed(double x, int q) {
  u64 b;
  __builtin_memcpy(&b, &x, 8);
  return to_fixed(b, q);
}
u64 t_sqrt(u64 r) { return isqrt64(r); }
i64 t_rank2(i64 a, i64 vr, i64 wr, i64 vc, i64 wc) {
  return rank2(a, hi31(vr), lo31(vr), hi31(wr), lo31(wr), hi31(vc), lo31(vc), hi31(wc), lo31(wc));
}
i64 t_dot(int n, const i64* a, const i64* b) {
  i64 hh = 0, cr = 0, sum = 0;
  for (int k = 0; k < n; ++k) {
    mac(hi31(a[k]), lo31(a[k]), hi31(b[k]), lo31(b[k]), hh, cr);
    if (k % 15 == 14 || k == n - 1) {
      sum += fold<4>(hh, cr);
      hh = cr = 0;
    }
  }
  return sum;
}
// out: none, shift, v0, g, gk; returns s
u64 t_reflector(u64 lo, u64 hi, i64 alpha, i64* out) {
  const Reflector f = reflector(lo, hi, alpha);
  const Scalars sc = scalars(f, alpha);
  out[0] = f.none;
  out[1] = f.shift;
  out[2] = f.v0;
  out[3] = sc.g;
  out[4] = sc.gk;
  return f.s;
}
// T of the symmetric A (n x n) with |A|_inf < 2^top
void t_reduce(int n, const double* A, int top, double* d, double* e) {
  const int q = FA - top;
  const double isc = pow2(-q);
  std::vector<i64> a((size_t)n * n), v(n), u(n), w(n);
  for (size_t t = 0; t < a.size(); ++t) a[t] = t_fixed(A[t], q);
  for (int j = 0; j < n - 1; ++j) {
    unsigned __int128 s2 = 0;
    for (int r = j + 1; r < n; ++r) {
      const i64 x = a[r + (size_t)j * n];
      s2 += (unsigned __int128)((__int128)x * x);
    }
    const i64 alpha = a[j + 1 + (size_t)j * n];
    const Reflector f = reflector((u64)s2, (u64)(s2 >> 64), alpha);
    const Scalars sc = scalars(f, alpha);
    d[j] = (double)a[j + (size_t)j * n] * isc;
    if (f.none) {
      e[j] = (double)alpha * isc;
      continue;
    }
    e[j] = (alpha < 0 ? 1.0 : -1.0) * ((double)f.s * 0x1p-64) * pow2(FV - f.shift) * isc;
    for (int r = j + 1; r < n; ++r)
      v[r] = r == j + 1 ? f.v0 : shifted(a[r + (size_t)j * n], f.shift);
    i64 kappa = 0;
    for (int r = j + 1; r < n; ++r) {
      u[r] = t_dot(n - j - 1, &a[j + 1 + (size_t)r * n], &v[j + 1]);
      kappa += kappa_term(u[r], v[r]);
    }
    const i64 K = k_of(kappa, sc.gk);
    for (int r = j + 1; r < n; ++r) w[r] = w_of(p_of(u[r], sc.g), K, v[r]);
    for (int c = j + 1; c < n; ++c)
      for (int r = j + 1; r < n; ++r)
        a[r + (size_t)c * n] = t_rank2(a[r + (size_t)c * n], v[r], w[r], v[c], w[c]);
  }
  d[n - 1] = (double)a[(size_t)n * n - 1] * isc;
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    d = tmp_path_factory.mktemp("trifx")
    (d / "harness.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CUDA_INCLUDE}",
                    f"-I{ROOT / 'tblite_gb300' / 'csrc'}", str(d / "harness.cpp"), "-o",
                    str(d / "harness.so")], check=True)
    so = ctypes.CDLL(str(d / "harness.so"))
    i64, u64, p = ctypes.c_longlong, ctypes.c_ulonglong, ctypes.c_void_p
    for name, res, args in (("t_fixed", i64, [ctypes.c_double, ctypes.c_int]),
                            ("t_sqrt", u64, [u64]), ("t_rank2", i64, [i64] * 5),
                            ("t_dot", i64, [ctypes.c_int, p, p]),
                            ("t_reflector", u64, [u64, u64, i64, p]),
                            ("t_reduce", None, [ctypes.c_int, p, ctypes.c_int, p, p])):
        f = getattr(so, name)
        f.restype, f.argtypes = res, args
    return so


def _nearest(x):
    """Half away from zero."""
    return int(math.copysign(math.floor(abs(x) + Fraction(1, 2)), x))


def test_to_fixed(lib):
    rng = random.Random(1)
    values = [0.0, -0.0, 1.0, -1.0, 0.5, 1.5 * 2.0 ** -61, 2.0 ** -61, -2.0 ** -61, 5e-324,
              -2.2e-308, 1.0 - 2.0 ** -53]
    values += [rng.uniform(-1, 1) * 2.0 ** rng.randint(-80, 0) for _ in range(2000)]
    for x in values:
        assert lib.t_fixed(x, FA) == _nearest(Fraction(x) * 2 ** FA), x
    for top in (-900, -300, 40, 900):  # the same digits at any scale
        for x in values[10:200]:
            y = math.ldexp(x, top)
            if abs(y) > 2.3e-308:
                assert lib.t_fixed(y, FA - top) == _nearest(Fraction(x) * 2 ** FA)


def test_square_root(lib):
    rng = random.Random(2)
    rs = [1 << 62, (1 << 62) + 1, (1 << 63) - 1, 1 << 63, (1 << 64) - 1]
    rs += [rng.randrange(1 << 62, 1 << 64) for _ in range(5000)]
    for r in rs:
        assert abs(lib.t_sqrt(r) - min(math.isqrt(r << 64), (1 << 64) - 1)) <= 16, r


def test_products(lib):
    rng = random.Random(3)
    lim_v, lim_w = (1 << FV) - 1, (1 << FA) - 1
    ends = [(lim_v, lim_w), (-lim_v, lim_w), (lim_v, -lim_w), (-lim_v, -lim_w), (0, 0), (1, -1)]
    cases = [(0, *x, *y) for x in ends for y in ends]
    cases += [(rng.randint(-lim_w, lim_w), rng.randint(-lim_v, lim_v), rng.randint(-lim_w, lim_w),
               rng.randint(-lim_v, lim_v), rng.randint(-lim_w, lim_w)) for _ in range(5000)]
    for a, vr, wr, vc, wc in cases:
        exact = a - Fraction(vr * wc + wr * vc, 1 << FV)
        assert abs(lib.t_rank2(a, vr, wr, vc, wc) - exact) <= 1
        # symmetric in (r, c)
        assert lib.t_rank2(a, vr, wr, vc, wc) == lib.t_rank2(a, vc, wc, vr, wr)
    for n in (1, 14, 15, 16, 31, 200):
        a = [rng.randint(-lim_w, lim_w) // n for _ in range(n)]
        b = [rng.randint(-lim_v, lim_v) for _ in range(n)]
        exact = Fraction(sum(x * y for x, y in zip(a, b)), 1 << FV)
        got = lib.t_dot(n, (ctypes.c_longlong * n)(*a), (ctypes.c_longlong * n)(*b))
        assert abs(got - exact) <= 1 + n / 15


def _reflector(lib, x):
    s2 = sum(t * t for t in x)
    out = (ctypes.c_longlong * 5)()
    s = lib.t_reflector(s2 & (2 ** 64 - 1), s2 >> 64, x[0], out)
    return s, list(out)


def test_reflectors(lib):
    rng = random.Random(4)
    vectors = []
    for _ in range(2000):
        scale = 2 ** rng.randint(3, 59)
        vectors.append([rng.randint(-scale, scale) for _ in range(rng.randint(2, 6))])
    vectors += [[0, 5], [0, -(1 << 59)], [1 << 59, 1], [-(1 << 59), 1], [1, 1], [-1, 1],
                [(1 << 59) - 1, (1 << 59) - 1], [3, 0, 0, 1 << 58]]
    for x in vectors:
        if not any(x[1:]):
            continue
        s, (none, shift, v0, g, gk) = _reflector(lib, x)
        assert not none
        norm = math.isqrt(sum(t * t for t in x) << 128)  # |x| 2^64
        unit = Fraction(norm, 1 << 64) * Fraction(2) ** (shift - FV)  # |x| in [1/2, 1)
        assert Fraction(1, 2) <= unit < 1
        assert abs(Fraction(s, 1 << 64) - unit) <= Fraction(1, 1 << 59)
        alpha = abs(x[0]) * Fraction(2) ** (shift - FV)
        assert (v0 < 0) == (x[0] < 0)
        assert abs(Fraction(abs(v0), 1 << FV) - (alpha + unit)) <= Fraction(4, 1 << FV)
        h = unit * (unit + alpha)
        # dg = g^2 dh, g <= 4, and h to a few units of 2^-60 from s and alpha
        assert abs(Fraction(g, 1 << FA) - 1 / h) <= 64 * Fraction(1, 1 << 58)
        assert abs(Fraction(gk, 1 << 58) - 1 / (2 * h * h)) <= 256 * Fraction(1, 1 << 58)
    for alpha in (0, 7, -7, 1 << 59, -(1 << 59)):  # nothing to reflect
        s, (none, _, _, g, gk) = _reflector(lib, [alpha, 0, 0])
        assert none and g == 0 and gk == 0


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -200, 2.0 ** 300])
@pytest.mark.parametrize("kind", ["random", "diagonal", "tridiagonal", "zero columns", "rank one",
                                  "graded"])
def test_reduction(lib, kind, scale):
    n = 40
    rng = np.random.default_rng(5)
    a = rng.standard_normal((n, n))
    a = a + a.T
    if kind == "diagonal":
        a = np.diag(np.diag(a))
    elif kind == "tridiagonal":
        a = np.triu(np.tril(a, 1), -1)
    elif kind == "zero columns":
        a[::3] = 0.0
        a[:, ::3] = 0.0
    elif kind == "rank one":
        v = rng.standard_normal(n)
        a = np.outer(v, v)
    elif kind == "graded":
        g = 10.0 ** -np.linspace(0, 9, n)
        a = a * g[:, None] * g
    a = a * scale
    norm = np.abs(a).sum(0).max()
    top = math.frexp(norm)[1]
    d, e = np.zeros(n), np.zeros(n)
    a = np.ascontiguousarray(a)
    lib.t_reduce(n, a.ctypes.data, top, d.ctypes.data, e.ctypes.data)
    t = np.diag(d) + np.diag(e[:-1], 1) + np.diag(e[:-1], -1)
    got = np.linalg.eigvalsh(t / scale)
    ref = np.linalg.eigvalsh(a / scale)
    # LAPACK's own error, a few units of 2^-53 |A|; the reduction's is n 2^-59
    assert np.max(np.abs(got - ref)) <= 16 * 2.0 ** -53 * norm / scale
