// Householder tridiagonalisation of a symmetric matrix in 64-bit fixed point.
//
// What bounds it: the reduction costs n^3 multiply-adds (full storage: two per element for the
// rank-2 update, one for the matrix-vector product) and a chain of n dependent steps.  This GPU
// issues an FP64 instruction of a warp once in 64-76 cycles per scheduler (measured; 1.7 FMA per
// clock and SM, 580 cycles for a warp sum, 384 for a division, 727 for a square root), but a
// 32 x 32 + 64 bit integer multiply-add once in 2.5.  So the matrix lives in shared memory as
// 64-bit integers: an element update and its term of the next product are 12 wide integer
// multiply-adds and a dozen additions and shifts (~46 cycles per warp against 228 on the FP64
// pipe), and the sums along the chain are integer sums.
//
// Accuracy: integers in units of 2^-60 of a power of two above |A|_inf.  An orthogonal
// similarity keeps every element below |A|_2, so nothing overflows, and the rounding of a step
// is 2^-60 |A| absolute, below the 2^-53 |A| of an FP64 reduction.  The reflectors are exact
// integers normalised to a 2-norm in [1/2, 1); square sums are exact (128 bits).
//
// One barrier per column.  The columns are dealt round-robin to the nb CTAs; the reflector of
// the next column, K and w are computed by every CTA for itself from two published vectors: the
// product u = A v (each CTA's own entries) and the next pivot column before its last update
// (from its owner).  The update of the owned columns with (v, w) and their products with the next
// reflector are then one pass over shared memory.
//
// With x = A(i+2:n, i+1) after the update, s = |x|, alpha = x_0: v = x + sign(alpha) s e_0,
// h = s (s + |alpha|) = v.v / 2, H = I - v v^T / h, u = A v, K = v.u / (2 h^2),
// w = u / h - K v, A <- A - v w^T - w v^T.  LAPACK's form (v_0 = 1) has tau = v_0^2 / h.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace tb {
namespace trifx {

constexpr int FA = 60;  // fractional bits of A, u = A v, K, 1/h and w
constexpr int FV = 58;  // fractional bits of the reflectors

// 64-bit value x = h 2^31 + l, 0 <= l < 2^31: both limbs enter signed wide multiply-adds
__host__ __device__ __forceinline__ int hi31(long long x) { return (int)(x >> 31); }
__host__ __device__ __forceinline__ int lo31(long long x) { return (int)(x & 0x7FFFFFFF); }
__host__ __device__ __forceinline__ long long join31(int h, int l) {
  return ((long long)h << 31) + l;
}
__host__ __device__ __forceinline__ long long mw(int a, int b, long long c) {
  return (long long)a * b + c;
}
// high 64 bits of a signed / an unsigned 64 x 64 bit product
__host__ __device__ __forceinline__ long long mulhi(long long a, long long b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return (long long)(((__int128)a * b) >> 64);
#endif
}
__host__ __device__ __forceinline__ unsigned long long umulhi(unsigned long long a,
                                                              unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
#endif
}
__host__ __device__ __forceinline__ int clz64(unsigned long long x) {  // x != 0
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}

// sum over the limb products of two factors: the value is hh 2^62 + cr 2^31 in the product's
// unit; the low x low product enters cr through the top bits of both (error 2^-15 of a unit of
// hh 2^-31).  a's low limb loses 15 bits, b's 16.
__host__ __device__ __forceinline__ void mac(int ah, int al, int bh, int bl, long long& hh,
                                             long long& cr) {
  hh = mw(ah, bh, hh);
  cr = mw(ah, bl, cr);
  cr = mw(al, bh, cr);
  cr = mw(al >> 15, bl >> 16, cr);
}
// (hh 2^62 + cr 2^31) / 2^(62 - sh), rounded
template <int SH>
__host__ __device__ __forceinline__ long long fold(long long hh, long long cr) {
  return (hh << SH) + ((cr + (1LL << (30 - SH))) >> (31 - SH));
}
// a - (v_r w_c + w_r v_c); symmetric in (r, c)
__host__ __device__ __forceinline__ long long rank2(long long a, int vrh, int vrl, int wrh,
                                                    int wrl, int vch, int vcl, int wch, int wcl) {
  // two sums of the cross terms: half the dependent chain
  const long long c0 = mw(wcl >> 15, vrl >> 16, mw(wcl, vrh, (long long)wch * vrl));
  const long long c1 = mw(wrl >> 15, vcl >> 16, mw(wrl, vch, (long long)wrh * vcl));
  return a - fold<4>(mw(wrh, vch, (long long)wch * vrh), c0 + c1);
}

// double -> integer units of 2^-q (round to nearest, ties away): |x| 2^q < 2^62; the FP64 pipe
// is not touched
__host__ __device__ __forceinline__ long long to_fixed(unsigned long long bits, int q) {
  const int ex = (int)((bits >> 52) & 0x7FF);
  if (ex == 0) return 0;  // zero and subnormals
  const unsigned long long m = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int sh = ex - 1075 + q;
  long long v;
  if (sh >= 0) v = (long long)(m << (sh > 10 ? 10 : sh));
  else if (sh > -64) v = (long long)(((m >> (-sh - 1)) + 1) >> 1);
  else v = 0;
  return (bits >> 63) ? -v : v;
}
// 2^k as a double (normal range)
__host__ __device__ __forceinline__ double pow2(int k) {
  const unsigned long long b = (unsigned long long)(k + 1023) << 52;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double d;
  __builtin_memcpy(&d, &b, 8);
  return d;
#endif
}

// sqrt of R 2^-64 in [1/4, 1), in units of 2^-64: float seed, two Newton steps
// s <- s + (R - s^2) y / 2 with y ~ 1/s (relative error of the seed 2^-22, then 2^-44, 2^-60)
__host__ __device__ __forceinline__ unsigned long long isqrt64(unsigned long long R) {
  const float f = (float)(unsigned)(R >> 40) * 0x1p-24f;
#ifdef __CUDA_ARCH__
  const float y = rsqrtf(f);
#else
  const float y = 1.0f / __builtin_sqrtf(f);
#endif
  const float yc = y < 1.9999999f ? y : 1.9999999f;
  const long long Y = (long long)(unsigned)(yc * 0x1p30f) << 32;  // units of 2^-62, < 2^63
  const unsigned long long s62 = umulhi(R, (unsigned long long)Y);
  unsigned long long s = s62 >= (1ull << 62) ? ~0ull : s62 << 2;
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const long long r = (long long)(R - umulhi(s, s));
    const long long d = mulhi(r, Y) * 2;
    const unsigned long long t = s + (unsigned long long)d;
    // s stays below 1: a correction that passes 2^64 saturates
    s = (d > 0 && t < s) ? ~0ull : t;
  }
  return s;
}

// x 2^shift, rounded
__host__ __device__ __forceinline__ long long shifted(long long x, int shift) {
  return shift >= 0 ? x << shift : (x + (1LL << (-shift - 1))) >> -shift;
}

// the reflector of x from the exact square sum (lo, hi) of all its elements and x_0 = alpha (in
// units of 2^-FA): the shift that takes x to units of 2^-FV with |x| in [1/2, 1), v_0, and s = |x|
// (units of 2^-64 after the shift); nothing to reflect (x_1.. all zero): none
struct Reflector {
  bool none;
  int shift;  // -2 .. : a right shift of up to FA - FV bits rounds
  long long v0;
  unsigned long long s;
};
__host__ __device__ __forceinline__ unsigned long long uabs(long long x) {
  return x < 0 ? 0ull - (unsigned long long)x : (unsigned long long)x;
}
__host__ __device__ __forceinline__ Reflector reflector(unsigned long long lo,
                                                        unsigned long long hi, long long alpha) {
  Reflector f;
  const unsigned long long aa = uabs(alpha);
  // 2^(2t) <= square sum < 2^(2t + 2); normalised R in [2^62, 2^64)
  const int msb = hi ? 127 - clz64(hi) : 63 - clz64(lo | 1);
  const int t = msb >> 1;
  const int up = 126 - 2 * t;  // left shift of the 128-bit sum, even, >= 4
  const unsigned long long R =
      up >= 64 ? lo << (up - 64) : (hi << up) | (lo >> (64 - up));
  f.s = isqrt64(R);
  f.shift = FV - 1 - t;
  const long long mag = shifted((long long)aa, f.shift) + (long long)(f.s >> (64 - FV));
  f.v0 = alpha < 0 ? -mag : mag;
  f.none = lo == aa * aa && hi == umulhi(aa, aa);
  return f;
}
// g = 1/h (units of 2^-FA, at most 4) and gk = g^2 / 2 (units of 2^-58) for the next step, off
// the chain: h = s (s + |alpha|) in [1/4, 2) in units of 2^-63, float seed, two Newton steps
// g <- g + g (1 - h g)
struct Scalars {
  long long g, gk;
};
__host__ __device__ __forceinline__ Scalars scalars(const Reflector& f, long long alpha) {
  Scalars o;
  const unsigned long long sa =
      (f.s >> 1) + ((unsigned long long)shifted((long long)uabs(alpha), f.shift) << 5);
  const unsigned long long h = umulhi(f.s, sa);
  const float hf = (float)(unsigned)(h >> 32) * 0x1p-31f;
#ifdef __CUDA_ARCH__
  const float y = __fdividef(1.0f, hf);
#else
  const float y = 1.0f / hf;
#endif
  unsigned long long g = (unsigned long long)(unsigned)((y < 3.9999998f ? y : 3.9999998f) * 0x1p30f)
                         << 30;
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const long long e = (1LL << 59) - (long long)umulhi(h, g);
    g += (unsigned long long)mulhi((long long)g, e * 32);
  }
  g = g < (1ull << 62) ? g : (1ull << 62);
  o.g = f.none ? 0 : (long long)g;
  o.gk = f.none ? 0 : (long long)(umulhi(g << 1, g << 1) >> 1);
  return o;
}
// K = v.u / (2 h^2): kappa = v.u and K in units of 2^-FA
__host__ __device__ __forceinline__ long long k_of(long long kappa, long long gk) {
  return (long long)(((__int128)kappa * gk) >> 58);
}
// a b / 2^sh of a 128-bit product, rounded
template <int SH>
__host__ __device__ __forceinline__ long long mulshift(long long a, long long b) {
  return (long long)(((__int128)a * b + ((__int128)1 << (SH - 1))) >> SH);
}
// one row's term of kappa, in units of 2^-FA
__host__ __device__ __forceinline__ long long kappa_term(long long u, long long v) {
  return mulshift<FV>(u, v);
}
// p = u / h, and w = p - K v, in units of 2^-FA
__host__ __device__ __forceinline__ long long p_of(long long u, long long g) {
  return mulshift<FA>(u, g);
}
__host__ __device__ __forceinline__ long long w_of(long long p, long long K, long long v) {
  return p - mulshift<FV>(K, v);
}
// the pivot column after the update, x = b + 2 K v_0 v_r with b = c - (v_r p_0 + p_r v_0):
// t = v_0 v_r (below 2 h < 4) in units of 2^-FA does not wait for K
__host__ __device__ __forceinline__ long long vv_of(long long v0, long long v) {
  return mulshift<2 * FV - FA>(v0, v);
}
__host__ __device__ __forceinline__ long long x_of(long long b, long long K, long long t) {
  return b + mulshift<FA - 1>(K, t);
}

}  // namespace trifx
}  // namespace tb
