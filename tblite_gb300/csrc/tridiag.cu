// Householder tridiagonalisation kernels of the eigensolver (fixed point, tridiag_fixed.cuh):
// one molecule per CTA, per thread-block cluster, or per cooperative grid, by how many columns
// fit one SM's shared memory; the batch runs one CTA or cluster per molecule.
//
// Output as LAPACK dsytrd('L'): diagonal d, off-diagonal e, tau, and the reflectors (v_0 = 1
// implied) below the subdiagonal of the column-major A, which the back-transformation reads.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <string>
#include <type_traits>

#include "engine.h"
#include "tridiag_fixed.cuh"

namespace cg = cooperative_groups;

namespace tb {

namespace {

using namespace trifx;

void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess)
    throw std::runtime_error(std::string("CUDA error '") + cudaGetErrorString(e) + "' in " + what);
}

constexpr size_t TF_SMEM_MAX = 220 * 1024;

// doubles (8 bytes) of dynamic shared memory of one of nb CTAs: columns, two landing buffers for
// u and for the pivot column (not in grid mode), v, next v, w, and per owned column the diagonal,
// s, alpha and shift from which d, e, tau and 1 / v_0 are formed at the end
constexpr size_t tf_words(int n, int nb, bool grid) {
  const size_t cols = (size_t)(n + nb - 1) / nb;
  return cols * n + (grid ? 3 : 7) * (size_t)n + 4 * cols;
}

struct TriArgs {
  int n;
  double* A;
  double *d, *e, *tau;
  long long* xch;  // grid mode: [4 n] exchange words, then 2 words per CTA for the scale
};

enum { ONE_CTA = 0, CLUSTER = 1, GRID = 2 };

__device__ __forceinline__ long long shfl_add(long long v, int o) {
  return v + __shfl_xor_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ long long warp_sum(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = shfl_add(v, o);
  return v;
}
__device__ __forceinline__ void add128(unsigned long long& lo, unsigned long long& hi,
                                       unsigned long long l, unsigned long long h) {
  asm("add.cc.u64 %0, %0, %2;\n\taddc.u64 %1, %1, %3;" : "+l"(lo), "+l"(hi) : "l"(l), "l"(h));
}
// the same on the warp-wide integer reduction: 26-bit pieces (32 of them stay below 2^31)
__device__ __forceinline__ long long redux_sum(long long v) {
  const int l = (int)(v & 0x3FFFFFF), m = (int)(v >> 26) & 0x3FFFFFF, h = (int)(v >> 52);
  const int sl = __reduce_add_sync(0xffffffffu, l), sm = __reduce_add_sync(0xffffffffu, m);
  const int sh = __reduce_add_sync(0xffffffffu, h);
  return ((long long)sh << 52) + ((long long)sm << 26) + sl;
}
__device__ __forceinline__ void redux_sum128(unsigned long long& lo, unsigned long long& hi) {
  const unsigned M = 0x3FFFFFF;
  const unsigned a0 = __reduce_add_sync(0xffffffffu, (unsigned)lo & M);
  const unsigned a1 = __reduce_add_sync(0xffffffffu, (unsigned)(lo >> 26) & M);
  const unsigned a2 =
      __reduce_add_sync(0xffffffffu, ((unsigned)(lo >> 52) | (unsigned)(hi << 12)) & M);
  const unsigned a3 = __reduce_add_sync(0xffffffffu, (unsigned)(hi >> 14) & M);
  const unsigned a4 = __reduce_add_sync(0xffffffffu, (unsigned)(hi >> 40));
  lo = (unsigned long long)a0 + ((unsigned long long)a1 << 26);  // < 2^58
  hi = ((unsigned long long)a2 >> 12) + ((unsigned long long)a3 << 14) +
       ((unsigned long long)a4 << 40);
  add128(lo, hi, (unsigned long long)a2 << 52, 0ull);
}

template <int MODE>
struct Exchange {
  int n, nb, b;
  long long *u, *c;  // [2][n] landing buffers (this CTA's shared memory, or global in grid mode)
  __device__ __forceinline__ long long get(const long long* p) const {
    if constexpr (MODE == GRID) return __ldcg(p);
    else return *p;
  }
  // store x to word `off` of buffer p of CTA `rank`
  __device__ __forceinline__ void put(long long* p, int rank, long long x) const {
    if constexpr (MODE == CLUSTER) {
      uint32_t local = (uint32_t)__cvta_generic_to_shared(p), remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
      asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(remote), "l"(x) : "memory");
    } else if constexpr (MODE == GRID) {
      __stcg(p, x);
    } else {
      *p = x;
    }
  }
  __device__ __forceinline__ int copies() const { return MODE == CLUSTER ? nb : 1; }
  __device__ __forceinline__ void barrier() const {
    if constexpr (MODE == CLUSTER) {
      asm volatile("barrier.cluster.arrive.release;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    } else if constexpr (MODE == GRID) {
      cg::this_grid().sync();
    } else {
      __syncthreads();
    }
  }
};

// one warp: the rank-2 update of the CG owned columns s .. s + CG - 1 (rows r0 .. n-1) with
// (v, w), their products with the next reflector, and the publication of these and of the next
// pivot column.  CG columns share each row's loads of v, w and the next v.
template <int MODE, int CG>
__device__ __forceinline__ void pass_group(const Exchange<MODE>& x, long long* a, int s, int ncpb,
                                           int r0, const int2* v, const int2* w, const int2* vn,
                                           long long* up, long long* cp) {
  const int n = x.n, lane = threadIdx.x & 31;
  int2 vc[CG], wc[CG];
  bool on[CG];
  long long hh[CG], cr[CG], sum[CG];
#pragma unroll
  for (int q = 0; q < CG; ++q) {
    on[q] = s + q < ncpb;
    const int j = on[q] ? x.b + (s + q) * x.nb : n - 1;
    vc[q] = v[j];
    wc[q] = w[j];
    hh[q] = cr[q] = sum[q] = 0;
  }
  const bool piv = x.b + s * x.nb == r0;  // column s is the next pivot column
  int cnt = 0;
  // RR rows per lane in flight: a row's chain from its loads to the product's sums is some 300
  // cycles, which few warps cannot fill with one row each
  auto rows = [&](auto rr, int base) {
    constexpr int RR = decltype(rr)::value;
    int2 vr[RR], wr[RR], xr[RR];
    long long t[RR][CG];
    bool in[RR];
#pragma unroll
    for (int k = 0; k < RR; ++k) {
      const int r = min(base + 32 * k + lane, n - 1);
      in[k] = base + 32 * k + lane < n;
      vr[k] = v[r];
      wr[k] = w[r];
      xr[k] = in[k] ? vn[r] : make_int2(0, 0);
#pragma unroll
      for (int q = 0; q < CG; ++q) t[k][q] = on[q] ? a[(size_t)(s + q) * n + r] : 0;
    }
#pragma unroll
    for (int k = 0; k < RR; ++k)
#pragma unroll
      for (int q = 0; q < CG; ++q) {
        t[k][q] = rank2(t[k][q], vr[k].x, vr[k].y, wr[k].x, wr[k].y, vc[q].x, vc[q].y, wc[q].x,
                        wc[q].y);
        mac(hi31(t[k][q]), lo31(t[k][q]), xr[k].x, xr[k].y, hh[q], cr[q]);
      }
#pragma unroll
    for (int k = 0; k < RR; ++k) {
      const int r = base + 32 * k + lane;
#pragma unroll
      for (int q = 0; q < CG; ++q)
        if (on[q] && in[k]) a[(size_t)(s + q) * n + r] = t[k][q];
      if (piv && in[k])
        for (int c = 0; c < x.copies(); ++c) x.put(cp + r, c, t[k][0]);
    }
    if ((cnt += RR) > 14) {  // cr stays below 2^63 for 16 terms
      cnt = 0;
#pragma unroll
      for (int q = 0; q < CG; ++q) {
        sum[q] += fold<4>(hh[q], cr[q]);
        hh[q] = cr[q] = 0;
      }
    }
  };
  constexpr int RR = CG > 2 ? 1 : 2;
  int base = r0;
  for (; base + 32 * (RR - 1) < n; base += 32 * RR) rows(std::integral_constant<int, RR>(), base);
  if (RR > 1 && base < n) rows(std::integral_constant<int, 1>(), base);
#pragma unroll
  for (int q = 0; q < CG; ++q) sum[q] += fold<4>(hh[q], cr[q]);
  // warp sums of the CG values, halving the values per exchange while more than one is left:
  // afterwards the 32 / CG lanes of group lane / (32 / CG) hold value number group
  if constexpr (CG == 4) {
    const bool up16 = lane & 16, up8 = lane & 8;
    long long k0 = up16 ? sum[2] : sum[0], k1 = up16 ? sum[3] : sum[1];
    k0 += __shfl_xor_sync(0xffffffffu, up16 ? sum[0] : sum[2], 16);
    k1 += __shfl_xor_sync(0xffffffffu, up16 ? sum[1] : sum[3], 16);
    long long k = up8 ? k1 : k0;
    k += __shfl_xor_sync(0xffffffffu, up8 ? k0 : k1, 8);
    sum[0] = shfl_add(shfl_add(shfl_add(k, 4), 2), 1);
  } else if constexpr (CG == 2) {
    const bool up16 = lane & 16;
    long long k = up16 ? sum[1] : sum[0];
    k += __shfl_xor_sync(0xffffffffu, up16 ? sum[0] : sum[1], 16);
    sum[0] = shfl_add(shfl_add(shfl_add(shfl_add(k, 8), 4), 2), 1);
  } else {
    sum[0] = warp_sum(sum[0]);
  }
  constexpr int L = 32 / CG;
  const int q = lane / L, sub = lane % L;
  if (s + q < ncpb)  // (columns past the last one hold a copy of row n - 1's limbs: not stored)
    for (int k = sub; k < x.copies(); k += L) x.put(up + x.b + (s + q) * x.nb, k, sum[0]);
}

// RPT: rows per thread of the vector steps (n <= RPT blockDim.x)
template <int MODE, int RPT>
__device__ __forceinline__ void tri_body(const TriArgs& g, int nb, int b) {
  extern __shared__ long long tf_sm[];
  __shared__ long long red[32];
  __shared__ unsigned long long redlo[32], redhi[32];
  __shared__ long long s_alpha, s_g, s_gk;
  __shared__ int s_E;
  __shared__ unsigned long long s_S;
  __shared__ long long s_scale[2 * 16];  // cluster: (E, S) of every CTA
  const int n = g.n;
  const int ncpb = b < n ? (n - b + nb - 1) / nb : 0;
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = T >> 5;
  Exchange<MODE> x;
  x.n = n;
  x.nb = nb;
  x.b = b;
  long long* p = tf_sm;
  if constexpr (MODE == GRID) {
    x.u = g.xch;
    x.c = g.xch + 2 * n;
  } else {  // first, so that every CTA of a cluster has them at the same offset
    x.u = p;
    x.c = p + 2 * n;
    p += 4 * n;
  }
  int2* v = reinterpret_cast<int2*>(p);
  int2* vn = v + n;
  int2* w = vn + n;
  const int cap = (n + nb - 1) / nb;
  long long* dg = reinterpret_cast<long long*>(w + n);  // [cap] diagonal of the owned columns
  unsigned long long* ss = reinterpret_cast<unsigned long long*>(dg + cap);  // [cap] s
  long long* sal = reinterpret_cast<long long*>(ss + cap);                   // [cap] alpha
  int* ssh = reinterpret_cast<int*>(sal + cap);  // [cap] shift, NONE without a reflector
  constexpr int NONE = 1 << 20;
  long long* a = sal + 2 * cap;

  // every CTA of a cluster runs before the first store into another's shared memory
  if constexpr (MODE == CLUSTER) x.barrier();

  // ---- own columns as raw bits, and their largest exponent field
  if (tid == 0) {
    s_E = 0;
    s_S = 0;
  }
  __syncthreads();
  {
    int E = 0;
    for (int s = wid; s < ncpb; s += nw) {
      const long long* src = reinterpret_cast<const long long*>(g.A) + (size_t)(b + s * nb) * n;
      for (int r = lane; r < n; r += 32) {
        const long long t = src[r];
        a[(size_t)s * n + r] = t;
        E = max(E, (int)((unsigned long long)t >> 52) & 0x7FF);
      }
    }
    E = __reduce_max_sync(0xffffffffu, E);
    if (lane == 0) atomicMax(&s_E, E);
  }
  __syncthreads();
  // ---- upper bound of the column sums of |A| in units of 2^(E - 1043)
  {
    const int E = s_E;
    for (int s = wid; s < ncpb; s += nw) {
      long long t = 0;
      for (int r = lane; r < n; r += 32) {
        const unsigned long long q = (unsigned long long)a[(size_t)s * n + r];
        const int ex = (int)(q >> 52) & 0x7FF;
        const unsigned m = ((unsigned)(q >> 32) & 0xFFFFFu) | 0x100000u;
        if (ex) t += (E - ex < 24 ? m >> (E - ex) : 0u) + 1u;
      }
      t = warp_sum(t);
      if (lane == 0) atomicMax(&s_S, (unsigned long long)t);
    }
  }
  __syncthreads();
  // ---- the same for the whole matrix: |A|_inf < 2^(L + E - 1043), L bits of S
  int q;
  bool bad = false;
  {
    if constexpr (MODE != ONE_CTA) {
      long long* sc = MODE == GRID ? g.xch + 4 * (size_t)n : s_scale;
      if (tid < 2 * x.copies())
        x.put(sc + 2 * b + (tid & 1), tid >> 1, (tid & 1) ? (long long)s_S : (long long)s_E);
      x.barrier();
      int top = -5000;
      for (int k = lane; k < nb; k += 32) {
        const int Ek = (int)x.get(sc + 2 * k);
        const unsigned long long Sk = (unsigned long long)x.get(sc + 2 * k + 1);
        if (Sk) top = max(top, 64 - clz64(Sk) + Ek - 1043);
        bad = bad || Ek == 0x7FF;
      }
      top = __reduce_max_sync(0xffffffffu, top);
      bad = __any_sync(0xffffffffu, bad ? 1 : 0);
      q = top > -5000 ? FA - top : 0;
    } else {
      bad = s_E == 0x7FF;
      q = s_S ? FA - (64 - clz64(s_S) + s_E - 1043) : 0;
    }
    q = min(q, 1000);
  }
  if (bad) {  // infinities or NaN: NaN throughout, as FP64 arithmetic would give
    const double nan = __longlong_as_double(0x7FF8000000000000ll);
    if (b == 0)
      for (int r = tid; r < n; r += T) {
        g.d[r] = nan;
        if (r < n - 1) {
          g.e[r] = nan;
          g.tau[r] = 0.0;
        }
      }
    return;
  }
  // ---- to fixed point; column 0 is the first pivot column, no update before it
  for (size_t t = tid; t < (size_t)ncpb * n; t += T)
    a[t] = to_fixed((unsigned long long)a[t], q);
  long long ur[RPT], br[RPT], vr[RPT], tr[RPT], xr[RPT];  // this thread's rows tid + k T
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int r = tid + k * T;
    vr[k] = 0;
    xr[k] = 0;
    if (r < n) {
      xr[k] = to_fixed((unsigned long long)(reinterpret_cast<const long long*>(g.A)[r]), q);
      v[r] = make_int2(0, 0);
      if (MODE == GRID) {
        if (b == 0) {
          __stcg(x.u + r, 0ll);
          __stcg(x.c + r, xr[k]);
        }
      } else {
        x.u[r] = 0;
        x.c[r] = xr[k];
      }
    }
  }
  if (tid == 0) s_g = s_gk = 0;
  if constexpr (MODE == GRID) x.barrier();
  else __syncthreads();

  int jm = 0, slot = 0;
  for (int i = -1; i < n - 1; ++i) {
    const int par = (i + 1) & 1;
    const long long* uin = x.u + par * n;
    const long long* cin = x.c + par * n;
    long long* un = x.u + (par ^ 1) * n;
    long long* cn = x.c + (par ^ 1) * n;
    // warps with rows >= i + 1
    const int wlo = RPT == 1 ? (i + 1) >> 5 : 0, whi = RPT == 1 ? (n + 31) >> 5 : nw;
    const bool active = wid >= wlo && wid < whi;
    const bool own = jm == b;  // column i + 1 = slot nb + jm
    // ---- kappa = v.u; everything of the update that does not wait for it
    if (active) {
      long long kap = 0, cr[RPT];
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        const int r = tid + k * T;
        const bool in = r > i && r < n;
        ur[k] = in ? x.get(uin + r) : 0;
        cr[k] = in ? x.get(cin + r) : 0;
        if (in) kap += kappa_term(ur[k], vr[k]);
      }
      const long long u1 = x.get(uin + i + 1);
      kap = redux_sum(kap);
      if (lane == 0) red[wid] = kap;
      const int2 v1s = v[i + 1];
      const long long v1 = join31(v1s.x, v1s.y);
      const long long gi = s_g, p1 = p_of(u1, gi);
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        ur[k] = p_of(ur[k], gi);  // p from here on
        br[k] = rank2(cr[k], hi31(vr[k]), lo31(vr[k]), hi31(ur[k]), lo31(ur[k]), v1s.x, v1s.y,
                      hi31(p1), lo31(p1));
        tr[k] = vv_of(v1, vr[k]);
      }
    }
    __syncthreads();
    long long K = 0;
    if (active) {
#pragma unroll 4
      for (int k = wlo; k < whi; ++k) K += red[k];
      K = k_of(K, s_gk);
      unsigned long long lo = 0, hi = 0;
#pragma unroll
      for (int k = 0; k < RPT; ++k) {
        const int r = tid + k * T;
        if (r > i && r < n) {
          xr[k] = x_of(br[k], K, tr[k]);
          if (r == i + 1) {
            if (own) dg[slot] = xr[k];
          } else {
            if (r == i + 2) s_alpha = xr[k];
            const unsigned long long ax = uabs(xr[k]);
            add128(lo, hi, ax * ax, __umul64hi(ax, ax));
          }
        }
      }
      redux_sum128(lo, hi);
      if (lane == 0) {
        redlo[wid] = lo;
        redhi[wid] = hi;
      }
    }
    if (i + 1 == n - 1) break;
    __syncthreads();
    // ---- reflector of column i + 1 by every warp with rows, its limbs, and w; the last warp
    // forms 1 / h for the next step
    if (active || wid == nw - 1) {
      unsigned long long lo = 0, hi = 0;
#pragma unroll 4
      for (int k = wlo; k < whi; ++k) add128(lo, hi, redlo[k], redhi[k]);
      const long long alpha = s_alpha;
      const Reflector f = reflector(lo, hi, alpha);
      if (active) {
        long long* acol = a + (size_t)slot * n;
#pragma unroll
        for (int k = 0; k < RPT; ++k) {
          const int r = tid + k * T;
          if (r > i && r < n) {
            const long long wr = w_of(ur[k], K, vr[k]);
            w[r] = make_int2(hi31(wr), lo31(wr));
            if (r > i + 1) {
              const long long t = f.none ? 0 : r == i + 2 ? f.v0 : shifted(xr[k], f.shift);
              vn[r] = make_int2(hi31(t), lo31(t));
              vr[k] = t;
              if (own) acol[r] = xr[k];
            }
            if (own && r == i + 1) {
              ss[slot] = f.s;
              sal[slot] = alpha;
              ssh[slot] = f.none ? NONE : f.shift;
            }
          }
        }
      }
      __syncthreads();
      if (wid == nw - 1) {
        const Scalars sc = scalars(f, alpha);
        if (lane == 0) {
          s_g = sc.g;
          s_gk = sc.gk;
        }
      }
    } else {
      __syncthreads();
    }
    // ---- update and product of the owned columns j >= i + 2
    const int r0 = i + 2;
    const int s0 = slot + (b <= jm ? 1 : 0);  // the first owned column after i + 1
    const int left = ncpb - s0;
    if (++jm == nb) {
      jm = 0;
      ++slot;
    }
    if (left > 2 * nw) {
      for (int s = s0 + 4 * wid; s < ncpb; s += 4 * nw)
        pass_group<MODE, 4>(x, a, s, ncpb, r0, v, w, vn, un, cn);
    } else if (left > nw) {
      for (int s = s0 + 2 * wid; s < ncpb; s += 2 * nw)
        pass_group<MODE, 2>(x, a, s, ncpb, r0, v, w, vn, un, cn);
    } else {
      for (int s = s0 + wid; s < ncpb; s += nw)
        pass_group<MODE, 1>(x, a, s, ncpb, r0, v, w, vn, un, cn);
    }
    int2* t = v;
    v = vn;
    vn = t;
    x.barrier();
  }
  __syncthreads();
  // ---- diagonal, off-diagonal, tau = 1 + |alpha| / s and the reflectors x / v_0 (v_0 = 1
  // implied) of the owned columns
  const double isc = pow2(-q);
  for (int s = wid; s < ncpb; s += nw) {
    const int j = b + s * nb;
    if (lane == 0) g.d[j] = (double)dg[s] * isc;
    if (j == n - 1) continue;
    const int sh = ssh[s];
    const long long al = sal[s];
    double ev = (double)al * isc, tv = 0.0, iv = 0.0;
    if (sh != NONE) {
      const double sn = (double)ss[s] * 0x1p-64;
      const double an = (double)shifted((long long)uabs(al), sh) * 0x1p-58;
      ev = (al < 0 ? sn : -sn) * pow2(FV - sh) * isc;
      tv = 1.0 + an / sn;
      iv = 1.0 / (sn + an) * pow2(sh - FV);
      if (al < 0) iv = -iv;
    }
    if (lane == 0) {
      g.e[j] = ev;
      g.tau[j] = tv;
    }
    double* dst = g.A + (size_t)j * n;
    for (int r = j + 2 + lane; r < n; r += 32) dst[r] = (double)a[(size_t)s * n + r] * iv;
  }
}

template <int MODE, int RPT>
__global__ void __launch_bounds__(512) k_tri_fixed(TriArgs g) {
  int nb = 1, b = 0;
  if constexpr (MODE != ONE_CTA) {
    nb = gridDim.x;
    b = blockIdx.x;
  }
  tri_body<MODE, RPT>(g, nb, b);
}
template <int MODE, int RPT>
__global__ void __launch_bounds__(512) kb_tri_fixed(const MolPtrs* __restrict__ mp,
                                                    const int* __restrict__ list) {
  const MolPtrs& q = mp[list[blockIdx.z]];
  TriArgs g;
  g.n = q.m.nao;
  g.A = q.A;
  g.d = q.ed;
  g.e = q.ee;
  g.tau = q.etau;
  g.xch = nullptr;
  tri_body<MODE, RPT>(g, gridDim.x, blockIdx.x);
}

// How many CTAs one molecule takes.  The columns have to fit (tf_words); past that, more CTAs
// shorten the pass over the columns but not the chain of reductions, and cost the SMs the other
// molecules of a batch want.  Measured, one molecule (us, 1 / 2 / 8 CTAs): n = 68 211 / 196 / 177,
// n = 100 417 / 343 / 279, n = 156 1000 / 738 / 507, n = 192 - / 1103 / 683; n = 384 8 CTAs 2358,
// grid of 152 CTAs 1666 (a grid barrier costs 1.2 us, a cluster barrier 0.2 us, so the grid pays
// from about 256 on).  The FP64 forms before took 620 (n = 68), 1795 (n = 192) and about 4900
// (n = 512, now 2450) for one molecule; 304 molecules of n = 50 405 (now 188), n = 156 4583 (2006),
// n = 256 24330 (11400).  304 molecules of n = 100: 1 CTA 659, 2 CTAs 971.
// More than the portable 8 CTAs are taken only where 8 do not hold the matrix (n > 430).
constexpr int TF_CLUSTER = 8, TF_CLUSTER_MAX = 16, TF_GRID_FROM = 257;
int cluster_fit(int n) {  // smallest cluster that holds an order-n matrix, 0: none
  for (int nb = 1; nb <= TF_CLUSTER_MAX; nb = nb < TF_CLUSTER ? nb + 1 : 2 * nb)
    if (sizeof(double) * tf_words(n, nb, false) <= TF_SMEM_MAX) return nb;
  return 0;
}
template <class F>
void tf_attributes(F* f) {
  ck(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TF_SMEM_MAX),
     "smem attr fixed-point tridiagonalisation");
}
void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int nb) {
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = nb;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = nb > 1 ? 1 : 0;
}

}  // namespace

size_t tridiag_exchange_words(int n) { return 4 * (size_t)n + 2 * (size_t)device_sm_count(); }

void tridiag_fixed(int n, double* A, double* d, double* e, double* tau, long long* xch,
                   cudaStream_t s) {
  TriArgs g{n, A, d, e, tau, xch};
  ++g_kernel_launches;
  if (n >= TF_GRID_FROM) {
    const int sms = device_sm_count();
    void* args[] = {&g};
    tf_attributes(k_tri_fixed<GRID, 1>);
    ck(cudaLaunchCooperativeKernel((void*)k_tri_fixed<GRID, 1>, sms, 512, args,
                                   sizeof(double) * tf_words(n, sms, true), s),
       "tridiagonalisation");
    return;
  }
  const int nb = n < 64 ? 1 : TF_CLUSTER;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(nb);
  cfg.blockDim = dim3(nb == 1 ? 512 : 256);
  cfg.dynamicSmemBytes = sizeof(double) * tf_words(n, nb, false);
  cfg.stream = s;
  cluster_config(cfg, attr, nb);
  auto launch = [&](auto* f) {
    tf_attributes(f);
    ck(cudaLaunchKernelEx(&cfg, f, g), "tridiagonalisation");
  };
  if (nb == 1) launch(k_tri_fixed<ONE_CTA, 1>);
  else launch(k_tri_fixed<CLUSTER, 1>);
}

static int g_tridiag_ctas_per_sm = 2;
static int g_tridiag_small = 1;
void set_tridiag_ctas_per_sm(int k) { g_tridiag_ctas_per_sm = k >= 2 ? 2 : 1; }
int get_tridiag_ctas_per_sm() { return g_tridiag_ctas_per_sm; }
void set_tridiag_small(int k) { g_tridiag_small = k ? 1 : 0; }
int get_tridiag_small() { return g_tridiag_small; }

// largest order the batch takes (cluster_fit reaches about 600; the other batched kernels are
// tuned and tested up to this)
int batch_tridiag_max_n() { return 547; }
void tridiag_fixed_b(const BatchLaunch& b) {
  const int n = b.nao_max, fit = cluster_fit(n);
  if (!fit) throw std::runtime_error("batched tridiagonalisation: molecule too large");
  // a wider cluster than needed only while the batch leaves half of the SMs to spare
  int nb = std::max(fit, n >= 64 && g_tridiag_ctas_per_sm == 2
                             ? std::min(TF_CLUSTER, device_sm_count() / (2 * b.count))
                             : 1);
  if (!g_tridiag_small) nb = std::max(nb, 2);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(nb, 1, b.count);
  cfg.dynamicSmemBytes = sizeof(double) * tf_words(n, nb, false);
  // 512 threads where shared memory leaves one CTA on an SM anyway, else 256: n = 50, 304
  // molecules 188 us with 256 threads, 272 us with 512; n = 156 2227 us and 2006 us
  cfg.blockDim = dim3(n > 256 || cfg.dynamicSmemBytes > TF_SMEM_MAX / 2 ? 512 : 256);
  cfg.stream = b.s;
  cluster_config(cfg, attr, nb);
  ++g_kernel_launches;
  const int tk = prof_kbegin(b.s);
  auto launch = [&](auto* f) {
    tf_attributes(f);
    if (nb > TF_CLUSTER)
      ck(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1),
         "cluster attr fixed-point tridiagonalisation");
    ck(cudaLaunchKernelEx(&cfg, f, b.mp, b.list), "batch tridiag");
  };
  if (nb == 1) launch(kb_tri_fixed<ONE_CTA, 1>);
  else if (n <= 512) launch(kb_tri_fixed<CLUSTER, 1>);
  else launch(kb_tri_fixed<CLUSTER, 2>);
  prof_kend(KS_TRIDIAG, tk, b.s);
}

}  // namespace tb
