// X = L^-T of the overlap S = L L^T in 64-bit fixed point, Cholesky factorisation and inverse in one
// elimination: the columns of [S | I] are eliminated together, and because column j of the identity
// part starts to fill exactly when column j of S is done, both share the lower triangle in place
// (row i holds the rows of L^-1 for c <= j and of the remaining S for c > j).
//
// What bounds it: n^3/3 multiply-adds and a chain of n pivots (about 1.4 us each: reciprocal square
// root, scaling, barrier).  On the FP64 pipe (64-76 cycles per warp instruction) the factorisation
// and the back substitution took 0.25 / 1.06 / 2.28 ms at 48 / 192 / 390 orbitals for one molecule;
// here it is 0.07 / 0.44 / 1.60 ms, and in an ensemble of 1024 molecules 5 ms instead of 22 ms.  An
// element update is four wide integer multiply-adds and a dozen additions and shifts, the rows are
// dealt round-robin to the CTAs of a cluster, and there is one barrier per column.  Every CTA forms
// the pivot's reciprocal square root and the scaled column and row for itself from the two
// published vectors (column j of S, row j of L^-1).
//
// Units: S and L 2^-60 (S scaled by a power of four so that its largest diagonal element is at most
// 1), L^-1 2^-55.  Error of X of Gaussian overlaps against an extended-precision elimination: 2e-16 /
// 5e-14 of the largest element at condition numbers 8e2 / 1e5 (FP64: 3e-15 / 4e-13).  A pivot below 2^-12 of the largest diagonal element (or not
// positive), or an element of L^-1 at or above 64, leaves the fixed-point range: nothing is
// written but the status, and the FP64 kernels (linalg.cu) take the matrix and decide.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <string>

#include "engine.h"
#include "tridiag_fixed.cuh"

namespace tb {

namespace {

using namespace trifx;

void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess)
    throw std::runtime_error(std::string("CUDA error '") + cudaGetErrorString(e) + "' in " + what);
}

constexpr size_t CI_SMEM_MAX = 220 * 1024;
constexpr int CI_CLUSTER = 8;
constexpr int FM = 55;  // fractional bits of L^-1

// first word of slot s (row b + s nb) in the packed rows of CTA b
__host__ __device__ __forceinline__ int ci_off(int s, int b, int nb) {
  return s * (b + 1) + nb * (s * (s - 1) / 2);
}
// 8-byte words of shared memory: packed rows of the fullest CTA, column and row landing buffers
// (two each), w
constexpr size_t ci_words(int n, int nb) {
  const size_t rows = (size_t)(n + nb - 1) / nb;
  return rows * nb + (size_t)nb * rows * (rows - 1) / 2 + 5 * (size_t)n;
}

// 1 / sqrt(a 2^-60) in units of 2^-56; 0 if a < 2^48 (above 64)
__device__ __forceinline__ long long rsqrt56(long long a) {
  if (a < (1LL << 48)) return 0;
  const int up = __clzll(a) & ~1;  // R in [2^62, 2^64)
  const unsigned long long R = (unsigned long long)a << up;
  const float y0 = rsqrtf((float)(unsigned)(R >> 40) * 0x1p-24f);
  unsigned long long y = (unsigned long long)(unsigned)(fminf(y0, 1.9999999f) * 0x1p30f) << 32;
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const long long e = (1LL << 60) - (long long)umulhi(R, umulhi(y, y));
    y += (unsigned long long)mulhi((long long)y, e * 8);
  }
  const int sh = 8 - up / 2;  // up <= 14 from a >= 2^48
  return (long long)((y + (1ull << (sh - 1))) >> sh);
}

template <bool CLUSTER>
__device__ __forceinline__ void put(long long* p, int rank, long long x) {
  if constexpr (CLUSTER) {
    uint32_t local = (uint32_t)__cvta_generic_to_shared(p), remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
    asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(remote), "l"(x) : "memory");
  } else {
    *p = x;
  }
}
template <bool CLUSTER>
__device__ __forceinline__ void barrier() {
  if constexpr (CLUSTER) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  } else {
    __syncthreads();
  }
}

// one warp: rows of the slots s0 + g ds, g < RG (all owned rows > j): B(i, c) -= l_i w_c for c <= i;
// then their elements of the next column go out (and leave a zero: the column of L^-1 starts
// there) and, for row j + 1, the row itself
template <bool CLUSTER, int RG>
__device__ __forceinline__ void ci_rows(long long* a, int n, int nb, int b, int s0, int ds, int ns,
                                        int j, const int2* w, long long* cn, long long* rn) {
  const int lane = threadIdx.x & 31;
  long long* row[RG];
  int2 l[RG];
  int len[RG];
#pragma unroll
  for (int g = 0; g < RG; ++g) {
    const int s = s0 + g * ds, i = b + s * nb;
    len[g] = s < ns ? i + 1 : 0;
    row[g] = a + ci_off(min(s, ns - 1), b, nb);
    l[g] = w[min(i, n - 1)];
  }
  const int top = min(b + (s0 + (RG - 1) * ds) * nb, n - 1) + 1;  // the last row's length or n
  for (int c = lane; c < top; c += 32) {
    const int2 wc = w[c];
    const int wt = wc.y >> 16;
#pragma unroll
    for (int g = 0; g < RG; ++g) {
      if (c < len[g]) {
        // mac and fold<2> with the rounding in the sum
        const long long hh = mw(l[g].x, wc.x, 0);
        long long cr = mw(l[g].x, wc.y, 1LL << 28);
        cr = mw(l[g].y, wc.x, cr);
        cr = mw(l[g].y >> 15, wt, cr);
        row[g][c] -= (hh << 2) + (cr >> 29);
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int g = 0; g < RG; ++g) {
    if (!len[g]) continue;
    const int i = len[g] - 1;
    const long long t = row[g][j + 1];
    if (CLUSTER ? lane < nb : lane == 0) put<CLUSTER>(cn + i, lane, t);
    if (i == j + 1) {
      for (int c = lane; c <= j; c += 32) {
        const long long x = row[g][c];
        for (int k = 0; k < (CLUSTER ? nb : 1); ++k) put<CLUSTER>(rn + c, k, x);
      }
    }
    __syncwarp();
    if (lane == 0) row[g][j + 1] = 0;
  }
}

// status: 0 done (X written), 1 outside the fixed-point range (X untouched)
template <bool CLUSTER>
__device__ __forceinline__ void ci_body(int n, const double* __restrict__ S, double* X, int* status,
                                        int nb, int b) {
  extern __shared__ long long ci_sm[];
  __shared__ int s_bad, s_E;
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, wid = tid >> 5, nw = T >> 5;
  const int ns = b < n ? (n - b + nb - 1) / nb : 0;  // owned rows
  long long* col = ci_sm;          // [2][n]
  long long* row = col + 2 * n;    // [2][n]
  int2* w = reinterpret_cast<int2*>(row + 2 * n);
  long long* a = reinterpret_cast<long long*>(w + n);
  if (tid == 0) {
    s_bad = 0;
    s_E = 0;
  }
  __syncthreads();
  // scale: 4^t above the largest diagonal element (every CTA reads the whole diagonal)
  {
    int E = 0;
    bool bad = false;
    for (int r = tid; r < n; r += T) {
      const unsigned long long q = (unsigned long long)__double_as_longlong(S[r + (size_t)r * n]);
      const int ex = (int)(q >> 52) & 0x7FF;
      bad = bad || (q >> 63) || ex == 0x7FF || ex == 0;
      // exactly a power of two still fits below it
      E = max(E, ex + ((q & 0xFFFFFFFFFFFFFull) > 0x10000 ? 1 : 0));
    }
    E = __reduce_max_sync(0xffffffffu, E);
    if (lane == 0) atomicMax(&s_E, E);
    if (bad) s_bad = 1;
  }
  __syncthreads();
  const int e2 = (s_E - 1023 + 1) & ~1;  // S 2^-e2 at most 1 (and a hair)
  bool bad = s_bad != 0 || e2 > 900 || e2 < -900;
  const int q = FA - e2;
  for (int s = wid; s < ns && !bad; s += nw) {
    const int i = b + s * nb;
    long long* p = a + ci_off(s, b, nb);
    bool out = false;
    for (int c = lane; c <= i; c += 32) {  // row i = column i (symmetric)
      const unsigned long long bits =
          (unsigned long long)__double_as_longlong(S[c + (size_t)i * n]);
      out = out || (int)((bits >> 52) & 0x7FF) > s_E;
      p[c] = c == 0 ? 0 : to_fixed(bits, q);
    }
    if (__any_sync(0xffffffffu, out ? 1 : 0)) s_bad = 1;
  }
  // column 0 for every CTA (symmetric: row 0); in the rows it is the first of L^-1
  for (int r = tid; r < n; r += T)
    col[r] = to_fixed((unsigned long long)__double_as_longlong(S[r]), q);
  // one agreement for the cluster: a bad element anywhere stops all (also the cluster's start
  // barrier before the first store into another CTA's shared memory)
  __syncthreads();
  if constexpr (CLUSTER) {
    barrier<CLUSTER>();
    if (tid < nb && s_bad) {
      uint32_t local = (uint32_t)__cvta_generic_to_shared(&s_bad), remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(tid));
      asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(remote), "r"(1) : "memory");
    }
    barrier<CLUSTER>();
  }
  bad = bad || s_bad != 0;
  int jm = 0, js = 0;  // j % nb, j / nb
  for (int j = 0; j < n && !bad; ++j) {
    const long long* cj = col + (j & 1) * n;
    const long long* rj = row + (j & 1) * n;
    long long* cn = col + ((j + 1) & 1) * n;
    long long* rn = row + ((j + 1) & 1) * n;
    const long long r = rsqrt56(cj[j]);
    bool over = r == 0;
    const bool own = jm == b;
    long long* dst = a + ci_off(js, b, nb);
    for (int c = tid; c < n; c += T) {
      const long long t = c < j    ? mulshift<56>(rj[c], r)
                          : c == j ? (r + 1) >> 1
                                   : mulshift<56>(cj[c], r);
      over = over || t >= (1LL << 61) || t <= -(1LL << 61);
      w[c] = make_int2(hi31(t), lo31(t));
      if (own && c <= j) dst[c] = t;
    }
    // every CTA sees the same numbers, so all of them leave together
    if (__syncthreads_or(over ? 1 : 0)) {
      bad = true;
      break;
    }
    const int first = js + (b <= jm ? 1 : 0);  // the first owned row after j
    if (++jm == nb) {
      jm = 0;
      ++js;
    }
    const int left = ns - first;
    if (left > 2 * nw) {
      for (int s = first + wid; s < ns; s += 4 * nw)
        ci_rows<CLUSTER, 4>(a, n, nb, b, s, nw, ns, j, w, cn, rn);
    } else if (left > nw) {
      for (int s = first + wid; s < ns; s += 2 * nw)
        ci_rows<CLUSTER, 2>(a, n, nb, b, s, nw, ns, j, w, cn, rn);
    } else {
      for (int s = first + wid; s < ns; s += nw)
        ci_rows<CLUSTER, 1>(a, n, nb, b, s, nw, ns, j, w, cn, rn);
    }
    barrier<CLUSTER>();
  }
  if (b == 0 && tid == 0) *status = bad ? 1 : 0;
  if (bad) return;
  // X(c, i) = L^-1(i, c): column i of X is row i
  const double f = pow2(-FM - e2 / 2);
  for (int s = wid; s < ns; s += nw) {
    const int i = b + s * nb;
    const long long* p = a + ci_off(s, b, nb);
    double* x = X + (size_t)i * n;
    for (int c = lane; c < n; c += 32) x[c] = c <= i ? (double)p[c] * f : 0.0;
  }
}

template <bool CLUSTER>
__global__ void __launch_bounds__(512) k_cholinv(int n, const double* __restrict__ S, double* X,
                                                 int* status) {
  ci_body<CLUSTER>(n, S, X, status, CLUSTER ? gridDim.x : 1, CLUSTER ? blockIdx.x : 0);
}
template <bool CLUSTER>
__global__ void __launch_bounds__(512) kb_cholinv(const MolPtrs* __restrict__ mp,
                                                  const int* __restrict__ list) {
  const MolPtrs& q = mp[list[blockIdx.z]];
  ci_body<CLUSTER>(q.m.nao, q.S, q.X, q.estatus, CLUSTER ? gridDim.x : 1,
                   CLUSTER ? blockIdx.x : 0);
}

int ci_fit(int n) {  // smallest cluster that holds an order-n matrix, 0: none
  for (int nb = 1; nb <= CI_CLUSTER; ++nb)
    if (sizeof(long long) * ci_words(n, nb) <= CI_SMEM_MAX) return nb;
  return 0;
}
void ci_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int n, int nb, int count,
               cudaStream_t s) {
  cfg.gridDim = dim3(nb, 1, count);
  cfg.dynamicSmemBytes = sizeof(long long) * ci_words(n, nb);
  cfg.blockDim = dim3(n > 128 || cfg.dynamicSmemBytes > CI_SMEM_MAX / 2 ? 512 : 256);
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = nb;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = nb > 1 ? 1 : 0;
}
template <class F>
void ci_attr(F* f) {
  ck(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CI_SMEM_MAX),
     "smem attr fixed-point Cholesky inverse");
}

}  // namespace

bool cholinv_fixed(int n, const double* S, double* X, int* status, cudaStream_t s) {
  const int fit = ci_fit(n);
  if (!fit || n > TRIDIAG_FIXED_MAX) return false;
  // one CTA has no cluster barrier, eight have an eighth of the work: 18 against 21 us at 12 orbitals,
  // 78 against 70 us at 48, 0.87 against 0.44 ms at 192
  const int nb = n < 48 ? 1 : CI_CLUSTER;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  ci_config(cfg, attr, n, nb, 1, s);
  ++g_kernel_launches;
  if (nb == 1) {
    ci_attr(k_cholinv<false>);
    ck(cudaLaunchKernelEx(&cfg, k_cholinv<false>, n, S, X, status), "Cholesky inverse");
  } else {
    ci_attr(k_cholinv<true>);
    ck(cudaLaunchKernelEx(&cfg, k_cholinv<true>, n, S, X, status), "Cholesky inverse");
  }
  return true;
}

bool cholinv_fixed_b(const BatchLaunch& b) {
  const int n = b.nao_max, fit = ci_fit(n);
  if (!fit) return false;
  // more CTAs than a molecule needs only while the batch leaves SMs free
  const int nb = std::max(
      fit, n < 48 ? 1 : std::min(CI_CLUSTER, device_sm_count() / std::max(b.count, 1)));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  ci_config(cfg, attr, n, nb, b.count, b.s);
  ++g_kernel_launches;
  if (nb == 1) {
    ci_attr(kb_cholinv<false>);
    ck(cudaLaunchKernelEx(&cfg, kb_cholinv<false>, b.mp, b.list), "batch Cholesky inverse");
  } else {
    ci_attr(kb_cholinv<true>);
    ck(cudaLaunchKernelEx(&cfg, kb_cholinv<true>, b.mp, b.list), "batch Cholesky inverse");
  }
  return true;
}

}  // namespace tb
