// Generalised symmetric eigenproblem  F C = S C e  of the SCF (reference
// src/tblite/lapack/sygvd.f90:125-151, LAPACK dsygvd itype 1, jobz V), written for GB300.
//
//   once per geometry   S = L L^T (Cholesky), X = L^-T                      (linalg.cu)
//   every iteration     A = X^T F X            two triangle-aware GEMMs
//                       A = Q T Q^T            Householder tridiagonalisation (tridiag.cu up to
//                                              512 orbitals, the kernels here above)
//                       T y = y e              all eigenvalues by Sturm-count bisection
//   after Fermi filling eigenvectors only for the occupied orbitals: inverse iteration on T,
//                       clusters of close eigenvalues re-orthonormalised + Rayleigh-Ritz,
//                       back-transformation Z = Q Y (column blocks per CTA, reflectors
//                       staged in shared memory), C = X Z (triangular GEMM).
//
// The reference refactorises S on every call of dsygvd; the factor is identical, so it is
// computed once here.  Eigenvector signs are arbitrary in both codes; every quantity the
// engine derives (density, energy weighted density, charges) is sign invariant.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <stdexcept>
#include <vector>

#include "engine.h"
#include "warp_sums.cuh"

namespace cg = cooperative_groups;

namespace tb {

static void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess)
    throw std::runtime_error(std::string("CUDA error '") + cudaGetErrorString(e) + "' in " + what);
}

// GEMMs of the one-molecule path go to the tensor cores from 128 orbitals on
static inline bool split_gemm(int n) { return g_split_gemm && n >= 128; }
extern bool g_pipe_gemm;
// The split products of a small molecule on the pipelined kernel: k_ogemm splits the operands of
// every tile pair anew, 65 us at 192 orbitals and two exponent launches of 3 us; operand split and
// pipelined product take 10 + 22 us, with a smaller error (28 products of balanced digits).  Above
// TRIDIAG_FIXED_MAX k_ogemm's results stay (see there); below 128 orbitals the FP64 tiles are
// faster (8 us at 68).
constexpr int PAIR_MAX = TRIDIAG_FIXED_MAX;
static inline bool pair_gemm(int n, const void* pair) {
  return pair && split_gemm(n) && g_pipe_gemm && n <= PAIR_MAX;
}

struct EigenSolver {
  int n = 0;
  cudaStream_t stream = nullptr;
  double *L = nullptr, *X = nullptr, *A = nullptr, *T1 = nullptr;
  double *d = nullptr, *e = nullptr, *tau = nullptr, *w = nullptr, *pv = nullptr, *scal = nullptr;
  long long* xch = nullptr;  // exchange of the grid-wide tridiagonalisation
  double *lu = nullptr;   // inverse iteration scratch [5][n][n]
  double *tw = nullptr;   // eigenvalue scratch: e^2 [n] (double), d and e^2 [n] (float)
  double *Y = nullptr;    // eigenvectors of T, column-major [k][n]
  int* status = nullptr;  // device
  void* pair = nullptr;   // workspace of the pipelined products up to PAIR_MAX orbitals
  bool pair_on = true;
  bool ordered = false;  // roundings of the FP64 kernels (eigen_set_ordered)
  int* gstatus = nullptr; // device: 1 once a tensor-core GEMM did not answer
  int* hstatus = nullptr; // pinned
  int coop_blocks = 0;
  int cap = 0;  // buffers hold problems up to this order
};

int eigen_capacity(const EigenSolver* e) { return e ? e->cap : 0; }
void eigen_resize(EigenSolver* e, int n) {
  if (n > e->cap) throw std::runtime_error("eigen solver capacity exceeded");
  e->n = n;
}

// ------------------------------------------------------------------------------------------
// Householder tridiagonalisation of the symmetric A (column-major, full storage), lower form
// as LAPACK dsytd2('L'): for column i, v = [1; A(i+2:n, i)], tau_i, e_i = beta, d_i = A(i,i).
// Warp 0 of block 0 owns the column that becomes the next pivot column: it updates that column
// during the rank-2 update of step i and immediately builds reflector i+1 from it, so every
// step needs two grid barriers (after the reflector, after the symmetric matrix-vector product).
// ------------------------------------------------------------------------------------------
// 1/x from the hardware approximation refined by two Newton steps (relative error ~1e-16);
// used where x is bounded away from zero and denormals (pivots, Sturm quotients).
__device__ __forceinline__ double frcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  double e = fma(-x, r, 1.0);
  r = fma(r, e, r);
  e = fma(-x, r, 1.0);
  return fma(r, e, r);
}

__device__ __forceinline__ double wred(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ double block_sum256(double v, double* red) {
  v = wred(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
  __syncthreads();
  return t;
}

// reflector for column i, built by all threads of one block; writes tau[i], e[i], scaled v
__device__ void make_reflector(int n, int i, double* A, double* tau, double* e, double* red) {
  double* col = A + (size_t)i * n;
  const double alpha = col[i + 1];
  double s = 0.0;
#pragma unroll 4
  for (int r = i + 2 + threadIdx.x; r < n; r += blockDim.x) s += col[r] * col[r];
  s = block_sum256(s, red);
  double t = 0.0, beta = alpha;
  if (s > 0.0) {
    beta = -copysign(sqrt(alpha * alpha + s), alpha);
    t = (beta - alpha) / beta;
    const double sc = 1.0 / (alpha - beta);
#pragma unroll 4
    for (int r = i + 2 + threadIdx.x; r < n; r += blockDim.x) col[r] *= sc;
  }
  if (threadIdx.x == 0) {
    tau[i] = t;
    e[i] = beta;
  }
}

__global__ void __launch_bounds__(256) k_tridiag(int n, double* A, double* d, double* e,
                                                 double* tau, double* pv, double* scal) {
  cg::grid_group grid = cg::this_grid();
  const int lane = threadIdx.x & 31;
  const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarp = (gridDim.x * blockDim.x) >> 5;
  const int bw = blockDim.x >> 5;  // warps per block
  // warps that update trailing columns 1..m-1 (block 0 owns column 0 and the next reflector)
  const bool solo = gridDim.x == 1;
  const int uw = solo ? gwarp : gwarp - bw, nuw = solo ? nwarp : nwarp - bw;
  __shared__ double red[32];
  __shared__ double sK;
  (void)scal;
  if (blockIdx.x == 0 && n > 1) make_reflector(n, 0, A, tau, e, red);
  grid.sync();
  for (int i = 0; i < n - 1; ++i) {
    const int m = n - i - 1;  // size of the trailing block A22 = A(i+1:n, i+1:n)
    const double* v = A + (size_t)i * n + (i + 1);  // v[0] is implicitly 1
    const double t = tau[i];
    // p = t * A22 v  (rows of A22 via its columns, symmetric), also p_r v_r
    for (int r = gwarp; r < m; r += nwarp) {
      const double* colr = A + (size_t)(i + 1 + r) * n + (i + 1);
      double s = 0.0;
      if (lane < m) s = lane == 0 ? colr[0] : colr[lane] * v[lane];
#pragma unroll 8
      for (int c = lane + 32; c < m; c += 32) s += colr[c] * v[c];
      s = wred(s) * t;
      if (lane == 0) {
        pv[r] = s;
        pv[n + r] = s * (r == 0 ? 1.0 : v[r]);
      }
    }
    grid.sync();
    // K = -1/2 t (p . v), reduced by every block in the same order
    {
      double s = 0.0;
      for (int r = threadIdx.x; r < m; r += blockDim.x) s += pv[n + r];
      s = block_sum256(s, red);
      if (threadIdx.x == 0) sK = -0.5 * t * s;
      __syncthreads();
    }
    const double K = sK;
    if (blockIdx.x == 0) {
      if (threadIdx.x == 0) d[i] = A[i + (size_t)i * n];
      // column 0 of A22 (global column i+1), then reflector i+1 from it
      if (t != 0.0) {
        const double wc = pv[0] + K;
        double* colc = A + (size_t)(i + 1) * n + (i + 1);
#pragma unroll 4
        for (int r = threadIdx.x; r < m; r += blockDim.x) {
          const double vr = r == 0 ? 1.0 : v[r];
          const double wr = pv[r] + K * vr;
          colc[r] -= vr * wc + wr;
        }
      }
      __syncthreads();
      if (i + 1 < n - 1) make_reflector(n, i + 1, A, tau, e, red);
      else if (threadIdx.x == 0) d[n - 1] = A[(n - 1) + (size_t)(n - 1) * n];
    }
    // rank-2 update of the remaining columns: A22 -= v w^T + w v^T, w = p + K v
    if (t != 0.0 && uw >= 0) {
      for (int c = 1 + uw; c < m; c += nuw) {
        const double vc = v[c];
        const double wc = pv[c] + K * vc;
        double* colc = A + (size_t)(i + 1 + c) * n + (i + 1);
        if (lane == 0) colc[0] -= wc + (pv[0] + K) * vc;
#pragma unroll 8
        for (int r = 1 + lane; r < m; r += 32) {
          const double vr = v[r];
          colc[r] -= vr * wc + (pv[r] + K * vr) * vc;
        }
      }
    }
    grid.sync();
  }
  if (n == 1 && gwarp == 0 && lane == 0) d[0] = A[0];
}

constexpr size_t TRIDIAG_SMEM_MAX = 220 * 1024;
constexpr int TRIDIAG_ROWS = 8;  // rows per thread of the vector steps: n <= 2048
constexpr size_t tridiag_smem_doubles(int n, int nb) {
  return ((size_t)(n + nb - 1) / nb + 3) * n;
}

// Shared-memory resident variant for n where every block can hold its columns: global column j
// lives in block j % nb (slot j / nb) for the whole reduction.  One grid barrier per column: p = t A v
// (each block's own entries) and the next pivot column before its last update (from its owner)
// travel through L2; K, w, the pivot column after the update and its reflector are formed by every
// block for itself, and the update of the owned columns and their products with the next reflector
// are one pass.  FP64 with the same operations in the same order as the two-barrier form before it,
// so the results are the same bit for bit; the sums over the warps and the scalars are left to one
// warp, because an FP64 instruction takes its scheduler 64 cycles whatever the lanes do.
__global__ void __launch_bounds__(256) k_tridiag_smem(int n, double* A, double* d, double* e,
                                                      double* tau, double* buf) {
  cg::grid_group grid = cg::this_grid();
  extern __shared__ double sm[];
  const int nb = (int)gridDim.x, b = (int)blockIdx.x;
  const int ncpb = (n + nb - 1) / nb;
  double* scol = sm;                   // [ncpb][n]
  double* sv = sm + (size_t)ncpb * n;  // [n]  reflector of the current step
  double* sn = sv + n;                 // [n]  pivot column, then the next reflector
  double* sp = sn + n;                 // [n]  w of the current step
  __shared__ double red[8];
  __shared__ double sK, s_t, s_sc;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nwb = blockDim.x >> 5;
  for (int s = 0; s < ncpb; ++s) {
    const int j = b + s * nb;
    if (j >= n) break;
    for (int r = tid; r < n; r += blockDim.x) scol[(size_t)s * n + r] = A[r + (size_t)j * n];
  }
  for (int r = tid; r < n; r += blockDim.x) sn[r] = A[r];
  grid.sync();  // column 0 has been read everywhere before its owner writes the reflector there
  double t = 0.0;
  for (int i = -1; i < n - 1; ++i) {
    const double* in = buf + (size_t)(i & 1) * 3 * n;
    double* out = buf + (size_t)((i + 1) & 1) * 3 * n;
    if (i >= 0) {
      // K = -1/2 t (p . v), same order in every block; w = p + K v once per row
      double pr[TRIDIAG_ROWS], qr[TRIDIAG_ROWS], cr[TRIDIAG_ROWS];
#pragma unroll
      for (int k = 0; k < TRIDIAG_ROWS; ++k) {
        const int r = i + 1 + tid + k * 256;
        const bool on = r < n;
        pr[k] = on ? __ldcg(in + r) : 0.0;
        qr[k] = on ? __ldcg(in + n + r) : 0.0;
        cr[k] = on ? __ldcg(in + 2 * n + r) : 0.0;
      }
      if (t != 0.0) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < TRIDIAG_ROWS; ++k)
          if (i + 1 + tid + k * 256 < n) s += qr[k];
        s = wred(s);
        if (lane == 0) red[wid] = s;
        __syncthreads();
        if (wid == 0) {
          double a = 0.0;
          for (int k = 0; k < nwb; ++k) a += red[k];
          if (lane == 0) sK = -0.5 * t * a;
        }
        __syncthreads();
        const double K = sK;
#pragma unroll
        for (int k = 0; k < TRIDIAG_ROWS; ++k) {
          const int r = i + 1 + tid + k * 256;
          if (r < n) {
            pr[k] = fma(K, sv[r], pr[k]);
            sp[r] = pr[k];
          }
        }
        __syncthreads();
        const double vc = sv[i + 1], wc = sp[i + 1];
#pragma unroll
        for (int k = 0; k < TRIDIAG_ROWS; ++k) {
          const int r = i + 1 + tid + k * 256;
          if (r < n) cr[k] = fma(-sv[r], wc, fma(-pr[k], vc, cr[k]));
        }
      }
#pragma unroll
      for (int k = 0; k < TRIDIAG_ROWS; ++k) {
        const int r = i + 1 + tid + k * 256;
        if (r < n) sn[r] = cr[k];
      }
      __syncthreads();
    }
    const bool own = (i + 1) % nb == b;
    if (own && tid == 0) d[i + 1] = sn[i + 1];
    if (i + 1 == n - 1) break;
    // reflector of column i + 1
    {
      double s = 0.0;
      for (int r = i + 3 + tid; r < n; r += blockDim.x) s += sn[r] * sn[r];
      s = wred(s);
      if (lane == 0) red[wid] = s;
      __syncthreads();
      if (wid < 2) {  // each of the two divisions on a scheduler of its own
        s = 0.0;
        for (int k = 0; k < nwb; ++k) s += red[k];
        const double alpha = sn[i + 2];
        const double beta = s > 0.0 ? -copysign(sqrt(alpha * alpha + s), alpha) : alpha;
        if (wid == 0) {
          const double sc = s > 0.0 ? 1.0 / (alpha - beta) : 0.0;
          if (lane == 0) s_sc = sc;
        } else {
          const double tn = s > 0.0 ? (beta - alpha) / beta : 0.0;
          if (lane == 0) {
            s_t = tn;
            if (own) {
              tau[i + 1] = tn;
              e[i + 1] = beta;
            }
          }
        }
      }
      __syncthreads();
      const double sc = s_sc;
      for (int r = i + 3 + tid; r < n; r += blockDim.x) {
        const double v = sn[r] * sc;
        sn[r] = v;
        if (own) A[r + (size_t)(i + 1) * n] = v;
      }
      if (tid == 0) sn[i + 2] = 1.0;
    }
    const double tn = s_t;
    __syncthreads();
    // owned columns j >= i + 2: A -= v w^T + w v^T (two FMAs per element), then
    // p_j = t A(i+2:n, j) . v with the next reflector; the next pivot column goes out too
    const int r0 = i + 2;
    for (int s = wid; s < ncpb; s += nwb) {
      const int j = b + s * nb;
      if (j < r0 || j >= n) continue;
      double* col = scol + (size_t)s * n;
      const bool piv = j == r0;
      double acc = 0.0;
      if (t != 0.0) {
        const double vc = sv[j], wc = sp[j];
#pragma unroll 4
        for (int r = r0 + lane; r < n; r += 32) {
          const double c = fma(-sv[r], wc, fma(-sp[r], vc, col[r]));
          col[r] = c;
          acc += c * sn[r];
          if (piv) __stcg(out + 2 * n + r, c);
        }
      } else {
        for (int r = r0 + lane; r < n; r += 32) {
          acc += col[r] * sn[r];
          if (piv) __stcg(out + 2 * n + r, col[r]);
        }
      }
      acc = wred(acc) * tn;
      if (lane == 0) {
        __stcg(out + j, acc);
        __stcg(out + n + j, acc * sn[j]);
      }
    }
    t = tn;
    double* x = sv;
    sv = sn;
    sn = x;
    grid.sync();
  }
}

// ------------------------------------------------------------------------------------------
// Eigenvalues of the tridiagonal T (one thread per eigenvalue, ascending order).
//
// GB300 executes FP32 about 60x faster than FP64, so each eigenvalue is found in three stages:
//   1. FP32 bisection on the Sturm count of fl32(T) down to a bracket of 2^-21 |T|;
//   2. the bracket is widened by 2^-16 |T| (the FP32 count is exact for a matrix within a few
//      FP32 ulps of T, i.e. within ~1e-6 |T| in its eigenvalues) and both ends are checked
//      with FP64 Sturm counts; a bracket that fails the check restarts from the Gershgorin
//      interval;
//   3. FP64: while the bracket holds exactly this eigenvalue, regula falsi with the Illinois
//      modification on det(T - x I) (superlinear; a point at a converged end is moved half a
//      tolerance inside); otherwise, and whenever three interpolation steps have not halved
//      the bracket, bisection.  About 7 FP64 counts per isolated eigenvalue instead of ~55.
// The stopping rule is the one of plain bisection (width <= 2 eps max(|lo|, |hi|) + 4 pivmin)
// and the result is the midpoint of the final bracket.  The FP64 sweep is the determinant
// recurrence p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}: division free, the pair rescaled by
// a power of two every 8 steps (the exponent is carried, so det(T - x I) = p * 2^E), an exact
// zero takes the sign opposite to its predecessor; the number of sign changes is the number
// of eigenvalues below x.
// ------------------------------------------------------------------------------------------
// One step of the FP64 recurrence.  FP64 issue slots are scarce on this GPU: the sign tests,
// the zero test and the exponent test read the high word with integer instructions, so per
// step the FP64 pipe sees one subtraction, one multiplication and one FMA.
__device__ __forceinline__ void step64(double a, double ee, double& p0, double& p1, int& h1,
                                       int& cnt) {
  double p2 = fma(a, p1, -ee * p0);
  const bool z = ((__double2hiint(p2) << 1) | __double2loint(p2)) == 0;
  p2 = z ? (h1 < 0 ? 0x1p-900 : -0x1p-900) : p2;  // exact zero: opposite sign to p1
  const int h2 = __double2hiint(p2);
  cnt += (unsigned)(h2 ^ h1) >> 31;
  p0 = p1;
  p1 = p2;
  h1 = h2;
}
__device__ __forceinline__ void rescale64(double& p0, double& p1, int& h1, int& E) {
  const int be = (h1 >> 20) & 0x7ff;  // biased exponent of |p1|
  if (be > 1023 + 400 || be < 1023 - 400) {
    const double sc = __hiloint2double((2046 - be) << 20, 0);  // 2^-(be - 1023), exact
    p1 *= sc;
    p0 *= sc;
    h1 = __double2hiint(p1);
    E += be - 1023;
  }
}
// Sturm count below x and det(T - x I) = fm * 2^fe.  Blocks of 8 steps load their d and e^2
// together, so the loads of a block overlap and the FMA chain runs back to back.
__device__ __forceinline__ int sweep64(int n, const double* __restrict__ d,
                                       const double* __restrict__ e2, double x, double& fm,
                                       int& fe) {
  double p0 = 1.0, p1 = d[0] - x;
  if (p1 == 0.0) p1 = -0x1p-900;
  int h1 = __double2hiint(p1);
  int cnt = (unsigned)h1 >> 31, E = 0;
  int i = 1;
  for (; i + 8 <= n; i += 8) {
    double dv[8], ev[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      dv[k] = d[i + k];
      ev[k] = e2[i + k - 1];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) step64(dv[k] - x, ev[k], p0, p1, h1, cnt);
    rescale64(p0, p1, h1, E);
  }
  for (; i < n; ++i) step64(d[i] - x, e2[i - 1], p0, p1, h1, cnt);
  fm = p1;
  fe = E;
  return cnt;
}

__device__ __forceinline__ void step32(float a, float ee, float& p0, float& p1, int& cnt) {
  float p2 = fmaf(a, p1, -ee * p0);
  p2 = p2 == 0.f ? -copysignf(0x1p-100f, p1) : p2;
  cnt += (unsigned)(__float_as_int(p2) ^ __float_as_int(p1)) >> 31;
  const float m = fabsf(p2);
  const float sc = m > 0x1p32f ? 0x1p-64f : (m < 0x1p-32f ? 0x1p64f : 1.f);
  p0 = p1 * sc;
  p1 = p2 * sc;
}
__device__ __forceinline__ int sweep32(int n, const float* __restrict__ d,
                                       const float* __restrict__ e2, float x) {
  float p0 = 1.f, p1 = d[0] - x;
  if (p1 == 0.f) p1 = -0x1p-100f;
  int cnt = p1 < 0.f;
  int i = 1;
  for (; i + 8 <= n; i += 8) {
    float dv[8], ev[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      dv[k] = d[i + k];
      ev[k] = e2[i + k - 1];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) step32(dv[k] - x, ev[k], p0, p1, cnt);
  }
  for (; i < n; ++i) step32(d[i] - x, e2[i - 1], p0, p1, cnt);
  return cnt;
}

// Gershgorin interval [lo, hi] (widened by 4 ulps) and pivmin of T, for every thread of the block
struct TriBounds {
  double lo, hi, tnorm, pivmin;
};
__device__ TriBounds tri_bounds(int n, const double* __restrict__ d,
                                const double* __restrict__ e) {
  __shared__ double red[3][32];
  __shared__ TriBounds out;
  double lo = 1e300, hi = -1e300, emax = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
    if (i < n - 1) emax = fmax(emax, e[i] * e[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) {
    red[0][w] = lo;
    red[1][w] = hi;
    red[2][w] = emax;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < nw; ++k) {
      lo = fmin(lo, red[0][k]);
      hi = fmax(hi, red[1][k]);
      emax = fmax(emax, red[2][k]);
    }
    const double tnorm = fmax(fabs(lo), fabs(hi));
    out.lo = lo - 8.9e-16 * tnorm - 1e-300;
    out.hi = hi + 8.9e-16 * tnorm + 1e-300;
    out.tnorm = fmax(fabs(out.lo), fabs(out.hi));
    out.pivmin = fmax(2.2250738585072014e-308 * fmax(1.0, emax), 1e-300);
  }
  __syncthreads();
  return out;
}

// The FP64 stage with 16 lanes per eigenvalue: every round counts at 16 ascending points and keeps
// the neighbouring pair that encloses the eigenvalue.  Round one takes both ends of the widened
// bracket and rungs of a ladder (factor 4) around the FP32 result; a bracket that misses falls back
// to the Gershgorin interval.  While the bracket of width W holds only this eigenvalue the points
// are a ladder (factor 8, W/4 down to half a tolerance) around the secant point, so the bracket
// shrinks to about the secant's error at every round; else, and within 8 tolerances (where the
// rungs round to the same few numbers), they are equidistant.  Four or five
// counts one after the other instead of nine (192 orbitals: see k_eigvals), same stopping rule.
__device__ double tri_ladder(int n, const double* __restrict__ d, const double* __restrict__ e2,
                             float flo, float fhi, int j, bool active, const TriBounds& b) {
  const int sub = threadIdx.x & 15, lead = (threadIdx.x & 31) - sub;
  const double wid = b.tnorm * 0x1p-16;
  double lo = fmax(b.lo, (double)flo - wid), hi = fmin(b.hi, (double)fhi + wid);
  double flm = 0.0, fhm = 0.0;
  int fle = 0, fhe = 0, clo = 0, chi = n;
  for (int it = 0; it < 80; ++it) {
    const double W = hi - lo;
    const double tol = 2.0 * 2.220446049250313e-16 * fmax(fabs(lo), fabs(hi)) + 4.0 * b.pivmin;
    const double mid = 0.5 * (lo + hi);
    const bool done = !active || W <= tol || !(mid > lo && mid < hi);
    if (it > 0 && __all_sync(0xffffffffu, done)) break;
    const bool iso = it > 0 && clo == j && chi == j + 1 && W > 8.0 * tol;
    double x;
    const int m = sub < 8 ? sub : 15 - sub;  // rung: 0 the outermost
    if (it == 0 || iso) {
      double c = 0.5 * ((double)flo + (double)fhi);
      if (iso) {
        const int E = max(fle, fhe);
        const double a = scalbn(flm, fle - E), q = scalbn(fhm, fhe - E);
        c = lo + a / (a - q) * W;
      }
      const double step = it == 0 ? scalbn(W, -1 - 2 * m) : fmax(scalbn(W, -2 - 3 * m), 0.5 * tol);
      x = fmin(fmax(sub < 8 ? c - step : c + step, lo), hi);
      if (it == 0) x = sub == 0 ? lo : sub == 15 ? hi : x;
    } else {
      x = lo + W * ((sub + 1) * (1.0 / 17.0));
    }
    double fm;
    int fe;
    const int c = sweep64(n, d, e2, x, fm, fe);
    const unsigned above = (__ballot_sync(0xffffffffu, c > j) >> lead) & 0xFFFFu;
    const int f = above ? __ffs(above) - 1 : 16;  // first point above the eigenvalue
    const int il = lead + max(f - 1, 0), ih = lead + min(f, 15);
    const double xl = __shfl_sync(0xffffffffu, x, il), xh = __shfl_sync(0xffffffffu, x, ih);
    const double ml = __shfl_sync(0xffffffffu, fm, il), mh = __shfl_sync(0xffffffffu, fm, ih);
    const int el = __shfl_sync(0xffffffffu, fe, il), eh = __shfl_sync(0xffffffffu, fe, ih);
    const int cl = __shfl_sync(0xffffffffu, c, il), ch = __shfl_sync(0xffffffffu, c, ih);
    if (it == 0 && (f == 0 || f == 16)) {  // the FP32 stage missed: full interval
      lo = b.lo;
      hi = b.hi;
      continue;
    }
    if (done && it > 0) continue;
    if (f > 0) {
      lo = xl;
      clo = cl;
      flm = ml;
      fle = el;
    }
    if (f < 16) {
      hi = xh;
      chi = ch;
      fhm = mh;
      fhe = eh;
    }
  }
  return 0.5 * (lo + hi);
}

// eigenvalue j of T; warp-collective (every lane of the warp calls it, inactive lanes too).  A group
// of 2^D neighbouring lanes shares one eigenvalue: in the FP32 stage its lanes evaluate the 2^D - 1
// midpoints of the next D bisection levels at once (the same midpoints as level by level, so the
// bracket is the same bit for bit; 2^D - 1 counts instead of D, in the time of one), and the FP64
// check takes both ends at once.  Every lane of the group returns the eigenvalue.
template <int D>
__device__ double tri_eigenvalue(int n, const double* __restrict__ d, const double* __restrict__ e2,
                                 const float* __restrict__ fd, const float* __restrict__ fe2,
                                 int j, bool active, const TriBounds& b, bool ladder = true) {
  constexpr int G = 1 << D;
  const int sub = threadIdx.x & (G - 1), lead = (threadIdx.x & 31) - sub;
  // 1. FP32 bisection
  float flo = __double2float_rd(b.lo), fhi = __double2float_ru(b.hi);
  const float ftol = (float)(b.tnorm * 0x1p-21);
  for (int it = 0; it < 64; ++it) {
    const float x = 0.5f * (flo + fhi);
    const bool done = !active || fhi - flo <= ftol || x <= flo || x >= fhi;
    if (__all_sync(0xffffffffu, done)) break;
    if constexpr (D == 0) {
      if (done) continue;
      if (sweep32(n, fd, fe2, x) > j) fhi = x;
      else flo = x;
    } else {
      // lane sub evaluates node sub of the heap (1 the root, 2 q below and 2 q + 1 above node q)
      float lo = flo, hi = fhi;
      const int node = sub ? sub : 1;
      for (int l = 30 - __clz(node); l >= 0; --l) {
        const float m = 0.5f * (lo + hi);
        if ((node >> l) & 1) lo = m;
        else hi = m;
      }
      const int above = sweep32(n, fd, fe2, 0.5f * (lo + hi)) > j;
      int q = 1;
#pragma unroll
      for (int l = 0; l < D; ++l) {
        const float m = 0.5f * (flo + fhi);
        const bool stop = !active || fhi - flo <= ftol || m <= flo || m >= fhi;
        const int c = __shfl_sync(0xffffffffu, above, lead + (q & (G - 1)));
        if (!stop) {
          if (c) fhi = m;
          else flo = m;
          q = 2 * q + (c ? 0 : 1);
        }
      }
    }
  }
  if constexpr (D == 4) {
    if (ladder && n <= TRIDIAG_FIXED_MAX) return tri_ladder(n, d, e2, flo, fhi, j, active, b);
  }
  // 2. widened bracket, checked in FP64
  const double wid = b.tnorm * 0x1p-16;
  double lo = fmax(b.lo, (double)flo - wid), hi = fmin(b.hi, (double)fhi + wid);
  double flm = 0.0, fhm = 0.0;
  int fle = 0, fhe = 0, clo = 0, chi = n;
  bool kl = false, kh = false;
  if constexpr (D == 0) {
    if (active) {
      clo = sweep64(n, d, e2, lo, flm, fle);
      chi = sweep64(n, d, e2, hi, fhm, fhe);
    }
  } else {  // even lanes the lower end, odd lanes the upper end
    double fm;
    int fe;
    const int c = sweep64(n, d, e2, (sub & 1) ? hi : lo, fm, fe);
    clo = __shfl_sync(0xffffffffu, c, lead);
    chi = __shfl_sync(0xffffffffu, c, lead + 1);
    flm = __shfl_sync(0xffffffffu, fm, lead);
    fhm = __shfl_sync(0xffffffffu, fm, lead + 1);
    fle = __shfl_sync(0xffffffffu, fe, lead);
    fhe = __shfl_sync(0xffffffffu, fe, lead + 1);
  }
  if (active) {
    kl = kh = true;
    if (clo > j || chi <= j) {  // the FP32 stage missed: full interval
      lo = b.lo;
      hi = b.hi;
      clo = 0;
      chi = n;
      kl = kh = false;
    }
  }
  // 3. FP64 regula falsi (Illinois) / bisection
  int last = 0, since = 0;
  double wref = hi - lo;
  for (int it = 0; it < 400; ++it) {
    const double tol = 2.0 * 2.220446049250313e-16 * fmax(fabs(lo), fabs(hi)) + 4.0 * b.pivmin;
    const bool done = !active || hi - lo <= tol;
    if (__all_sync(0xffffffffu, done)) break;
    if (done) continue;
    double x = 0.5 * (lo + hi);
    const bool iso = kl && kh && clo == j && chi == j + 1;  // only eigenvalue j inside
    bool bis = !iso;
    if (iso && since >= 3) {  // three interpolation steps must halve the bracket
      if (hi - lo > 0.5 * wref) {
        bis = true;
      } else {
        since = 0;
        wref = hi - lo;
      }
    }
    if (!bis) {
      const int E = max(fle, fhe);
      const double a = scalbn(flm, fle - E), c = scalbn(fhm, fhe - E);
      double xr = lo + a / (a - c) * (hi - lo);
      // a point at the converged end moves half a tolerance inside, so that the next count
      // closes the bracket instead of leaving it to bisection
      xr = fmin(fmax(xr, lo + 0.5 * tol), hi - 0.5 * tol);
      if (xr > lo && xr < hi) x = xr;
      else bis = true;
    }
    if (!(x > lo && x < hi)) {  // no representable point inside: the bracket is final
      lo = hi = x;
      continue;
    }
    if (bis) {
      since = 0;
      wref = 0.5 * (hi - lo);
    } else {
      ++since;
    }
    double fm;
    int fe;
    const int c = sweep64(n, d, e2, x, fm, fe);
    if (c > j) {
      hi = x;
      chi = c;
      fhm = fm;
      fhe = fe;
      kh = true;
      if (last == 1) flm *= 0.5;  // Illinois: the stale end's value is halved
      last = 1;
    } else {
      lo = x;
      clo = c;
      flm = fm;
      fle = fe;
      kl = true;
      if (last == -1) fhm *= 0.5;
      last = -1;
    }
  }
  return 0.5 * (lo + hi);
}

// TRI_SENTINEL stands for eigenvalues above the computed range: (e - ef)/kT >= 50 for any
// Fermi level, so their occupation is exactly zero
constexpr double TRI_SENTINEL = 1e300;

// one-molecule path, stage 0: e^2, FP32 copies and the Gershgorin data into scratch
//   ws layout: e2[n] (double), then fd[n], fe2[n] (float)
__global__ void k_tri_prep(int n, const double* __restrict__ d, const double* __restrict__ e,
                           double* ws, double* scal) {
  float* fd = reinterpret_cast<float*>(ws + n);
  float* fe2 = fd + n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double ee = i < n - 1 ? e[i] * e[i] : 0.0;
    ws[i] = ee;
    fd[i] = (float)d[i];
    fe2[i] = (float)ee;
  }
  if (blockIdx.x == 0) {
    const TriBounds b = tri_bounds(n, d, e);
    if (threadIdx.x == 0) {
      scal[1] = b.tnorm;  // |T| estimate for the inverse iteration
      scal[2] = b.lo;
      scal[3] = b.hi;
      scal[4] = b.pivmin;
    }
  }
}
// one-molecule path: eigenvalues j0 <= j < j1; with fill, w[j1 .. n) = TRI_SENTINEL.  One warp per
// block (the warps of a single molecule spread over as many SMs as possible), 16 lanes per
// eigenvalue: 2 warps per SM at 600 eigenvalues, so the extra FP32 counts cost no time
constexpr int EIG_D = 4;
// fill: bit 0 mark the eigenvalues not computed, bit 1 the order of large molecules (no ladder)
__global__ void __launch_bounds__(32) k_eigvals(int n, int j0, int j1, int fill,
                                                 const double* __restrict__ d,
                                                 const double* __restrict__ ws,
                                                 const double* __restrict__ scal, double* w) {
  const int j = j0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> EIG_D);
  const float* fd = reinterpret_cast<const float*>(ws + n);
  const float* fe2 = fd + n;
  if (j0 + (int)((blockIdx.x * blockDim.x) >> EIG_D) >= j1) {  // a warp of unwanted eigenvalues
    if ((fill & 1) && (threadIdx.x & ((1 << EIG_D) - 1)) == 0 && j < n) w[j] = TRI_SENTINEL;
    return;
  }
  TriBounds b;
  b.tnorm = scal[1];
  b.lo = scal[2];
  b.hi = scal[3];
  b.pivmin = scal[4];
  const bool active = j < j1;
  const double v = tri_eigenvalue<EIG_D>(n, d, ws, fd, fe2, j, active, b, !(fill & 2));
  if ((threadIdx.x & ((1 << EIG_D) - 1)) != 0) return;
  if (active) w[j] = v;
  else if ((fill & 1) && j < n) w[j] = TRI_SENTINEL;
}

// ------------------------------------------------------------------------------------------
// inverse iteration: one thread per eigenvector (column j < k), Gaussian elimination with
// partial pivoting of the tridiagonal T - w_j I, two solves from a pseudo-random start.
//
// Bound by the chain of FP64 instructions of one warp (64-71 cycles each, whatever the active
// lanes): about 25 per row, six of them the division.  So the two pivot cases share one division
// and one update by selecting operands, comparisons read the bit patterns, the reciprocals of the
// pivots are formed once, the second superdiagonal is read back from e (it is e[r + 1] where rows
// were interchanged, else 0), and the rows move through registers in blocks of 8, the next block's
// loads issued before the current block's chain.  Scratch rows are contiguous over the warp's
// vectors ([row][vector]); the finished columns go to Y (column-major [j][n]) through a
// shared-memory transpose.  C200H402 (1202 rows, 601 vectors) 4.45 -> 1.89 ms, 192 rows and 96
// vectors 540 -> 290 us, with the same bits.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ double hash_uniform(unsigned a, unsigned b) {
  unsigned h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u) * 0x85EBCA77u;
  h ^= h >> 15;
  h *= 0x2C1B3C6Du;
  h ^= h >> 12;
  h *= 0x297A2D39u;
  h ^= h >> 15;
  return (double)(int)(h ^ 0x80000000u) * 0x1p-31;  // 2 h / 2^32 - 1, exactly
}

constexpr int INV_B = 8;       // rows in registers
constexpr int INV_WARP = 32;   // threads of a block
__device__ __forceinline__ void invit_dev(int n, int k0, int k, const double* __restrict__ d,
                        const double* __restrict__ e, const double* __restrict__ w,
                        const double* __restrict__ scal, double* lu, double* Y) {
  __shared__ double tile[32][33];
  if ((int)(blockIdx.x * blockDim.x) >= k) return;
  const int lane = threadIdx.x;
  const int jb = blockIdx.x * blockDim.x;
  const int j = min(jb + lane, k - 1);  // vector k0 + j; idle lanes repeat the last one
  const bool mine = jb + lane < k;
  const size_t nk = (size_t)n * k;
  double* __restrict__ U1 = lu + j;           // first superdiagonal
  double* __restrict__ R0 = lu + nk + j;      // 1 / pivot
  double* __restrict__ Lm = lu + 2 * nk + j;  // multiplier
  double* __restrict__ Yt = lu + 3 * nk + j;  // the vector
  unsigned* PV = reinterpret_cast<unsigned*>(lu + 4 * nk) + j;  // interchange bits of 32 rows
  const double lam = w[k0 + j];
  const double tnorm = scal[1] > 0 ? scal[1] : 1.0;
  const double tiny = 2.220446049250313e-16 * tnorm;
  auto absbits = [](double x) {
    return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
  };
  const unsigned long long btiny = absbits(tiny);
  // factorise T - lam I
  double u0 = d[0] - lam, u1 = n > 1 ? e[0] : 0.0;
  unsigned bits = 0u;
  double ec = u1;  // e[r]
  for (int r = 0; r < n - 1; ++r) {
    const double c = ec;                                    // sub-diagonal of row r+1
    const double a1 = d[r + 1] - lam, b1 = r + 1 < n - 1 ? e[r + 1] : 0.0;
    const bool keep = absbits(u0) >= absbits(c);
    if (keep && absbits(u0) < btiny) u0 = copysign(tiny, u0 == 0.0 ? 1.0 : u0);
    const double piv = keep ? u0 : c;
    const double l = (keep ? c : u0) / piv;
    if (mine) {
      U1[(size_t)r * k] = keep ? u1 : a1;
      R0[(size_t)r * k] = frcp(piv);
      Lm[(size_t)r * k] = l;
    }
    if (!keep) bits |= 1u << (r & 31);
    if ((r & 31) == 31) {
      if (mine) PV[(size_t)(r >> 5) * k] = bits;
      bits = 0u;
    }
    // kept: u0' = a1 - l u1, u1' = b1; interchanged: u0' = u1 - l a1, u1' = -l b1
    u0 = fma(-l, keep ? u1 : a1, keep ? a1 : u1);
    u1 = keep ? b1 : -l * b1;
    ec = b1;
  }
  if (mine) PV[(size_t)((n - 1) >> 5) * k] = bits;
  if (absbits(u0) < btiny) u0 = copysign(tiny, u0 == 0.0 ? 1.0 : u0);
  const double rlast = frcp(u0);
  double scale = 1.0;
  for (int iter = 0; iter < 2; ++iter) {
    // forward: apply row operations to the right-hand side (start vector, or the scaled result of
    // the first solve)
    double cur = iter ? Yt[0] * scale : hash_uniform(k0 + j + 1, 1);
    double yn[INV_B], ln[INV_B];
#pragma unroll
    for (int t = 0; t < INV_B; ++t) {
      const int r = min(t, n - 2);
      if (n > 1) {
        ln[t] = Lm[(size_t)r * k];
        if (iter) yn[t] = Yt[(size_t)(r + 1) * k];
      }
    }
    for (int r0 = 0; r0 < n - 1; r0 += INV_B) {
      double yv[INV_B], lv[INV_B];
#pragma unroll
      for (int t = 0; t < INV_B; ++t) {
        yv[t] = iter ? yn[t] * scale : hash_uniform(k0 + j + 1, r0 + t + 2);
        lv[t] = ln[t];
      }
      const unsigned pv = PV[(size_t)(r0 >> 5) * k] >> (r0 & 31);
#pragma unroll
      for (int t = 0; t < INV_B; ++t) {  // next block
        const int r = min(r0 + INV_B + t, n - 2);
        ln[t] = Lm[(size_t)r * k];
        if (iter) yn[t] = Yt[(size_t)(r + 1) * k];
      }
#pragma unroll
      for (int t = 0; t < INV_B; ++t)
        if (r0 + t < n - 1) {
          const bool sw = (pv >> t) & 1u;
          const double p = sw ? yv[t] : cur, q = sw ? cur : yv[t];
          if (mine) Yt[(size_t)(r0 + t) * k] = p;
          cur = fma(-lv[t], p, q);
        }
    }
    if (mine) Yt[(size_t)(n - 1) * k] = cur;
    // backward: U x = y
    double x1 = cur * rlast, x2 = 0.0;
    if (mine) Yt[(size_t)(n - 1) * k] = x1;
    double rn[INV_B], un[INV_B];
#pragma unroll
    for (int t = 0; t < INV_B; ++t) {
      const size_t r = (size_t)max(n - 2 - t, 0) * k;
      yn[t] = Yt[r];
      un[t] = U1[r];
      rn[t] = R0[r];
    }
    for (int r0 = n - 2; r0 >= 0; r0 -= INV_B) {  // rows r0, r0 - 1, ..
      double yv[INV_B], uv[INV_B], rv[INV_B], ev[INV_B];
      unsigned pv = 0u;
#pragma unroll
      for (int t = 0; t < INV_B; ++t) {
        const int r = max(r0 - t, 0);
        yv[t] = yn[t];
        uv[t] = un[t];
        rv[t] = rn[t];
        ev[t] = r + 1 < n - 1 ? e[r + 1] : 0.0;
      }
      {
        const int rl = max(r0 - INV_B + 1, 0);
        const unsigned wl = PV[(size_t)(rl >> 5) * k], wh = PV[(size_t)(r0 >> 5) * k];
        pv = __funnelshift_r(wl, (r0 >> 5) == (rl >> 5) ? 0u : wh, rl & 31) << (INV_B - 1 - (r0 - rl));
      }  // bit INV_B - 1 - t: row r0 - t
#pragma unroll
      for (int t = 0; t < INV_B; ++t) {  // next block
        const size_t r = (size_t)max(r0 - INV_B - t, 0) * k;
        yn[t] = Yt[r];
        un[t] = U1[r];
        rn[t] = R0[r];
      }
      const bool any = __any_sync(0xffffffffu, (pv & ((1u << INV_B) - 1)) != 0u);
#pragma unroll
      for (int t = 0; t < INV_B; ++t)
        if (r0 - t >= 0) {
          double v = fma(-uv[t], x1, yv[t]);
          if (any) v = fma(-(((pv >> (INV_B - 1 - t)) & 1u) ? ev[t] : 0.0), x2, v);
          v *= rv[t];
          if (mine) Yt[(size_t)(r0 - t) * k] = v;
          x2 = x1;
          x1 = v;
        }
    }
    double nrm = 0.0;
    {
#pragma unroll
      for (int t = 0; t < INV_B; ++t) yn[t] = Yt[(size_t)min(t, n - 1) * k];
      for (int r0 = 0; r0 < n; r0 += INV_B) {
        double yv[INV_B];
#pragma unroll
        for (int t = 0; t < INV_B; ++t) {
          yv[t] = yn[t];
          yn[t] = Yt[(size_t)min(r0 + INV_B + t, n - 1) * k];
        }
#pragma unroll
        for (int t = 0; t < INV_B; ++t)
          if (r0 + t < n) nrm += yv[t] * yv[t];
      }
    }
    scale = 1.0 / sqrt(nrm);
  }
  // Y[k0 + j][r], 32 rows at a time
  const int cols = min(32, k - jb);
  for (int r0 = 0; r0 < n; r0 += 32) {
    __syncwarp();
#pragma unroll 8
    for (int t = 0; t < 32; ++t)
      if (r0 + t < n) tile[t][lane] = Yt[(size_t)(r0 + t) * k] * scale;
    __syncwarp();
    if (r0 + lane < n)
#pragma unroll 8
      for (int t = 0; t < cols; ++t)
        Y[(size_t)(k0 + jb + t) * n + r0 + lane] = tile[lane][t];
  }
}
__global__ void __launch_bounds__(INV_WARP) k_invit(int n, int k0, int k,
                        const double* __restrict__ d, const double* __restrict__ e,
                        const double* __restrict__ w, const double* __restrict__ scal, double* lu,
                        double* Y) {
  invit_dev(n, k0, k, d, e, w, scal, lu, Y);
}

// Clusters of close eigenvalues (gap < tol |T|): modified Gram-Schmidt, then Rayleigh-Ritz
// with T inside the cluster (Jacobi on the small projected matrix).  One block per cluster
// start; vectors of a cluster are consecutive columns of Y.
constexpr int MAXCL = 32;
__device__ __forceinline__ void clusters_dev(int n, int k0, int k, const double* __restrict__ d,
                           const double* __restrict__ e, const double* __restrict__ w,
                           const double* __restrict__ scal, double tolrel, double* Y) {
  const int j0 = k0 + blockIdx.x;  // clusters are looked for among vectors k0 .. k-1
  if (j0 >= k) return;
  const double tol = tolrel * (scal[1] > 0 ? scal[1] : 1.0);
  if (j0 > k0 && w[j0] - w[j0 - 1] < tol) return;  // not a cluster start
  int c = 1;
  while (j0 + c < k && w[j0 + c] - w[j0 + c - 1] < tol) ++c;
  if (c == 1) return;
  __shared__ double red[32];
  __shared__ double H[MAXCL][MAXCL], V[MAXCL][MAXCL];
  auto bsum = [&](double v) {
    v = wred(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x < 32) {
      t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
      t = wred(t);
      if (threadIdx.x == 0) red[0] = t;
    }
    __syncthreads();
    t = red[0];
    __syncthreads();
    return t;
  };
  // MGS
  for (int a = 0; a < c; ++a) {
    double* ya = Y + (size_t)(j0 + a) * n;
    for (int b = 0; b < a; ++b) {
      const double* yb = Y + (size_t)(j0 + b) * n;
      double s = 0.0;
      for (int r = threadIdx.x; r < n; r += blockDim.x) s += ya[r] * yb[r];
      s = bsum(s);
      for (int r = threadIdx.x; r < n; r += blockDim.x) ya[r] -= s * yb[r];
      __syncthreads();
    }
    double s = 0.0;
    for (int r = threadIdx.x; r < n; r += blockDim.x) s += ya[r] * ya[r];
    s = 1.0 / sqrt(bsum(s));
    for (int r = threadIdx.x; r < n; r += blockDim.x) ya[r] *= s;
    __syncthreads();
  }
  if (c > MAXCL) return;
  // H = Y_c^T T Y_c
  for (int a = 0; a < c; ++a)
    for (int b = a; b < c; ++b) {
      const double* ya = Y + (size_t)(j0 + a) * n;
      const double* yb = Y + (size_t)(j0 + b) * n;
      double s = 0.0;
      for (int r = threadIdx.x; r < n; r += blockDim.x) {
        double ty = d[r] * yb[r];
        if (r > 0) ty += e[r - 1] * yb[r - 1];
        if (r < n - 1) ty += e[r] * yb[r + 1];
        s += ya[r] * ty;
      }
      s = bsum(s);
      if (threadIdx.x == 0) {
        H[a][b] = s;
        H[b][a] = s;
      }
    }
  __syncthreads();
  // cyclic Jacobi on H (thread 0), V accumulates rotations
  if (threadIdx.x == 0) {
    for (int a = 0; a < c; ++a)
      for (int b = 0; b < c; ++b) V[a][b] = a == b ? 1.0 : 0.0;
    for (int sweep = 0; sweep < 30; ++sweep) {
      double off = 0.0;
      for (int a = 0; a < c; ++a)
        for (int b = a + 1; b < c; ++b) off += H[a][b] * H[a][b];
      if (off < 1e-60) break;
      for (int p = 0; p < c; ++p)
        for (int q = p + 1; q < c; ++q) {
          if (H[p][q] == 0.0) continue;
          const double th = (H[q][q] - H[p][p]) / (2.0 * H[p][q]);
          const double t = copysign(1.0, th) / (fabs(th) + sqrt(th * th + 1.0));
          const double cs = 1.0 / sqrt(t * t + 1.0), sn = t * cs;
          for (int r = 0; r < c; ++r) {
            const double hp = H[r][p], hq = H[r][q];
            H[r][p] = cs * hp - sn * hq;
            H[r][q] = sn * hp + cs * hq;
          }
          for (int r = 0; r < c; ++r) {
            const double hp = H[p][r], hq = H[q][r];
            H[p][r] = cs * hp - sn * hq;
            H[q][r] = sn * hp + cs * hq;
          }
          for (int r = 0; r < c; ++r) {
            const double vp = V[r][p], vq = V[r][q];
            V[r][p] = cs * vp - sn * vq;
            V[r][q] = sn * vp + cs * vq;
          }
        }
    }
    // sort by Ritz value (ascending) -- columns of V
    for (int a = 0; a < c; ++a) {
      int mn = a;
      for (int b = a + 1; b < c; ++b)
        if (H[b][b] < H[mn][mn]) mn = b;
      if (mn != a) {
        const double t = H[a][a];
        H[a][a] = H[mn][mn];
        H[mn][mn] = t;
        for (int r = 0; r < c; ++r) {
          const double v = V[r][a];
          V[r][a] = V[r][mn];
          V[r][mn] = v;
        }
      }
    }
  }
  __syncthreads();
  // Y_c <- Y_c V (row by row through registers)
  for (int r = threadIdx.x; r < n; r += blockDim.x) {
    double row[MAXCL];
    for (int a = 0; a < c; ++a) row[a] = Y[(size_t)(j0 + a) * n + r];
    for (int b = 0; b < c; ++b) {
      double s = 0.0;
      for (int a = 0; a < c; ++a) s += row[a] * V[a][b];
      Y[(size_t)(j0 + b) * n + r] = s;
    }
  }
}
__global__ void k_clusters(int n, int k0, int k, const double* __restrict__ d,
                           const double* __restrict__ e, const double* __restrict__ w,
                           const double* __restrict__ scal, double tolrel, double* Y) {
  clusters_dev(n, k0, k, d, e, w, scal, tolrel, Y);
}

// ------------------------------------------------------------------------------------------
// back-transformation Z = Q Y = H_0 H_1 ... H_{n-2} Y  (apply H_{n-2} first).  Each block owns
// a set of columns (one warp per column); reflectors are staged in shared memory in chunks.
// ------------------------------------------------------------------------------------------
// Back-transformation Z = Q Y of the eigenvectors of T.  The reflectors are taken in blocks of
// four, [4g, 4g+3], from the top block down, each block as one compact-WY update
//     y <- y - V (T (V^T y))      (V = the block's four reflectors, T upper triangular 4 x 4)
// so that a column makes one pass for the four dot products and one for the update, and the
// four warp reductions are independent.  T (LAPACK dlarft, forward, column-wise) is formed
// once per block by k_bt_tmat.  One warp per column; the block's reflectors are staged in
// shared memory (zero above each reflector's first row), the column too when it fits.
// warps (columns) per block: 4 on the one-molecule path (more blocks for small k), 8 in the batch
// (the reflectors staged per block serve twice the columns; measured 2131 -> 2104 ms on the
// 4096-molecule ensemble, while 8 slowed the 192-orbital single point)
constexpr int BT_WARPS = 4, BT_WARPS_B = 8;
constexpr int BT_CHUNK_MAX = 16;  // reflectors staged per round (a multiple of 4)
constexpr size_t BT_SMEM_MAX = 200 * 1024;
// the columns live in shared memory too when at least one block of reflectors fits beside them
__host__ __device__ static inline bool bt_ysmem(int n, int w = BT_WARPS) {
  return (int)(BT_SMEM_MAX / (sizeof(double) * (size_t)n)) - w >= 4;
}
__host__ __device__ static inline int bt_chunk(int n, int w = BT_WARPS) {
  int c = (int)(BT_SMEM_MAX / (sizeof(double) * (size_t)n)) - (bt_ysmem(n, w) ? w : 0);
  c = c < 4 ? 4 : (c > BT_CHUNK_MAX ? BT_CHUNK_MAX : c);
  return c & ~3;
}
__host__ __device__ static inline size_t bt_smem(int n, int w = BT_WARPS) {
  return sizeof(double) * (size_t)n * (bt_chunk(n, w) + (bt_ysmem(n, w) ? w : 0));
}
// reflector j: v[j+1] = 1, v[r] = A[r + j n] for r > j+1; j > n-2 does not exist (zero)
__device__ __forceinline__ double bt_v(int n, const double* __restrict__ A, int j, int r) {
  if (j > n - 2 || r <= j) return 0.0;
  return r == j + 1 ? 1.0 : A[r + (size_t)j * n];
}
// T of block g (reflectors 4g .. 4g+3), one warp: Tm[16 g + a + 4 b], upper triangular
__device__ __forceinline__ void bt_tmat_dev(int n, const double* __restrict__ A,
                                            const double* __restrict__ tau, double* Tm, int g,
                                            int lane) {
  const int j0 = 4 * g;
  double dd[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) dd[a][b] = 0.0;
#pragma unroll
  for (int b = 1; b < 4; ++b) {
    const int rb = j0 + b + 1;  // first row of reflector b (v = 1 there)
#pragma unroll
    for (int a = 0; a < b; ++a) {
      double acc = 0.0;
      for (int r = rb + lane; r < n; r += 32) acc += bt_v(n, A, j0 + a, r) * bt_v(n, A, j0 + b, r);
      dd[a][b] = wred(acc);
    }
  }
  if (lane != 0) return;
  double t[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int j = j0 + a;
#pragma unroll
    for (int b = 0; b < 4; ++b) t[a][b] = 0.0;
    t[a][a] = j <= n - 2 ? tau[j] : 0.0;
  }
#pragma unroll
  for (int b = 1; b < 4; ++b)
#pragma unroll
    for (int a = 0; a < b; ++a) {
      double acc = 0.0;
#pragma unroll
      for (int c = a; c < b; ++c) acc += t[a][c] * dd[c][b];
      t[a][b] = -t[b][b] * acc;
    }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) Tm[16 * g + a + 4 * b] = t[a][b];
}
__global__ void k_bt_tmat(int n, const double* __restrict__ A, const double* __restrict__ tau,
                          double* Tm) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (g * 4 > n - 2) return;
  bt_tmat_dev(n, A, tau, Tm, g, threadIdx.x & 31);
}

template <int W>
__device__ __forceinline__ void backtransform_dev(int n, int k, int chunk, bool ysmem,
                                                  const double* __restrict__ A,
                                                  const double* __restrict__ Tm, double* Y) {
  extern __shared__ double smem[];  // [chunk][n] reflectors, then [W][n] columns
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int col = blockIdx.x * W + wid;
  double* yg = col < k ? Y + (size_t)col * n : nullptr;
  double* y = !yg ? nullptr : (ysmem ? smem + (size_t)chunk * n + (size_t)wid * n : yg);
  if (y && ysmem)
    for (int r = lane; r < n; r += 32) y[r] = yg[r];
  const int cb = chunk / 4;  // blocks per round
  for (int gtop = (n - 2) / 4; gtop >= 0; gtop -= cb) {
    const int gbot = max(0, gtop - cb + 1);
    __syncthreads();
    // a warp per reflector: its rows are in flight together (one after the other per thread they
    // took as long as the arithmetic)
    for (int q = wid; q < 4 * (gtop - gbot + 1); q += W) {
      const int j = 4 * (gtop - (q >> 2)) + (q & 3);
      double* sv = smem + (size_t)q * n;
#pragma unroll 8
      for (int r = (j & ~3) + 1 + lane; r < n; r += 32) sv[r] = bt_v(n, A, j, r);
    }
    __syncthreads();
    if (y) {
      for (int g = gtop; g >= gbot; --g) {
        const double* v0 = smem + (size_t)((gtop - g) * 4) * n;
        const double* v1 = v0 + n;
        const double* v2 = v1 + n;
        const double* v3 = v2 + n;
        double w[4] = {0.0, 0.0, 0.0, 0.0};
        // z = T w (upper triangular, column-major): row b on lane b, from its diagonal on, four
        // operations for all rows
        const int b = lane & 3;
        const double* T = Tm + 16 * g + 5 * b;
        const double t0 = T[0], t1 = b < 3 ? T[4] : 0.0, t2 = b < 2 ? T[8] : 0.0,
                     t3 = b < 1 ? T[12] : 0.0;
        for (int r = 4 * g + 1 + lane; r < n; r += 32) {
          const double yr = y[r];
          w[0] = fma(v0[r], yr, w[0]);
          w[1] = fma(v1[r], yr, w[1]);
          w[2] = fma(v2[r], yr, w[2]);
          w[3] = fma(v3[r], yr, w[3]);
        }
        const double s = warp_sums4(w);  // six additions instead of twenty
        const double x0 = warp_sum4_of(s, b), x1 = warp_sum4_of(s, b + 1),
                     x2 = warp_sum4_of(s, b + 2), x3 = warp_sum4_of(s, b + 3);
        const double zb = fma(t3, x3, fma(t2, x2, fma(t0, x0, __dmul_rn(t1, x1))));
        const double z0 = __shfl_sync(0xffffffffu, zb, 0), z1 = __shfl_sync(0xffffffffu, zb, 1);
        const double z2 = __shfl_sync(0xffffffffu, zb, 2), z3 = __shfl_sync(0xffffffffu, zb, 3);
        for (int r = 4 * g + 1 + lane; r < n; r += 32)
          y[r] -= fma(v0[r], z0, fma(v1[r], z1, fma(v2[r], z2, v3[r] * z3)));
        __syncwarp();
      }
    }
  }
  if (y && ysmem)
    for (int r = lane; r < n; r += 32) yg[r] = y[r];
}
__global__ void __launch_bounds__(BT_WARPS * 32) k_backtransform(int n, int k, int chunk, bool ysmem,
                                                                 const double* __restrict__ A,
                                                                 const double* __restrict__ Tm,
                                                                 double* Y) {
  backtransform_dev<BT_WARPS>(n, k, chunk, ysmem, A, Tm, Y);
}

// ------------------------------------------------------------------------------------------
EigenSolver* eigen_create(int n, cudaStream_t s) {
  auto* e = new EigenSolver();
  e->n = n;
  e->cap = n;
  e->stream = s;
  const size_t nn = (size_t)n * n;
  ck(cudaMalloc(&e->L, sizeof(double) * nn), "L");
  ck(cudaMalloc(&e->X, sizeof(double) * nn), "X");
  ck(cudaMalloc(&e->A, sizeof(double) * nn), "A");
  ck(cudaMalloc(&e->T1, sizeof(double) * nn), "T1");
  ck(cudaMalloc(&e->Y, sizeof(double) * nn), "Y");
  ck(cudaMalloc(&e->lu, sizeof(double) * 5 * nn), "lu");
  ck(cudaMalloc(&e->d, sizeof(double) * (n + 1)), "d");
  ck(cudaMalloc(&e->e, sizeof(double) * (n + 1)), "e");
  ck(cudaMalloc(&e->tau, sizeof(double) * (n + 1)), "tau");
  ck(cudaMalloc(&e->w, sizeof(double) * (n + 1)), "w");
  ck(cudaMalloc(&e->pv, sizeof(double) * 6 * (n + 1)), "pv");
  ck(cudaMalloc(&e->tw, sizeof(double) * 2 * (n + 1)), "tw");
  ck(cudaMalloc(&e->xch, sizeof(long long) * tridiag_exchange_words(n)), "xch");
  ck(cudaMalloc(&e->scal, sizeof(double) * 8), "scal");
  ck(cudaMalloc(&e->status, sizeof(int)), "status");
  if (n >= 128) ck(cudaMalloc(&e->pair, pair_work_bytes(std::min(n, PAIR_MAX))), "pair");
  ck(cudaMalloc(&e->gstatus, sizeof(int)), "gstatus");
  ck(cudaMemsetAsync(e->gstatus, 0, sizeof(int), s), "gstatus");
  ck(cudaMallocHost(&e->hstatus, sizeof(int)), "hstatus");
  int dev = 0, nsm = 0, per_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tridiag, 256, 0);
  (void)per_sm;
  e->coop_blocks = nsm;  // one block per SM keeps the grid barrier cheap
  // shared memory of the back-transformation
  ck(cudaFuncSetAttribute(k_tridiag_smem, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)TRIDIAG_SMEM_MAX),
     "smem attr tridiag");
  ck(cudaFuncSetAttribute(k_backtransform, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)BT_SMEM_MAX + (int)(BT_WARPS * sizeof(double) * 64)),
     "smem attr");
  return e;
}

void eigen_destroy(EigenSolver* e) {
  if (!e) return;
  for (double* p : {e->L, e->X, e->A, e->T1, e->Y, e->lu, e->d, e->e, e->tau, e->w, e->pv, e->tw,
                    e->scal})
    cudaFree(p);
  cudaFree(e->xch);
  cudaFree(e->status);
  cudaFree(e->gstatus);
  cudaFree(e->pair);
  cudaFreeHost(e->hstatus);
  delete e;
}

int cholesky_inverse(int n, double* L, double* X, int* d_status, int* h_status, cudaStream_t s);

int eigen_set_overlap(EigenSolver* e, const double* S) {
  const int n = e->n;
  // a new geometry: the tensor-core status word starts clear
  ck(cudaMemsetAsync(e->gstatus, 0, sizeof(int), e->stream), "gstatus");
  if (!e->ordered && cholinv_fixed(n, S, e->X, e->status, e->stream)) {
    ck(cudaMemcpyAsync(e->hstatus, e->status, sizeof(int), cudaMemcpyDeviceToHost, e->stream),
       "Cholesky status");
    stream_wait(e->stream);
    if (*e->hstatus == 0) return 0;  // else outside the fixed-point range: in FP64
  }
  ck(cudaMemcpyAsync(e->L, S, sizeof(double) * (size_t)n * n, cudaMemcpyDeviceToDevice, e->stream),
     "copy S");
  return cholesky_inverse(n, e->L, e->X, e->status, e->hstatus, e->stream);
}

int eigen_values(EigenSolver* es, const double* F, double* w_out, int nev) {
  const int n = es->n;
  cudaStream_t s = es->stream;
  // A = X^T (F X): X upper triangular
  if (split_gemm(n)) {  // BF16 tensor cores, FP64-accurate splitting (exponents in tw)
    if (pair_gemm(n, eigen_gemm_pair(es))) {
      pgemm_pair(n, false, false, n, n, n, F, n, es->X, n, es->T1, n, false, es->pair, es->gstatus,
                 s);
      pgemm_pair(n, true, false, n, n, n, es->X, n, es->T1, n, es->A, n, true, es->pair,
                 es->gstatus, s);
    } else {
      int* ex = reinterpret_cast<int*>(es->tw);
      ogemm(false, false, n, n, n, F, es->X, es->T1, n, KM_LT_COLEND, ex, es->gstatus, s);
      ogemm(true, false, n, n, n, es->X, es->T1, es->A, n, KM_LT_ROWEND | KM_SYM, ex, es->gstatus,
            s);
    }
  } else {
    gemm64(false, false, n, n, n, 1.0, F, n, es->X, n, 0.0, es->T1, n, KM_LT_COLEND, s);
    gemm64(true, false, n, n, n, 1.0, es->X, n, es->T1, n, 0.0, es->A, n, KM_LT_ROWEND | KM_SYM, s);
  }
  // tridiagonalise
  {
    const int tk = prof_kbegin(s);
    if (n <= TRIDIAG_FIXED_MAX && !es->ordered) {
      tridiag_fixed(n, es->A, es->d, es->e, es->tau, es->xch, s);
    } else {
      int nn = n, blocks = std::min(es->coop_blocks, (n * 32 + 255) / 256);
      // shared-memory resident while every block can hold its columns
      const size_t smem = sizeof(double) * tridiag_smem_doubles(n, blocks);
      ++g_kernel_launches;
      if (smem <= TRIDIAG_SMEM_MAX && n <= 256 * TRIDIAG_ROWS) {
        void* args[] = {&nn, &es->A, &es->d, &es->e, &es->tau, &es->pv};
        ck(cudaLaunchCooperativeKernel((void*)k_tridiag_smem, blocks, 256, args, smem, s),
           "tridiag_smem");
      } else {
        void* args[] = {&nn, &es->A, &es->d, &es->e, &es->tau, &es->pv, &es->scal};
        ck(cudaLaunchCooperativeKernel((void*)k_tridiag, blocks, 256, args, 0, s), "tridiag");
      }
    }
    prof_kend(KS_TRIDIAG, tk, s);
  }
  if (nev <= 0 || nev > n) nev = n;
  g_kernel_launches += 2;
  const int tm = prof_kbegin(s);
  k_tri_prep<<<(n + 255) / 256, 256, 0, s>>>(n, es->d, es->e, es->tw, es->scal);
  k_eigvals<<<((n << EIG_D) + 31) / 32, 32, 0, s>>>(n, 0, nev, es->ordered ? 3 : 1, es->d,
                                                             es->tw, es->scal, es->w);
  prof_kend(KS_MULTISECT, tm, s);
  ck(cudaMemcpyAsync(w_out, es->w, sizeof(double) * n, cudaMemcpyDeviceToDevice, s), "w");
  return 0;
}

void eigen_values_rest(EigenSolver* es, int nev, double* w_out) {
  const int n = es->n;
  if (nev >= n) return;
  cudaStream_t s = es->stream;
  g_kernel_launches += 2;
  const int tm = prof_kbegin(s);
  k_tri_prep<<<(n + 255) / 256, 256, 0, s>>>(n, es->d, es->e, es->tw, es->scal);
  k_eigvals<<<(((n - nev) << EIG_D) + 31) / 32, 32, 0, s>>>(n, nev, n, es->ordered ? 2 : 0,
                                                                     es->d, es->tw, es->scal, es->w);
  prof_kend(KS_MULTISECT, tm, s);
  ck(cudaMemcpyAsync(w_out + nev, es->w + nev, sizeof(double) * (n - nev), cudaMemcpyDeviceToDevice, s),
     "w");
}

void eigen_vectors_range(EigenSolver* es, int k0, int k1, double* C) {
  const int n = es->n;
  cudaStream_t s = es->stream;
  const int k = k1 - k0;
  if (k <= 0) return;
  ++g_kernel_launches;
  const int ti = prof_kbegin(s);
  k_invit<<<(k + INV_WARP - 1) / INV_WARP, INV_WARP, 0, s>>>(n, k0, k, es->d, es->e, es->w, es->scal, es->lu, es->Y);
  prof_kend(KS_INVIT, ti, s);
  ++g_kernel_launches;
  k_clusters<<<k, 256, 0, s>>>(n, k0, k1, es->d, es->e, es->w, es->scal, 1e-5, es->Y);
  const int chunk = bt_chunk(n);
  double* Yk = es->Y + (size_t)k0 * n;
  ++g_kernel_launches;
  const int tb_ = prof_kbegin(s);
  ++g_kernel_launches;  // T of the blocks of four reflectors, into lu (free after the solves)
  k_bt_tmat<<<(((n - 2) / 4 + 1) * 32 + 127) / 128, 128, 0, s>>>(n, es->A, es->tau, es->lu);
  k_backtransform<<<(k + BT_WARPS - 1) / BT_WARPS, BT_WARPS * 32, bt_smem(n), s>>>(
      n, k, chunk, bt_ysmem(n), es->A, es->lu, Yk);
  prof_kend(KS_BACKTRANSFORM, tb_, s);
  // C = X Y (X upper triangular)
  if (pair_gemm(n, eigen_gemm_pair(es)))
    pgemm_pair(n, false, false, n, k, n, es->X, n, Yk, n, C + (size_t)k0 * n, n, false, es->pair,
               es->gstatus, s);
  else if (split_gemm(n))
    ogemm(false, false, n, k, n, es->X, Yk, C + (size_t)k0 * n, n, KM_GE_ROWBEG,
          reinterpret_cast<int*>(es->tw), es->gstatus, s);
  else
    gemm64(false, false, n, k, n, 1.0, es->X, n, Yk, n, 0.0, C + (size_t)k0 * n, n, KM_GE_ROWBEG,
           s);
}

void eigen_vectors(EigenSolver* es, int k, double* C) { eigen_vectors_range(es, 0, k, C); }

// P = sum_{m<k} f_m C_m C_m^T: scale columns into work, then one GEMM
__device__ __forceinline__ void scale_cols_dev(int n, int k, const double* C, const double* f, double* out) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (t >= (size_t)n * k) return;
  out[t] = C[t] * f[t / n];
}
__global__ void k_scale_cols(int n, int k, const double* C, const double* f, double* out) {
  scale_cols_dev(n, k, C, f, out);
}

void density_matrix(int n, int k, const double* C, const double* f, double* P, double* work,
                    cudaStream_t s, int* status, void* pair) {
  if (k <= 0) {
    cudaMemsetAsync(P, 0, sizeof(double) * (size_t)n * n, s);
    return;
  }
  const size_t tot = (size_t)n * k;
  ++g_kernel_launches;
  k_scale_cols<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(n, k, C, f, work);
  // the split GEMM keeps its 2n exponents behind the scaled columns (needs k < n)
  if (status && pair_gemm(n, pair) && k < n)
    pgemm_pair(n, false, true, n, n, k, work, n, C, n, P, n, true, pair, status, s);
  else if (status && split_gemm(n) && k < n)
    ogemm(false, true, n, n, k, work, C, P, n, KM_NONE | KM_SYM,
          reinterpret_cast<int*>(work + tot), status, s);
  else
    gemm64(false, true, n, n, k, 1.0, work, n, C, n, 0.0, P, n, KM_NONE | KM_SYM, s);
}

int* eigen_gemm_status(EigenSolver* es) { return es->gstatus; }
void* eigen_gemm_pair(EigenSolver* es) {
  return es->pair_on && !es->ordered ? es->pair : nullptr;
}
void eigen_set_ordered(EigenSolver* es, bool ordered) { es->ordered = ordered; }
void eigen_set_pair(EigenSolver* es, bool on) { es->pair_on = on; }
bool eigen_pair_failed(EigenSolver* es) {
  int h = 0;
  return pair_gemm(es->n, eigen_gemm_pair(es)) &&
         cudaMemcpyAsync(&h, es->gstatus, sizeof(int), cudaMemcpyDeviceToHost, es->stream) ==
             cudaSuccess &&
         cudaStreamSynchronize(es->stream) == cudaSuccess && h != 0;
}
bool eigen_gemm_failed(EigenSolver* es) {
  int h = 0;
  ck(cudaMemcpyAsync(&h, es->gstatus, sizeof(int), cudaMemcpyDeviceToHost, es->stream), "gstatus");
  stream_wait(es->stream);
  return h != 0;
}

// ------------------------------------------------------------------------------------------
// Batched eigensolver: blockIdx.z over molecules (the tridiagonalisation in tridiag.cu: one CTA or
// thread-block cluster per molecule).  The eigenvalues
// are written straight into emo; icount (from the Fermi filling) bounds the vectors.
// ------------------------------------------------------------------------------------------
#define BMOL const MolPtrs& q = mp[list[blockIdx.z]]
#define BARGS const MolPtrs* __restrict__ mp, const int* __restrict__ list

// Eigenvalues for the batch, one thread per eigenvalue (tri_eigenvalue: FP32 bisection, FP64
// check, FP64 Illinois / bisection).  d, e^2 and their FP32 copies are staged in shared memory
// (every thread reads the same element at the same step).  rest = 0: eigenvalues j < nev and
// the sentinel above them; rest = 1 (after the SCF): the eigenvalues nev <= j < n.
constexpr int BIS_MAXN = 1024;
// one warp per block, so that a molecule's eigenvalues spread over the SMs; each block stages d
// and e^2 again.  2^D lanes per eigenvalue (tri_eigenvalue)
constexpr int EIG_BLOCK = 32;
template <int D>
__global__ void __launch_bounds__(EIG_BLOCK) kb_eigvals(BARGS, int rest) {
  BMOL;
  const int n = q.m.nao;
  const int j0 = rest ? q.nev : 0, j1 = rest ? n : q.nev;
  const int jw = j0 + (int)((blockIdx.x * EIG_BLOCK) >> D);  // the warp's first eigenvalue
  const int j = j0 + (int)((blockIdx.x * EIG_BLOCK + threadIdx.x) >> D);
  const bool head = (threadIdx.x & ((1 << D) - 1)) == 0;
  if (jw >= n) return;
  if (jw >= j1) {
    if (!rest && head && j < n) q.emo[j] = TRI_SENTINEL;
    return;
  }
  __shared__ double sd[BIS_MAXN], se2[BIS_MAXN];
  __shared__ float fd[BIS_MAXN], fe2[BIS_MAXN];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double ee = i < n - 1 ? q.ee[i] * q.ee[i] : 0.0;
    sd[i] = q.ed[i];
    se2[i] = ee;
    fd[i] = (float)q.ed[i];
    fe2[i] = (float)ee;
  }
  const TriBounds b = tri_bounds(n, q.ed, q.ee);  // ends with a block barrier
  if (blockIdx.x == 0 && threadIdx.x == 0 && !rest) q.escal[1] = b.tnorm;
  const bool active = j < j1;
  const double v = tri_eigenvalue<D>(n, sd, se2, fd, fe2, j, active, b);
  if (!head) return;
  if (active) q.emo[j] = v;
  else if (!rest && j < n) q.emo[j] = TRI_SENTINEL;
}
// lanes per eigenvalue: 16, 4 or 1, as many as keep a launch at about eight warps per SM (the FP32
// counts of a group are 15 for 4 levels, 3 for 2: time is saved only while issue slots are free)
static void eigvals_launch(const BatchLaunch& b, int rest) {
  const long long warps = (long long)b.nao_max * b.count, limit = 8LL * 32 * device_sm_count();
  const int D = warps * 16 <= limit ? 4 : warps * 4 <= limit ? 2 : 0;
  const dim3 grid((unsigned)(((b.nao_max << D) + EIG_BLOCK - 1) / EIG_BLOCK), 1, b.count);
  ++g_kernel_launches;
  if (D == 4) kb_eigvals<4><<<grid, EIG_BLOCK, 0, b.s>>>(b.mp, b.list, rest);
  else if (D == 2) kb_eigvals<2><<<grid, EIG_BLOCK, 0, b.s>>>(b.mp, b.list, rest);
  else kb_eigvals<0><<<grid, EIG_BLOCK, 0, b.s>>>(b.mp, b.list, rest);
}

__global__ void __launch_bounds__(INV_WARP) kb_invit(BARGS) {
  BMOL;
  invit_dev(q.m.nao, 0, *q.icount, q.ed, q.ee, q.emo, q.escal, q.lu, q.Y);
}
__global__ void kb_clusters(BARGS) {
  BMOL;
  clusters_dev(q.m.nao, 0, *q.icount, q.ed, q.ee, q.emo, q.escal, 1e-5, q.Y);
}
__global__ void __launch_bounds__(BT_WARPS_B * 32) kb_backtransform(BARGS) {
  BMOL;
  const int n = q.m.nao, k = *q.icount;
  if ((int)blockIdx.x * BT_WARPS_B >= k) return;  // no column of this molecule here
  backtransform_dev<BT_WARPS_B>(n, k, bt_chunk(n, BT_WARPS_B), bt_ysmem(n, BT_WARPS_B), q.A, q.lu,
                                q.Y);
}
__global__ void kb_bt_tmat(BARGS) {
  BMOL;
  const int n = q.m.nao;
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (g * 4 > n - 2) return;
  bt_tmat_dev(n, q.A, q.etau, q.lu, g, threadIdx.x & 31);
}
// mode 0: occupations (total), 1: occupations x energies (vec_out), 2 + c: spin channel c of
// the bond orders (a closed shell's channel 0 is the total occupation)
__global__ void kb_scale_cols(BARGS, int mode) {
  BMOL;
  const int n = q.m.nao;
  const double* f = mode == 0 ? q.focc : mode == 1 ? q.vec_out
                  : q.wbo_ch == 2 ? q.focc + (size_t)(mode - 1) * n : q.focc;
  scale_cols_dev(n, *q.icount, q.C, f, q.scratch);
}

static void batch_attributes() {
  static bool done = false;
  if (done) return;
  ck(cudaFuncSetAttribute(kb_backtransform, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)BT_SMEM_MAX + (int)(BT_WARPS_B * sizeof(double) * 64)),
     "smem attr batch backtransform");
  done = true;
}

void eigen_values_b(const BatchLaunch& b) {
  if (!b.count) return;
  batch_attributes();
  gemm_b(b, GS_FX);
  gemm_b(b, GS_XTT);
  tridiag_fixed_b(b);
  const int tm = prof_kbegin(b.s);
  if (b.nao_max > BIS_MAXN) throw std::runtime_error("batched eigenvalues: molecule too large");
  eigvals_launch(b, 0);
  prof_kend(KS_MULTISECT, tm, b.s);
}

void eigen_values_rest_b(const BatchLaunch& b) {
  if (!b.count) return;
  eigvals_launch(b, 1);
}

void eigen_vectors_b(const BatchLaunch& b) {
  if (!b.count) return;
  batch_attributes();
  g_kernel_launches += 3;
  const int ti = prof_kbegin(b.s);
  kb_invit<<<dim3((b.nao_max + INV_WARP - 1) / INV_WARP, 1, b.count), INV_WARP, 0, b.s>>>(b.mp,
                                                                                          b.list);
  prof_kend(KS_INVIT, ti, b.s);
  kb_clusters<<<dim3(b.nao_max, 1, b.count), 256, 0, b.s>>>(b.mp, b.list);
  const int tb_ = prof_kbegin(b.s);
  ++g_kernel_launches;
  kb_bt_tmat<<<dim3((((b.nao_max - 2) / 4 + 1) * 32 + 127) / 128, 1, b.count), 128, 0, b.s>>>(
      b.mp, b.list);
  kb_backtransform<<<dim3((b.nao_max + BT_WARPS_B - 1) / BT_WARPS_B, 1, b.count),
                     BT_WARPS_B * 32, bt_smem(b.nao_max, BT_WARPS_B), b.s>>>(b.mp, b.list);
  prof_kend(KS_BACKTRANSFORM, tb_, b.s);
  gemm_b(b, GS_XY);
}

void density_b(const BatchLaunch& b, bool weighted) {
  if (!b.count) return;
  const size_t tot = (size_t)b.nao_max * b.nao_max;
  ++g_kernel_launches;
  kb_scale_cols<<<dim3((unsigned)((tot + 255) / 256), 1, b.count), 256, 0, b.s>>>(
      b.mp, b.list, weighted ? 1 : 0);
  gemm_b(b, weighted ? GS_WDENS : GS_DENS);
}

void wbo_b(const BatchLaunch& b, int channel) {
  if (!b.count) return;
  if (b.sp2) {  // closed shells without orbitals: P S directly
    pipe_site_b(b, GS_PS);
    launch_wbo_b(b, channel);
    return;
  }
  const size_t tot = (size_t)b.nao_max * b.nao_max;
  ++g_kernel_launches;
  kb_scale_cols<<<dim3((unsigned)((tot + 255) / 256), 1, b.count), 256, 0, b.s>>>(
      b.mp, b.list, 2 + channel);
  gemm_b(b, GS_WDENS);  // the channel's density into F (W is no longer needed)
  gemm_b(b, GS_FS);
  launch_wbo_b(b, channel);
}

#undef BMOL
#undef BARGS

}  // namespace tb
