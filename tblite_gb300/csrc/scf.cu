// SCF kernels: coordination number, self energies, electrostatics (isotropic, third order,
// anisotropic multipoles), repulsion, Fock assembly, Mulliken analysis, Fermi filling,
// Broyden mixing, and the pair gradients.
//
// Restated from the reference:
//   self energies            src/tblite/xtb/h0.f90:113-217
//   AES radii                src/tblite/coulomb/multipole.f90:389-420
//   isotropic Coulomb        src/tblite/coulomb/charge/effective.f90:238-286, 487-556
//   third order              src/tblite/coulomb/thirdorder.f90:109-172
//   AES matrices/potential   src/tblite/coulomb/multipole.f90:197-350, 488-535, 746-852
//   repulsion                src/tblite/repulsion/effective.f90:187-247
//   Fock assembly            src/tblite/scf/potential.f90:122-255
//   Mulliken                 src/tblite/wavefunction/mulliken.f90:37-100
//   Fermi filling            src/tblite/wavefunction/fermi.f90:31-106, scf/iterator.f90:347-353
//   Broyden                  src/tblite/scf/mixer/broyden.f90:148-278
// Interaction matrices (gamma, AES) are tabulated per pair once per geometry, or evaluated inside the
// potential kernels where there is no table: one warp per atom walks all partners.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>

#include "engine.h"
#include "warp_sums.cuh"

namespace tb {

std::atomic<unsigned long long> g_kernel_launches{0};
std::atomic<unsigned long long> g_split_flops{0};

void stream_wait(cudaStream_t s) {
  thread_local cudaEvent_t ev = nullptr;
  if (!ev) cudaEventCreateWithFlags(&ev, cudaEventBlockingSync | cudaEventDisableTiming);
  cudaEventRecord(ev, s);
  // a short wait is polled (waking a sleeping thread takes tens of microseconds, which every SCF
  // iteration of a small molecule would pay), a longer one sleeps
  if (cudaPeekAtLastError() == cudaSuccess) {  // (an error waiting to be read is left as it is)
    const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(400);
    do {
      if (cudaEventQuery(ev) != cudaErrorNotReady) return;
      cudaGetLastError();  // "not ready" counts as the last error
    } while (std::chrono::steady_clock::now() < until);
  }
  cudaEventSynchronize(ev);
}

// x^e for the small integer exponents of the damping functions, pow() otherwise
__device__ __forceinline__ double powe(double x, double e) {
  if (e == 2.0) return x * x;
  if (e == 3.0) return x * x * x;
  if (e == 4.0) { const double x2 = x * x; return x2 * x2; }
  return pow(x, e);
}

// average hardness of a shell pair: arithmetic (GFN2) or harmonic (GFN1) mean
__device__ __forceinline__ double eta_avg(double a, double b, int harmonic) {
  return harmonic ? 2.0 / (1.0 / a + 1.0 / b) : 0.5 * (a + b);
}

// isotropic kernel 1/(r^g + eta^-g)^(1/g); g = 2 is the GFN2 case
__device__ __forceinline__ double gam_kernel(double r1, double eta, double g) {
  if (g == 2.0) return rsqrt(r1 * r1 + 1.0 / (eta * eta));
  return 1.0 / pow(pow(r1, g) + pow(eta, -g), 1.0 / g);
}

// ------------------------------------------------------------------------------------
// coordination number (double exponential counting function, see oracle for the form)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void dexp_count(double r, double r0, const Gfn2Scalars& p, double& c,
                                           double& dc) {
  if (p.method == 1) {  // GFN1: single exponential 1/(1 + exp(-k (r0/r - 1)))
    const double e = exp(-p.cn_exp_k * (r0 / r - 1.0));
    c = 1.0 / (1.0 + e);
    dc = -c * c * e * p.cn_exp_k * r0 / (r * r);
    return;
  }
  const double e1 = exp(-p.cn_ka * (r0 / r - 1.0));
  const double e2 = exp(-p.cn_kb * ((r0 + p.cn_rshift) / r - 1.0));
  const double f1 = 1.0 / (1.0 + e1), f2 = 1.0 / (1.0 + e2);
  c = f1 * f2;
  const double d1 = -f1 * f1 * e1 * p.cn_ka * r0 / (r * r);
  const double d2 = -f2 * f2 * e2 * p.cn_kb * (r0 + p.cn_rshift) / (r * r);
  dc = d1 * f2 + f1 * d2;
}

__device__ __forceinline__ void cn_dev(DevMol m, Gfn2Scalars p, double* cn) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= m.nat) return;
  const int i = warp;
  const double xi = m.xyz[3 * i], yi = m.xyz[3 * i + 1], zi = m.xyz[3 * i + 2];
  const double cut2 = p.cn_cutoff * p.cn_cutoff;
  double acc = 0.0;
  for (int j = lane; j < m.nat; j += 32) {
    if (j == i) continue;
    const double dx = xi - m.xyz[3 * j], dy = yi - m.xyz[3 * j + 1], dz = zi - m.xyz[3 * j + 2];
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (r2 > cut2 || r2 < 1e-12) continue;
    double c, dc;
    dexp_count(sqrt(r2), m.at_rcov[i] + m.at_rcov[j], p, c, dc);
    acc += c;
  }
  acc = warp_sum(acc);
  if (lane == 0) cn[i] = acc;
}
__global__ void k_cn(DevMol m, Gfn2Scalars p, double* cn) {
  cn_dev(m, p, cn);
}

void launch_cn(const DevMol& m, const Gfn2Scalars& p, double* cn, cudaStream_t s) {
  if (m.nat == 1) {
    cudaMemsetAsync(cn, 0, sizeof(double), s);
    return;
  }
  ++g_kernel_launches;
  k_cn<<<(m.nat * 32 + 63) / 64, 64, 0, s>>>(m, p, cn);
}

// grad_i += sum_j (dEdcn_i + dEdcn_j) dcount/dr (R_i - R_j)/r ; per-atom sigma partials
__device__ __forceinline__ void cn_grad_dev(DevMol m, Gfn2Scalars p, const double* __restrict__ dEdcn, double* grad,
                          double* sig_at) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= m.nat) return;
  const int i = warp;
  const double cut2 = p.cn_cutoff * p.cn_cutoff;
  double g[3] = {0, 0, 0}, sg[9] = {0};
  for (int j = lane; j < m.nat; j += 32) {
    if (j == i) continue;
    double v[3], r2 = 0;
    for (int k = 0; k < 3; ++k) {
      v[k] = m.xyz[3 * i + k] - m.xyz[3 * j + k];
      r2 += v[k] * v[k];
    }
    if (r2 > cut2 || r2 < 1e-12) continue;
    const double r = sqrt(r2);
    double c, dc;
    dexp_count(r, m.at_rcov[i] + m.at_rcov[j], p, c, dc);
    const double f = (dEdcn[i] + dEdcn[j]) * dc / r;
    for (int k = 0; k < 3; ++k) g[k] += f * v[k];
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b) sg[3 * a + b] += 0.5 * f * v[a] * v[b];
  }
  warp_sums_grad(g, sg);
  if (lane == 0) {
    for (int k = 0; k < 3; ++k) grad[3 * i + k] += g[k];
    for (int k = 0; k < 9; ++k) sig_at[9 * i + k] += sg[k];
  }
}
__global__ void k_cn_grad(DevMol m, Gfn2Scalars p, const double* __restrict__ dEdcn, double* grad,
                          double* sig_at) {
  cn_grad_dev(m, p, dEdcn, grad, sig_at);
}

void launch_cn_grad(const DevMol& m, const Gfn2Scalars& p, const double* dEdcn, double* grad,
                    double* sig_at, cudaStream_t s) {
  if (m.nat == 1) return;
  ++g_kernel_launches;
  k_cn_grad<<<(m.nat * 32 + 63) / 64, 64, 0, s>>>(m, p, dEdcn, grad, sig_at);
}

// ------------------------------------------------------------------------------------
// self energies and AES damping radii
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void levels_dev(DevMol m, Gfn2Scalars p, const double* __restrict__ cn, double* se,
                         double* mrad, double* dmrdcn) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < m.nsh) se[t] = m.sh_se0[t] - m.sh_kcn[t] * cn[m.sh_atom[t]];
  if (t < m.nat) {
    const double arg = cn[t] - m.at_vcn[t] - p.mp_shift;
    const double t1 = exp(-p.mp_kexp * arg);
    const double t2 = (p.mp_rmax - m.at_mprad[t]) / (1.0 + t1);
    mrad[t] = m.at_mprad[t] + t2;
    dmrdcn[t] = -t2 * p.mp_kexp * t1 / (1.0 + t1);
  }
}
__global__ void k_levels(DevMol m, Gfn2Scalars p, const double* __restrict__ cn, double* se,
                         double* mrad, double* dmrdcn) {
  levels_dev(m, p, cn, se, mrad, dmrdcn);
}

void launch_setup_levels(const DevMol& m, const Gfn2Scalars& p, const double* cn, double* se,
                         double* mrad, double* dmrdcn, cudaStream_t s) {
  const int nt = m.nsh > m.nat ? m.nsh : m.nat;
  ++g_kernel_launches;
  k_levels<<<(nt + 127) / 128, 128, 0, s>>>(m, p, cn, se, mrad, dmrdcn);
}

// ------------------------------------------------------------------------------------
// homogeneous external electric field (external/field.f90:64-90): atomic and dipole
// potentials of the constant field, and its energy with the output moments
// ------------------------------------------------------------------------------------
struct Field3 {
  double e[3];
};
__global__ void k_field_potential(int nat, const double* __restrict__ xyz, Field3 f, double* vat,
                                  double* vdp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nat) return;
  vat[i] -= f.e[0] * xyz[3 * i] + f.e[1] * xyz[3 * i + 1] + f.e[2] * xyz[3 * i + 2];
  for (int k = 0; k < 3; ++k) vdp[3 * i + k] -= f.e[k];
}
__global__ void k_field_energy(int nat, const double* __restrict__ xyz, Field3 f,
                               const double* __restrict__ qat, const double* __restrict__ dpat,
                               double* eat) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nat) return;
  const double v = f.e[0] * xyz[3 * i] + f.e[1] * xyz[3 * i + 1] + f.e[2] * xyz[3 * i + 2];
  eat[i] -= v * qat[i] + f.e[0] * dpat[3 * i] + f.e[1] * dpat[3 * i + 1] + f.e[2] * dpat[3 * i + 2];
}
void launch_field_potential(int nat, const double* xyz, const double* efield, double* vat,
                            double* vdp, cudaStream_t s) {
  const Field3 f{{efield[0], efield[1], efield[2]}};
  ++g_kernel_launches;
  k_field_potential<<<(nat + 127) / 128, 128, 0, s>>>(nat, xyz, f, vat, vdp);
}
void launch_field_energy(int nat, const double* xyz, const double* efield, const double* qat,
                         const double* dpat, double* eat, cudaStream_t s) {
  const Field3 f{{efield[0], efield[1], efield[2]}};
  ++g_kernel_launches;
  k_field_energy<<<(nat + 127) / 128, 128, 0, s>>>(nat, xyz, f, qat, dpat, eat);
}

// ------------------------------------------------------------------------------------
// electrostatics: one warp per atom i, partners j strided over lanes
// MODE 0: potentials (vsh, vat, vdp, vqp);  MODE 1: per-atom energy (added to eat)
// ------------------------------------------------------------------------------------
constexpr int MAXSH = 3;

// AES pair scalars of atoms i, j at distance r1: g3 f3, g5 f5, g3 f5 with g = 1/r and the
// damping f_n = 1/(1 + 6 (rr)^dmp_n), rr = (mrad_i + mrad_j) / (2 r)
__device__ __forceinline__ void aes_pair(double r1, double mri, double mrj, const Gfn2Scalars& p,
                                         double& g3f3, double& g5f5, double& g3f5) {
  const double g1 = 1.0 / r1, g3 = g1 * g1 * g1, g5 = g3 * g1 * g1;
  const double rr = 0.5 * (mrj + mri) * g1;
  const double f3 = 1.0 / (1.0 + 6.0 * powe(rr, p.mp_dmp3));
  const double f5 = 1.0 / (1.0 + 6.0 * powe(rr, p.mp_dmp5));
  g3f3 = g3 * f3;
  g5f5 = g5 * f5;
  g3f5 = g3 * f5;
}

// Pair table of the electrostatics, once per geometry (one warp per atom i, partners over the
// lanes): gamma of every shell pair of different atoms and the AES pair scalars.  The kernels
// below then read instead of evaluating square roots, divisions and powers per pair in every
// SCF iteration (FP64 arithmetic is the scarce resource of this GPU; the table costs 8 bytes of
// HBM traffic per entry and iteration).
__device__ __forceinline__ void coulomb_table_dev(DevMol m, Gfn2Scalars p,
                                                  const double* __restrict__ mrad, double* tab) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= m.nat) return;
  const int i = warp, nsh = m.nsh, nat = m.nat;
  const int is0 = m.at_sh[i], nsi = m.at_sh[i + 1] - is0;
  double* aes = tab + (size_t)nsh * nsh;
  const size_t plane = (size_t)nat * nat;
  for (int j = lane; j < nat; j += 32) {
    if (j == i) continue;
    double r2 = 0.0;
    for (int k = 0; k < 3; ++k) {
      const double d = m.xyz[3 * i + k] - m.xyz[3 * j + k];
      r2 += d * d;
    }
    const double r1 = sqrt(r2);
    const int js0 = m.at_sh[j], nsj = m.at_sh[j + 1] - js0;
    for (int a = 0; a < nsi; ++a)
      for (int b = 0; b < nsj; ++b)
        tab[(size_t)(is0 + a) * nsh + js0 + b] =
            gam_kernel(r1, eta_avg(m.sh_hub[is0 + a], m.sh_hub[js0 + b], p.harmonic), p.gexp);
    if (!p.aes) continue;
    double g3f3, g5f5, g3f5;
    aes_pair(r1, mrad[i], mrad[j], p, g3f3, g5f5, g3f5);
    const size_t ij = (size_t)i * nat + j;
    aes[ij] = g3f3;
    aes[plane + ij] = g5f5;
    aes[2 * plane + ij] = g3f5;
  }
}

// gamma of the shells s and t of two atoms at distance r1, from the table where there is one
__device__ __forceinline__ double gam_pair(const DevMol& m, const Gfn2Scalars& p, const double* tab,
                                           double r1, int s, int t) {
  return tab ? tab[(size_t)s * m.nsh + t]
             : gam_kernel(r1, eta_avg(m.sh_hub[s], m.sh_hub[t], p.harmonic), p.gexp);
}
__device__ __forceinline__ void aes_scalars(const DevMol& m, const Gfn2Scalars& p,
                                            const double* tab, const double* mrad, double r1,
                                            int i, int j, double& g3f3, double& g5f5,
                                            double& g3f5) {
  if (tab) {
    const size_t plane = (size_t)m.nat * m.nat, ij = (size_t)i * m.nat + j;
    const double* aes = tab + (size_t)m.nsh * m.nsh;
    g3f3 = aes[ij];
    g5f5 = aes[plane + ij];
    g3f5 = aes[2 * plane + ij];
  } else {
    aes_pair(r1, mrad[i], mrad[j], p, g3f3, g5f5, g3f5);
  }
}

// tab: the pair table of coulomb_table_dev, or nullptr to evaluate the pair terms here.  The sixteen
// sums over the warp cost as much as the pairs of a molecule of 50 atoms when each is taken alone.
// 1500 atoms 756 us without the table, 330 with it; 96 atoms 28 and 15 us (energy: 736 and 217, 28
// and 12 us, the contraction by pairs included).
__device__ __forceinline__ void coulomb_potential_dev(DevMol m, Gfn2Scalars p,
                          const double* __restrict__ mrad, const double* __restrict__ qsh,
                          const double* __restrict__ qat, const double* __restrict__ dpat,
                          const double* __restrict__ qpat, double* vsh, double* vat, double* vdp,
                          double* vqp, const double* __restrict__ tab) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= m.nat) return;
  const int i = warp;
  const int is0 = m.at_sh[i], nsi = m.at_sh[i + 1] - is0;
  double xi[3], di[3], qi[6];
  for (int k = 0; k < 3; ++k) {
    xi[k] = m.xyz[3 * i + k];
    di[k] = dpat[3 * i + k];
  }
  for (int k = 0; k < 6; ++k) qi[k] = qpat[6 * i + k];
  const double qa_i = qat[i], ri = mrad[i];
  double ush[MAXSH] = {0, 0, 0};     // sum_j gamma q_j for shells of i
  double uat = 0.0;                  // vat_i
  double ud[3] = {0, 0, 0};          // vdp_i: charges of the partners
  double udd[3] = {0, 0, 0};         // vdp_i: their dipoles
  double uq[6] = {0, 0, 0, 0, 0, 0};  // vqp_i
  const int nsh = m.nsh, nat = m.nat;
  const double* aes = tab + (size_t)nsh * nsh;
  const size_t plane = (size_t)nat * nat;
  for (int j = lane; j < nat; j += 32) {
    if (j == i) continue;
    double v[3];
    for (int k = 0; k < 3; ++k) v[k] = xi[k] - m.xyz[3 * j + k];  // R_i - R_j
    const double r1 = tab ? 0.0 : sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    // isotropic: gamma = 1/sqrt(r^2 + eta^-2) for gexp = 2; general form kept
    const int js0 = m.at_sh[j], nsj = m.at_sh[j + 1] - js0;
    for (int a = 0; a < nsi; ++a) {
      const double hi = m.sh_hub[is0 + a];
      double acc = 0.0;
      for (int b = 0; b < nsj; ++b) {
        const double t = tab ? tab[(size_t)(is0 + a) * nsh + js0 + b]
                             : gam_kernel(r1, eta_avg(hi, m.sh_hub[js0 + b], p.harmonic), p.gexp);
        acc += t * qsh[js0 + b];
      }
      ush[a] += acc;
    }
    if (!p.aes) continue;
    // AES (multipole.f90:488-535), amat(:, jat, iat) with vec = R_iat - R_jat
    double g3f3, g5f5, g3f5;
    if (tab) {
      const size_t ij = (size_t)i * nat + j;
      g3f3 = aes[ij];
      g5f5 = aes[plane + ij];
      g3f5 = aes[2 * plane + ij];
    } else {
      aes_pair(r1, ri, mrad[j], p, g3f3, g5f5, g3f5);
    }
    const double* dj = dpat + 3 * j;
    const double* qj = qpat + 6 * j;
    const double qa_j = qat[j];
    // vat_i += sum_j amat_sd(:, j, i) . dpat_j + amat_sq(:, j, i) . qpat_j   (v = R_i - R_j)
    const double sq[6] = {v[0] * v[0] * g5f5, 2 * v[0] * v[1] * g5f5, v[1] * v[1] * g5f5,
                          2 * v[0] * v[2] * g5f5, 2 * v[1] * v[2] * g5f5, v[2] * v[2] * g5f5};
    uat += (v[0] * dj[0] + v[1] * dj[1] + v[2] * dj[2]) * g3f3;
    for (int k = 0; k < 6; ++k) uat += sq[k] * qj[k];
    // vdp_i += sum_j amat_sd(:, i, j) q_j + amat_dd(:, i, :, j) dpat_j ; amat_sd(:, i, j) = -v g3 f3
    const double vd = v[0] * dj[0] + v[1] * dj[1] + v[2] * dj[2];
    for (int k = 0; k < 3; ++k) {
      ud[k] += -v[k] * g3f3 * qa_j;
      const double dd = dj[k] * g3f5 - v[k] * vd * 3.0 * g5f5;
      udd[k] += dd;
    }
    for (int k = 0; k < 6; ++k) uq[k] += sq[k] * qa_j;
  }
  double u[MAXSH + 13] = {ush[0], ush[1], ush[2], uat,   ud[0], ud[1], ud[2], udd[0],
                          udd[1], udd[2], uq[0],  uq[1], uq[2], uq[3], uq[4], uq[5]};
  static_assert(MAXSH == 3, "three shells per atom");
  constexpr int UAT = MAXSH, UD = UAT + 1, UDD = UD + 3, UQ = UDD + 3;
  if (tab) {
    warp_sums(u);
  } else {  // one by one, as the loop above was compiled with: its roundings stay the same
    for (int k = 0; k < MAXSH + 13; ++k) u[k] = warp_sum(u[k]);
  }
  if (lane != 0) return;
#pragma unroll
  for (int a = 0; a < MAXSH; ++a) {
    if (a >= nsi) break;
    double acc = u[a];  // and the on-site gamma block
    for (int b = 0; b < nsi; ++b)
      acc += eta_avg(m.sh_hub[is0 + a], m.sh_hub[is0 + b], p.harmonic) * qsh[is0 + b];
    const double q = qsh[is0 + a];
    vsh[is0 + a] = acc + (p.third_atom ? 0.0 : q * q * m.sh_gam3[is0 + a]);
  }
  const double mpscale[6] = {1, 2, 1, 2, 2, 1};
  vat[i] = u[UAT] + (p.third_atom ? qa_i * qa_i * m.at_gam3[i] : 0.0);
  for (int k = 0; k < 3; ++k)
    vdp[3 * i + k] =
        p.aes ? u[UD + k] + u[UDD + k] + 2.0 * m.at_dkern[i] * di[k] : 0.0;
  for (int k = 0; k < 6; ++k)
    vqp[6 * i + k] =
        p.aes ? u[UQ + k] + 2.0 * m.at_qkern[i] * qi[k] * mpscale[k] : 0.0;
}

// energy of atom i (added to eat): the potentials of i contracted with its charges and moments
// pair by pair, half the FP64 work of forming them, and one sum over the warp
__device__ __forceinline__ void coulomb_energy_dev(DevMol m, Gfn2Scalars p,
                          const double* __restrict__ mrad, const double* __restrict__ qsh,
                          const double* __restrict__ qat, const double* __restrict__ dpat,
                          const double* __restrict__ qpat, double* eat,
                          const double* __restrict__ tab) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= m.nat) return;
  const int i = warp;
  const int is0 = m.at_sh[i], nsi = m.at_sh[i + 1] - is0;
  const double mpscale[6] = {1, 2, 1, 2, 2, 1};
  double xi[3], di[3], qi[6], qs[MAXSH] = {0.0, 0.0, 0.0};
  for (int k = 0; k < 3; ++k) {
    xi[k] = m.xyz[3 * i + k];
    di[k] = dpat[3 * i + k];
  }
  for (int k = 0; k < 6; ++k) qi[k] = mpscale[k] * qpat[6 * i + k];
#pragma unroll
  for (int a = 0; a < MAXSH; ++a)
    if (a < nsi) qs[a] = 0.5 * qsh[is0 + a];
  double e = 0.0;
  const int nat = m.nat;
  for (int j = lane; j < nat; j += 32) {
    if (j == i) continue;
    double v[3];
    for (int k = 0; k < 3; ++k) v[k] = xi[k] - m.xyz[3 * j + k];  // R_i - R_j
    const double r1 = tab ? 0.0 : sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    const int js0 = m.at_sh[j], nsj = m.at_sh[j + 1] - js0;
#pragma unroll
    for (int a = 0; a < MAXSH; ++a) {
      if (a >= nsi) break;
      double acc = 0.0;
      for (int b = 0; b < nsj; ++b)
        acc += gam_pair(m, p, tab, r1, is0 + a, js0 + b) * qsh[js0 + b];
      e += qs[a] * acc;
    }
    if (!p.aes) continue;
    double g3f3, g5f5, g3f5;
    aes_scalars(m, p, tab, mrad, r1, i, j, g3f3, g5f5, g3f5);
    const double* dj = dpat + 3 * j;
    const double vi = v[0] * di[0] + v[1] * di[1] + v[2] * di[2];
    const double vj = v[0] * dj[0] + v[1] * dj[1] + v[2] * dj[2];
    const double dd = di[0] * dj[0] + di[1] * dj[1] + di[2] * dj[2];
    const double qv = (qi[0] * v[0] + qi[1] * v[1] + qi[3] * v[2]) * v[0] +
                      (qi[2] * v[1] + qi[4] * v[2]) * v[1] + qi[5] * v[2] * v[2];
    // charge-dipole, charge-quadrupole, half of the dipole-dipole term
    e += qat[j] * (g5f5 * qv - g3f3 * vi);
    e += 0.5 * dd * g3f5 - 1.5 * vi * vj * g5f5;
  }
  e = warp_sum(e);
  if (lane != 0) return;
  for (int a = 0; a < nsi; ++a) {
    const double q = qsh[is0 + a];
    double acc = 0.0;  // on-site gamma block
    for (int b = 0; b < nsi; ++b)
      acc += eta_avg(m.sh_hub[is0 + a], m.sh_hub[is0 + b], p.harmonic) * qsh[is0 + b];
    e += 0.5 * acc * q + (p.third_atom ? 0.0 : q * q * q * m.sh_gam3[is0 + a] / 3.0);
  }
  if (p.third_atom) {
    const double q = qat[i];
    e += q * q * q * m.at_gam3[i] / 3.0;
  }
  if (p.aes) {
    double d2 = 0.0, q2 = 0.0;
    for (int k = 0; k < 3; ++k) d2 += di[k] * di[k];
    for (int k = 0; k < 6; ++k) q2 += qi[k] * qpat[6 * i + k];
    e += m.at_dkern[i] * d2 + m.at_qkern[i] * q2;
  }
  eat[i] += e;
}
template <int MODE, bool TAB>
__global__ void k_coulomb(DevMol m, Gfn2Scalars p, const double* __restrict__ mrad,
                          const double* __restrict__ qsh, const double* __restrict__ qat,
                          const double* __restrict__ dpat, const double* __restrict__ qpat,
                          double* vsh, double* vat, double* vdp, double* vqp, double* eat,
                          const double* __restrict__ tab) {
  if (MODE == 0)
    coulomb_potential_dev(m, p, mrad, qsh, qat, dpat, qpat, vsh, vat, vdp, vqp,
                          TAB ? tab : nullptr);
  else
    coulomb_energy_dev(m, p, mrad, qsh, qat, dpat, qpat, eat, TAB ? tab : nullptr);
}
__global__ void k_coulomb_table(DevMol m, Gfn2Scalars p, const double* __restrict__ mrad,
                                double* tab) {
  coulomb_table_dev(m, p, mrad, tab);
}

void launch_coulomb_table(const DevMol& m, const Gfn2Scalars& p, const double* mrad, double* tab,
                          cudaStream_t s) {
  ++g_kernel_launches;
  k_coulomb_table<<<(m.nat * 32 + 63) / 64, 64, 0, s>>>(m, p, mrad, tab);
}

void launch_coulomb_potential(const DevMol& m, const Gfn2Scalars& p, const double* mrad,
                              const double* qsh, const double* qat, const double* dpat,
                              const double* qpat, double* vsh, double* vat, double* vdp,
                              double* vqp, const double* tab, cudaStream_t s) {
  ++g_kernel_launches;
  auto kernel = tab ? k_coulomb<0, true> : k_coulomb<0, false>;
  kernel<<<(m.nat * 32 + 63) / 64, 64, 0, s>>>(m, p, mrad, qsh, qat, dpat, qpat, vsh, vat, vdp, vqp,
                                               nullptr, tab);
}

void launch_coulomb_energy(const DevMol& m, const Gfn2Scalars& p, const double* mrad,
                           const double* qsh, const double* qat, const double* dpat,
                           const double* qpat, double* eat, const double* tab, cudaStream_t s) {
  ++g_kernel_launches;
  auto kernel = tab ? k_coulomb<1, true> : k_coulomb<1, false>;
  kernel<<<(m.nat * 32 + 63) / 64, 64, 0, s>>>(m, p, mrad, qsh, qat, dpat, qpat, nullptr, nullptr,
                                               nullptr, nullptr, eat, tab);
}

// ------------------------------------------------------------------------------------
// electrostatic gradient at fixed charges/moments (es2 + AES); dEdcn += dEdr dmrdcn
// per-atom formulation: atom i sums its own share of every pair (no atomics)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void coulomb_grad_dev(DevMol m, Gfn2Scalars p, const double* __restrict__ mrad,
                               const double* __restrict__ dmrdcn, const double* __restrict__ qsh,
                               const double* __restrict__ qat, const double* __restrict__ dpat,
                               const double* __restrict__ qpat, double* grad, double* sig_at,
                               double* dEdcn) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= m.nat) return;
  const int i = warp;
  const int is0 = m.at_sh[i], nsi = m.at_sh[i + 1] - is0;
  double g[3] = {0, 0, 0}, sg[9] = {0}, dEdr = 0.0;
  const double* di = dpat + 3 * i;
  const double* qi = qpat + 6 * i;
  for (int j = lane; j < m.nat; j += 32) {
    if (j == i) continue;
    double w[3];
    for (int k = 0; k < 3; ++k) w[k] = m.xyz[3 * i + k] - m.xyz[3 * j + k];  // R_i - R_j
    const double r2 = w[0] * w[0] + w[1] * w[1] + w[2] * w[2], r1 = sqrt(r2);
    // es2: d/dR_i of 1/2 sum q gamma q  (pair counted once per atom)
    const int js0 = m.at_sh[j], nsj = m.at_sh[j + 1] - js0;
    double f = 0.0;
    for (int a = 0; a < nsi; ++a)
      for (int b = 0; b < nsj; ++b) {
        const double gm = eta_avg(m.sh_hub[is0 + a], m.sh_hub[js0 + b], p.harmonic);
        double d;
        if (p.gexp == 2.0) {
          d = 1.0 / (r2 + 1.0 / (gm * gm));
          d = -d * sqrt(d);
        } else {
          d = 1.0 / (pow(r1, p.gexp) + pow(gm, -p.gexp));
          d = -pow(r1, p.gexp - 2.0) * d * pow(d, 1.0 / p.gexp);
        }
        f += d * qsh[is0 + a] * qsh[js0 + b];
      }
    double gp[3];
    for (int k = 0; k < 3; ++k) gp[k] = f * w[k];
    if (!p.aes) {  // no anisotropic electrostatics (GFN1)
      for (int k = 0; k < 3; ++k) g[k] += gp[k];
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) sg[3 * a + b] += 0.5 * gp[a] * w[b];
      continue;
    }
    // AES pair term written as in the reference with (iat, jat) = (i, j), vec = R_j - R_i
    const double* dj = dpat + 3 * j;
    const double* qj = qpat + 6 * j;
    const double qai = qat[i], qaj = qat[j];
    double v[3] = {-w[0], -w[1], -w[2]};
    const double rr = 0.5 * (mrad[i] + mrad[j]);
    const double g1 = 1.0 / r1, g3 = g1 * g1 * g1, g5 = g3 * g1 * g1, g7 = g5 * g1 * g1;
    const double f3 = 1.0 / (1.0 + 6.0 * powe(rr * g1, p.mp_dmp3));
    const double d3 = -3 * g5 * f3 - p.mp_dmp3 * f3 * (f3 - 1.0) * g5;
    const double f5 = 1.0 / (1.0 + 6.0 * powe(rr * g1, p.mp_dmp5));
    const double d5 = -5 * f5 - p.mp_dmp5 * (f5 * f5 - f5);
    const double dpiqj = (v[0] * di[0] + v[1] * di[1] + v[2] * di[2]) * qaj;
    const double qidpj = (v[0] * dj[0] + v[1] * dj[1] + v[2] * dj[2]) * qai;
    double fddr = 3.0 * (dpiqj - qidpj) * p.mp_dmp3 * f3 * g3 * (f3 / rr) * powe(rr * g1, p.mp_dmp3);
    double ga[3];
    for (int k = 0; k < 3; ++k)
      ga[k] = -d3 * v[k] * (dpiqj - qidpj) + f3 * g3 * (qai * dj[k] - qaj * di[k]);
    const double dpidpj = di[0] * dj[0] + di[1] * dj[1] + di[2] * dj[2];
    const double dpiv = di[0] * v[0] + di[1] * v[1] + di[2] * v[2];
    const double dpjv = dj[0] * v[0] + dj[1] * v[1] + dj[2] * v[2];
    const double edd = dpidpj * r2 - 3 * dpjv * dpiv;
    fddr += 3.0 * edd * p.mp_dmp5 * f5 * g5 * (f5 / rr) * powe(rr * g1, p.mp_dmp5);
    for (int k = 0; k < 3; ++k)
      ga[k] += -2.0 * f5 * g5 * dpidpj * v[k] + 3.0 * f5 * g5 * (dpiv * dj[k] + dpjv * di[k])
               - edd * d5 * g7 * v[k];
    const double eq = 2 * (qaj * qi[1] + qj[1] * qai) * v[0] * v[1]
                      + 2 * (qaj * qi[3] + qj[3] * qai) * v[0] * v[2]
                      + 2 * (qaj * qi[4] + qj[4] * qai) * v[1] * v[2]
                      + (qaj * qi[0] + qj[0] * qai) * v[0] * v[0]
                      + (qaj * qi[2] + qj[2] * qai) * v[1] * v[1]
                      + (qaj * qi[5] + qj[5] * qai) * v[2] * v[2];
    fddr += eq * 3.0 * p.mp_dmp5 * f5 * g5 * f5 / rr * powe(rr * g1, p.mp_dmp5);
    const double qjv[3] = {v[0] * qj[0] + v[1] * qj[1] + v[2] * qj[3],
                           v[0] * qj[1] + v[1] * qj[2] + v[2] * qj[4],
                           v[0] * qj[3] + v[1] * qj[4] + v[2] * qj[5]};
    const double qiv[3] = {v[0] * qi[0] + v[1] * qi[1] + v[2] * qi[3],
                           v[0] * qi[1] + v[1] * qi[2] + v[2] * qi[4],
                           v[0] * qi[3] + v[1] * qi[4] + v[2] * qi[5]};
    for (int k = 0; k < 3; ++k)
      ga[k] += -eq * d5 * g7 * v[k] - 2.0 * f5 * g5 * qai * qjv[k] - 2.0 * f5 * g5 * qaj * qiv[k];
    dEdr += fddr;
    for (int k = 0; k < 3; ++k) g[k] += gp[k] + ga[k];
    // virial, half of each pair per atom
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b)
        sg[3 * a + b] += 0.5 * gp[a] * w[b] - 0.25 * (v[a] * ga[b] + ga[a] * v[b]);
  }
  warp_sums_grad(g, sg, dEdr);
  if (lane == 0) {
    for (int k = 0; k < 3; ++k) grad[3 * i + k] += g[k];
    for (int k = 0; k < 9; ++k) sig_at[9 * i + k] += sg[k];
    dEdcn[i] += dEdr * dmrdcn[i];
  }
}
__global__ void k_coulomb_grad(DevMol m, Gfn2Scalars p, const double* __restrict__ mrad,
                               const double* __restrict__ dmrdcn, const double* __restrict__ qsh,
                               const double* __restrict__ qat, const double* __restrict__ dpat,
                               const double* __restrict__ qpat, double* grad, double* sig_at,
                               double* dEdcn) {
  coulomb_grad_dev(m, p, mrad, dmrdcn, qsh, qat, dpat, qpat, grad, sig_at, dEdcn);
}

void launch_coulomb_gradient(const DevMol& m, const Gfn2Scalars& p, const double* mrad,
                             const double* dmrdcn, const double* qsh, const double* qat,
                             const double* dpat, const double* qpat, double* grad, double* sig_at,
                             double* dEdcn, cudaStream_t s) {
  if (m.nat == 1) return;
  ++g_kernel_launches;
  k_coulomb_grad<<<(m.nat * 32 + 63) / 64, 64, 0, s>>>(m, p, mrad, dmrdcn, qsh, qat, dpat, qpat,
                                                          grad, sig_at, dEdcn);
}

// ------------------------------------------------------------------------------------
// repulsion energy + gradient (per atom, each pair seen from both atoms)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void repulsion_dev(DevMol m, Gfn2Scalars p, double* erep, double* grad, double* sig_at) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= m.nat) return;
  const int i = warp;
  const double cut2 = p.rep_cutoff * p.rep_cutoff;
  double e = 0.0, g[3] = {0, 0, 0}, sg[9] = {0};
  for (int j = lane; j < m.nat; j += 32) {
    if (j == i) continue;
    double v[3], r2 = 0;
    for (int k = 0; k < 3; ++k) {
      v[k] = m.xyz[3 * i + k] - m.xyz[3 * j + k];
      r2 += v[k] * v[k];
    }
    if (r2 > cut2 || r2 < 1e-12) continue;
    const double r1 = sqrt(r2);
    const double ke = (m.at_z[i] > 2 || m.at_z[j] > 2) ? p.rep_kexp : p.rep_kexp_light;
    const double a = sqrt(m.at_repa[i] * m.at_repa[j]), z = m.at_repz[i] * m.at_repz[j];
    const double r1k = pow(r1, ke), exa = exp(-a * r1k), r1r = pow(r1, p.rep_rexp);
    const double dE = z * exa / r1r;
    e += 0.5 * dE;
    const double f = -(a * r1k * ke + p.rep_rexp) * dE / r2;
    for (int k = 0; k < 3; ++k) g[k] += f * v[k];
    for (int a2 = 0; a2 < 3; ++a2)
      for (int c = 0; c < 3; ++c) sg[3 * a2 + c] += 0.5 * f * v[a2] * v[c];
  }
  warp_sums_grad(g, sg, e);
  if (lane == 0) {
    erep[i] = e;
    if (grad) {
      for (int k = 0; k < 3; ++k) grad[3 * i + k] += g[k];
      for (int k = 0; k < 9; ++k) sig_at[9 * i + k] += sg[k];
    }
  }
}
__global__ void k_repulsion(DevMol m, Gfn2Scalars p, double* erep, double* grad, double* sig_at) {
  repulsion_dev(m, p, erep, grad, sig_at);
}

void launch_repulsion(const DevMol& m, const Gfn2Scalars& p, double* erep, double* grad,
                      double* sig_at, cudaStream_t s) {
  ++g_kernel_launches;
  k_repulsion<<<(m.nat * 32 + 63) / 64, 64, 0, s>>>(m, p, erep, grad, sig_at);
}

// ------------------------------------------------------------------------------------
// orbital potential: vao = vsh(ao) + vat(atom)
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void vao_dev(DevMol m, const double* vsh, const double* vat, double* vao) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m.nao) return;
  vao[t] = vsh[m.ao_sh[t]] + vat[m.ao_at[t]];
}
__global__ void k_vao(DevMol m, const double* vsh, const double* vat, double* vao) {
  vao_dev(m, vsh, vat, vao);
}

void launch_vao(const DevMol& m, const double* vsh, const double* vat, double* vao,
                cudaStream_t s) {
  ++g_kernel_launches;
  k_vao<<<(m.nao + 255) / 256, 256, 0, s>>>(m, vsh, vat, vao);
}

// ------------------------------------------------------------------------------------
// Fock assembly, tiles of 32x32; block (32, 8).  For a tile pair (I <= J) the block reads
// the (I,J) tiles of H, S, D, Q and the (J,I) tiles of D, Q (staged through shared memory),
// writes F(I,J) and its transpose F(J,I).  Every input element is read once.
//   F_rc = H_rc - 1/2 S_rc (v_r + v_c) - 1/2 sum_k (M_k,rc u_k,A(c) + M_k,cr u_k,A(r))
// The two multipole products are summed in an order that depends only on min/max(r,c),
// so F is exactly symmetric.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void fock_dev(int n, const int* __restrict__ ao_at,
                                              const double* __restrict__ H,
                                              const double* __restrict__ S,
                                              const double* __restrict__ D,
                                              const double* __restrict__ Q,
                                              const double* __restrict__ vao,
                                              const double* __restrict__ vdp,
                                              const double* __restrict__ vqp, double* F) {
  const int I = blockIdx.y, J = blockIdx.x;
  if (I > J) return;
  __shared__ double sh2[2][32][33];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const size_t nn = (size_t)n * n;
  const int c = J * 32 + tx;
  const bool cin = c < n;
  double acc[4];
  int rows[4];
  const int atc = cin ? ao_at[c] : 0;
  const double vc = cin ? vao[c] : 0.0;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int r = I * 32 + ty + 8 * s;
    rows[s] = r;
    acc[s] = 0.0;
    if (r < n && cin) {
      const size_t rc = (size_t)r * n + c;
      acc[s] = H[rc] - 0.5 * S[rc] * (vao[r] + vc);
    }
  }
  // multipole terms (absent, D == nullptr, for a Hamiltonian without anisotropic electrostatics).  A
  // small molecule's time is the latency of its loads, so the next matrix is loaded while this one
  // is used, with one barrier each (67 -> 54 us at 1202 orbitals, 13.6 -> 13.0 at 192)
  double tile[4], mrc[4];
  auto load = [&](int k) {
    const double* M = k < 3 ? D + k * nn : Q + (k - 3) * nn;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int rr = J * 32 + ty + 8 * s, cc = I * 32 + tx;  // tile (J, I) of M
      tile[s] = (rr < n && cc < n) ? M[(size_t)rr * n + cc] : 0.0;
      mrc[s] = (rows[s] < n && cin) ? M[(size_t)rows[s] * n + c] : 0.0;
    }
  };
  if (D != nullptr) load(0);
  for (int k = 0; D != nullptr && k < 9; ++k) {
    const double* u = k < 3 ? vdp : vqp;
    const int ku = k < 3 ? k : k - 3, su = k < 3 ? 3 : 6;
    double(&sh)[32][33] = sh2[k & 1];  // sh[a][b] = M[J*32 + a][I*32 + b]
    double m[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      sh[ty + 8 * s][tx] = tile[s];
      m[s] = mrc[s];
    }
    __syncthreads();
    if (k < 8) load(k + 1);
    const double uc = cin ? u[su * atc + ku] : 0.0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int r = rows[s];
      if (r < n && cin) {
        const double t1 = m[s] * uc;                                   // M_rc u_A(c)
        const double t2 = sh[tx][ty + 8 * s] * u[su * ao_at[r] + ku];  // M_cr u_A(r)
        acc[s] -= 0.5 * (r <= c ? (t1 + t2) : (t2 + t1));
      }
    }
  }
  double(&sh)[32][33] = sh2[1];  // (the last matrix used the other buffer)
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int r = rows[s];
    if (r < n && cin) F[(size_t)r * n + c] = acc[s];
  }
  if (I == J) return;
  // transpose write of F(J,I)
#pragma unroll
  for (int s = 0; s < 4; ++s) sh[ty + 8 * s][tx] = acc[s];
  __syncthreads();
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int rr = J * 32 + ty + 8 * s, cc = I * 32 + tx;
    if (rr < n && cc < n) F[(size_t)rr * n + cc] = sh[tx][ty + 8 * s];
  }
}
__global__ void __launch_bounds__(256) k_fock(int n, const int* __restrict__ ao_at,
                                              const double* __restrict__ H,
                                              const double* __restrict__ S,
                                              const double* __restrict__ D,
                                              const double* __restrict__ Q,
                                              const double* __restrict__ vao,
                                              const double* __restrict__ vdp,
                                              const double* __restrict__ vqp, double* F) {
  fock_dev(n, ao_at, H, S, D, Q, vao, vdp, vqp, F);
}

void launch_fock(int n, const int* ao_at, const double* H, const double* S, const double* D,
                 const double* Q, const double* vao, const double* vdp, const double* vqp, double* F,
                 cudaStream_t s) {
  const int nt = (n + 31) / 32;
  ++g_kernel_launches;
  const int tk = prof_kbegin(s);
  k_fock<<<dim3(nt, nt), dim3(32, 8), 0, s>>>(n, ao_at, H, S, D, Q, vao, vdp, vqp, F);
  prof_kend(KS_FOCK, tk, s);
}

// ------------------------------------------------------------------------------------
// Mulliken: column sums over row chunks.  partial[chunk][11][n]:
//   0: sum_r P S, 1-3: sum_r P D_k, 4-9: sum_r P Q_q, 10: sum_r P H
// ------------------------------------------------------------------------------------
// rows per chunk: 11 FP64 multiply-adds per row and column, so short chunks spread a molecule
// over more SMs (68 orbitals: 64 rows 80 us, 16 rows 21 us)
// (64 where a molecule keeps its order of summation, see tridiag_fixed)
constexpr int MULL_SHORT = 16, MULL_LONG = 64;
__host__ __device__ constexpr int mull_rows(int n) { return n <= 512 ? MULL_SHORT : MULL_LONG; }

int mulliken_chunks(int n) { return (n + mull_rows(n) - 1) / mull_rows(n); }

// FLIGHT rows with their loads in flight: four for one molecule, whose few blocks wait for them (21 ->
// 10 us at 192 orbitals, 207 -> 73 us at 1202; 245 us where the rows of a chunk are not a constant of
// the kernel), one in a batch, where other blocks fill the time (four take 95 us a launch instead of
// 65 there)
template <int FLIGHT>
__device__ __forceinline__ void mull_partial_dev(int n, int rows, const double* __restrict__ P,
                                                      const double* __restrict__ S,
                                                      const double* __restrict__ H,
                                                      const double* __restrict__ D,
                                                      const double* __restrict__ Q,
                                                      double* partial) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int chunk = blockIdx.y;
  if (c >= n) return;
  const size_t nn = (size_t)n * n;
  double acc[11];
#pragma unroll
  for (int k = 0; k < 11; ++k) acc[k] = 0.0;
  const int r0 = chunk * rows, r1 = min(n, r0 + rows);
#pragma unroll FLIGHT
  for (int r = r0; r < r1; ++r) {
    const size_t rc = (size_t)r * n + c;
    const double pv = P[rc];
    acc[0] += pv * S[rc];
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[1 + k] += pv * D[k * nn + rc];
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[4 + q] += pv * Q[q * nn + rc];
    acc[10] += pv * H[rc];
  }
#pragma unroll
  for (int k = 0; k < 11; ++k) partial[((size_t)chunk * 11 + k) * n + c] = acc[k];
}
template <int ROWS>
__global__ void __launch_bounds__(128) k_mull_partial(int n, const double* __restrict__ P,
                                                      const double* __restrict__ S,
                                                      const double* __restrict__ H,
                                                      const double* __restrict__ D,
                                                      const double* __restrict__ Q,
                                                      double* partial) {
  mull_partial_dev<4>(n, ROWS, P, S, H, D, Q, partial);
}

// 16 threads per atom, one per sum (population, 3 dipole, 6 quadrupole, band energy): reduce the
// chunks of its orbitals, fill shells/atoms
constexpr int MULL_LANES = 16;
__device__ __forceinline__ void mull_reduce_dev(DevMol m, const double* __restrict__ partial, int nchunk,
                              double* qsh, double* qat, double* dpat, double* qpat,
                              double* eband) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t / MULL_LANES, k = t % MULL_LANES;
  if (i >= m.nat || k >= 11) return;
  const int n = m.nao;
  const double* __restrict__ pk = partial + (size_t)k * n;
  double sum = 0.0, qa = 0.0;
  for (int s = m.at_sh[i]; s < m.at_sh[i + 1]; ++s) {
    const int o = m.sh_ao[s], no = 2 * m.sh_l[s] + 1;
    if (k == 0) sum = 0.0;
    for (int mu = o; mu < o + no; ++mu) {
#pragma unroll 4
      for (int ch = 0; ch < nchunk; ++ch) sum += pk[(size_t)ch * 11 * n + mu];
    }
    if (k == 0) {
      const double v = m.sh_refocc[s] - sum;
      qsh[s] = v;
      qa += v;
    }
  }
  if (k == 0) qat[i] = qa;
  else if (k < 4) dpat[3 * i + k - 1] = -sum;
  else if (k < 10) qpat[6 * i + k - 4] = -sum;
  else eband[i] = sum;
}
__global__ void k_mull_reduce(DevMol m, const double* __restrict__ partial, int nchunk,
                              double* qsh, double* qat, double* dpat, double* qpat,
                              double* eband) {
  mull_reduce_dev(m, partial, nchunk, qsh, qat, dpat, qpat, eband);
}

void launch_mulliken(const DevMol& m, const double* P, const double* S, const double* H,
                     const double* D, const double* Q, double* partial, bool ordered, double* qsh,
                     double* qat, double* dpat, double* qpat, double* eband, cudaStream_t s) {
  const int n = m.nao, rows = ordered ? MULL_LONG : mull_rows(n), nchunk = (n + rows - 1) / rows;
  auto partial_sums = rows == MULL_LONG ? k_mull_partial<MULL_LONG> : k_mull_partial<MULL_SHORT>;
  ++g_kernel_launches;
  const int tk = prof_kbegin(s);
  partial_sums<<<dim3((n + 127) / 128, nchunk), 128, 0, s>>>(n, P, S, H, D, Q, partial);
  prof_kend(KS_MULLIKEN, tk, s);
  ++g_kernel_launches;
  k_mull_reduce<<<(m.nat * MULL_LANES + 127) / 128, 128, 0, s>>>(m, partial, nchunk, qsh, qat, dpat,
                                                                 qpat, eband);
}

// threads of a one-block kernel over n elements: no more warps than elements need, since every
// warp of a block sum takes its scheduler the same five FP64 additions (the sums are the same bit
// for bit as with 1024 threads, the missing warps would add zeros)
static int one_block(int n) { return n >= 1024 ? 1024 : n <= 32 ? 32 : (n + 31) / 32 * 32; }

// ------------------------------------------------------------------------------------
// Fermi filling (one block).  Both spin channels share the eigenvalues.
// ------------------------------------------------------------------------------------
__device__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  double t = threadIdx.x < nw ? red[threadIdx.x] : 0.0;
  if (w == 0) t = warp_sum(t);
  __syncthreads();
  if (threadIdx.x == 0) red[0] = t;
  __syncthreads();
  const double r = red[0];
  __syncthreads();
  return r;
}

// returns the highest Fermi level at which occupations were evaluated (-1e300 if none)
__device__ double fermi_channel(int n, const double* emo, double nel, double kt, double* occ,
                                double* red, double* ts) {
  double ef_max = -1e300;
  // Aufbau
  int homo = (int)floor(nel);
  const double frac = fmod(nel, 1.0);
  for (int k = threadIdx.x; k < n; k += blockDim.x)
    occ[k] = k < homo ? 1.0 : (k == homo ? frac : 0.0);
  __syncthreads();
  homo = frac > 0.5 ? homo + 1 : homo;
  if (homo > 0) {
    double ef = 0.5 * (emo[max(homo, 1) - 1] + emo[min(homo + 1, n) - 1]);
    const double occt = homo;
    const double thr = 1.4901161193847656e-08;      // sqrt(epsilon)
    const double sqrttiny = 1.4916681462400413e-154;  // sqrt(tiny)
    for (int cyc = 0; cyc < 200; ++cyc) {
      ef_max = fmax(ef_max, ef);
      double tn = 0.0, td = 0.0;
      for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const double x = (emo[k] - ef) / kt;
        double f = 0.0, df = 0.0;
        if (x < 50.0) {
          const double ex = exp(x);
          f = 1.0 / (ex + 1.0);
          df = ex / (kt * (ex + 1.0) * (ex + 1.0));
        }
        occ[k] = f;
        tn += f;
        td += df;
      }
      tn = block_sum(tn, red);
      td = block_sum(td, red);
      const double change = td > sqrttiny ? (occt - tn) / td : 0.0;
      ef += change;
      if (fabs(occt - tn) <= thr) break;
    }
  }
  __syncthreads();
  double s = 0.0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const double o = occ[k];
    if (o != 0.0 && o != 1.0) s += log(pow(o, o) * pow(1.0 - o, 1.0 - o));  // else log(1) = 0
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) *ts += s * kt;
  __syncthreads();
  return ef_max;
}

// emo[nev..n) may be placeholders (1e300) for levels that were not computed: valid as long as
// the highest computed level lies 51 kT above every Fermi level used (the occupation is then
// exactly zero above it, as for the true levels); otherwise ncols[1] = 1
__device__ __forceinline__ void fermi_dev(int n, const double* emo, double nalp, double nbet, double kt, double* fa,
                        double* fb, double* focc, double* ts, int* ncols, int nev) {
  __shared__ double red[32];
  if (threadIdx.x == 0) *ts = 0.0;
  __syncthreads();
  const double efa = fermi_channel(n, emo, nalp, kt, fa, red, ts);
  double efb = efa;
  if (nalp == nbet) {  // closed shell: the same filling twice
    for (int k = threadIdx.x; k < n; k += blockDim.x) fb[k] = fa[k];
    if (threadIdx.x == 0) *ts += *ts;
  } else {
    efb = fermi_channel(n, emo, nbet, kt, fb, red, ts);
  }
  if (threadIdx.x == 0)
    ncols[1] = (nev < n && !(emo[nev - 1] >= fmax(efa, efb) + 51.0 * kt)) ? 1 : 0;
  int last = -1;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const double f = fa[k] + fb[k];
    focc[k] = f;
    if (f != 0.0) last = max(last, k);
  }
  // block max
  __shared__ int mx;
  if (threadIdx.x == 0) mx = -1;
  __syncthreads();
  atomicMax(&mx, last);
  __syncthreads();
  if (threadIdx.x == 0) *ncols = mx + 1;
}
__global__ void k_fermi(int n, const double* emo, double nalp, double nbet, double kt, double* fa,
                        double* fb, double* focc, double* ts, int* ncols, int nev) {
  fermi_dev(n, emo, nalp, nbet, kt, fa, fb, focc, ts, ncols, nev);
}

void launch_fermi(int n, const double* emo, double nalp, double nbet, double kt, double* focc,
                  double* ts, int* ncols, cudaStream_t s, int nev) {
  // fa, fb scratch follow focc in memory: focc[n], fa[n], fb[n]
  ++g_kernel_launches;
  k_fermi<<<1, one_block(n), 0, s>>>(n, emo, nalp, nbet, kt, focc + n, focc + 2 * n, focc, ts, ncols,
                             nev > 0 ? nev : n);
}

// ------------------------------------------------------------------------------------
// mixer vector packing  [qsh | dpat | qpat]
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void pack_dev(int nsh, int nat, const double* qsh, const double* dpat, const double* qpat,
                       double* vec) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nd = nsh + 9 * nat;
  if (t >= nd) return;
  if (t < nsh) vec[t] = qsh[t];
  else if (t < nsh + 3 * nat) vec[t] = dpat[t - nsh];
  else vec[t] = qpat[t - nsh - 3 * nat];
}
__global__ void k_pack(int nsh, int nat, const double* qsh, const double* dpat, const double* qpat,
                       double* vec) {
  pack_dev(nsh, nat, qsh, dpat, qpat, vec);
}

void launch_pack(const DevMol& m, const double* qsh, const double* dpat, const double* qpat,
                 double* vec, cudaStream_t s, bool with_mp) {
  const int nmp = with_mp ? m.nat : 0;  // atoms whose multipoles enter the mixer
  const int nd = m.nsh + 9 * nmp;
  ++g_kernel_launches;
  k_pack<<<(nd + 255) / 256, 256, 0, s>>>(m.nsh, nmp, qsh, dpat, qpat, vec);
}

__device__ __forceinline__ void unpack_dev(DevMol m, const double* vec, double* qsh, double* qat, double* dpat,
                         double* qpat, int with_mp) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int nsh = m.nsh, nat = m.nat;
  if (t < nsh) qsh[t] = vec[t];
  if (with_mp && t < 3 * nat) dpat[t] = vec[nsh + t];
  if (with_mp && t < 6 * nat) qpat[t] = vec[nsh + 3 * nat + t];
  if (t < nat) {
    double a = 0.0;
    for (int s = m.at_sh[t]; s < m.at_sh[t + 1]; ++s) a += vec[s];
    qat[t] = a;
  }
}
__global__ void k_unpack(DevMol m, const double* vec, double* qsh, double* qat, double* dpat,
                         double* qpat, int with_mp) {
  unpack_dev(m, vec, qsh, qat, dpat, qpat, with_mp);
}

void launch_unpack(const DevMol& m, const double* vec, double* qsh, double* qat, double* dpat,
                   double* qpat, cudaStream_t s, bool with_mp) {
  const int nt = m.nsh > 6 * m.nat ? m.nsh : 6 * m.nat;
  ++g_kernel_launches;
  k_unpack<<<(nt + 255) / 256, 256, 0, s>>>(m, vec, qsh, qat, dpat, qpat, with_mp ? 1 : 0);
}

__device__ __forceinline__ void diff_dev(int nd, const double* vout, const double* q, double* dq, double* err) {
  __shared__ double red[32];
  double s = 0.0;
  for (int t = threadIdx.x; t < nd; t += blockDim.x) {
    const double d = vout[t] - q[t];
    dq[t] = d;
    s += d * d / nd;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) *err = sqrt(s);
}
__global__ void k_diff(int nd, const double* vout, const double* q, double* dq, double* err) {
  diff_dev(nd, vout, q, dq, err);
}

void launch_diff(int nd, const double* vout, const double* q, double* dq, double* err,
                 cudaStream_t s) {
  ++g_kernel_launches;
  k_diff<<<1, one_block(nd), 0, s>>>(nd, vout, q, dq, err);
}

// ------------------------------------------------------------------------------------
// Broyden step (one block).  Same recurrences as the reference; the overlap matrix a(i,j)
// is kept between calls and only the row of the newest history vector is recomputed
// (the other rows are unchanged dot products).  ordered: dot products and back substitution keep
// the order of summation of a block sum and of a row by row solution.
// ------------------------------------------------------------------------------------
__device__ double block_dot(int nd, const double* x, const double* y, double* red) {
  double s = 0.0;
  for (int t = threadIdx.x; t < nd; t += blockDim.x) s += x[t] * y[t];
  return block_sum(s, red);
}

__device__ __forceinline__ void broyden_dev(int nd, int memory, int iter, double alpha, double* q, double* qlast,
                          const double* dq, double* dqlast, double* df, double* u, double* a,
                          double* omega, double* work, int* status, bool ordered) {
  __shared__ double red[32];
  if (iter == 1) {
    for (int t = threadIdx.x; t < nd; t += blockDim.x) {
      dqlast[t] = dq[t];
      qlast[t] = q[t];
      q[t] = q[t] + alpha * dq[t];
    }
    if (threadIdx.x == 0) *status = 0;
    return;
  }
  const int itn = iter - 1;
  const int it1 = (itn - 1) % memory;
  const int nhist = min(memory, itn);
  const int first = max(1, itn - memory + 1);
  const double omega0 = 0.01, minw = 1.0, maxw = 100000.0, wfac = 0.01;
  double w = sqrt(block_dot(nd, dq, dq, red));
  w = w > wfac / maxw ? wfac / w : maxw;
  if (w < minw) w = minw;
  if (threadIdx.x == 0) omega[it1] = w;
  double* dfn = df + (size_t)it1 * nd;
  for (int t = threadIdx.x; t < nd; t += blockDim.x) dfn[t] = dq[t] - dqlast[t];
  __syncthreads();
  double inv = sqrt(block_dot(nd, dfn, dfn, red));
  inv = inv > 2.220446049250313e-16 ? inv : 2.220446049250313e-16;
  inv = 1.0 / inv;
  for (int t = threadIdx.x; t < nd; t += blockDim.x) dfn[t] *= inv;
  __syncthreads();
  // history indices, c vector, a row: one warp per dot product (a block sum would take every warp
  // five FP64 additions per product)
  constexpr int NS = 48;  // histories up to this order are solved in shared memory
  __shared__ double sbeta[NS * NS], sfac[NS], sc[NS];
  double* beta = nhist <= NS ? sbeta : work;                  // [nhist][nhist]
  double* cvec = nhist <= NS ? sc : work + memory * memory;   // [nhist]
  double* fac = nhist <= NS ? sfac : cvec + memory;           // [nhist]
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (ordered) {
    for (int ih = 0; ih < nhist; ++ih) {
      const int i = (first + ih - 1) % memory;
      const double dfi_dq = block_dot(nd, df + (size_t)i * nd, dq, red);
      const double aij = block_dot(nd, df + (size_t)i * nd, dfn, red);
      if (threadIdx.x == 0) {
        cvec[ih] = omega[i] * dfi_dq;
        a[(size_t)i * memory + it1] = aij;
        a[(size_t)it1 * memory + i] = aij;
      }
    }
  }
  for (int t = wid; !ordered && t < 2 * nhist; t += nw) {
    const int ih = t >> 1, i = (first + ih - 1) % memory;
    const double *x = df + (size_t)i * nd, *y = (t & 1) ? dfn : dq;
    double s0 = 0.0, s1 = 0.0;
    int k = lane;
    for (; k + 32 < nd; k += 64) {
      s0 = fma(x[k], y[k], s0);
      s1 = fma(x[k + 32], y[k + 32], s1);
    }
    if (k < nd) s0 = fma(x[k], y[k], s0);
    s0 = warp_sum(s0 + s1);
    if (lane == 0) {
      if (t & 1) {
        a[(size_t)i * memory + it1] = s0;
        a[(size_t)it1 * memory + i] = s0;
      } else {
        cvec[ih] = omega[i] * s0;
      }
    }
  }
  __syncthreads();
  // solve beta^T x = c by Gaussian elimination with partial pivoting (getrf + getrs 't'); warp 0
  // finds and swaps the pivot row and forms the multipliers, all threads apply them
  for (int t = threadIdx.x; t < nhist * nhist; t += blockDim.x) {
    const int jh = t / nhist, ih = t % nhist;  // transposed
    const int i = (first + ih - 1) % memory, j = (first + jh - 1) % memory;
    beta[t] = omega[i] * omega[j] * a[(size_t)i * memory + j] + (ih == jh ? omega0 * omega0 : 0.0);
  }
  __shared__ int fail;
  if (threadIdx.x == 0) fail = 0;
  __syncthreads();
  for (int k = 0; k < nhist; ++k) {
    if (wid == 0) {
      unsigned long long best = 0ull;  // |value| as bits, then the first row that has it
      for (int i = k + lane; i < nhist; i += 32)
        best = max(best, (unsigned long long)__double_as_longlong(fabs(beta[i * nhist + k])));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
      int p = nhist;
      for (int i = k + lane; i < nhist; i += 32)
        if ((unsigned long long)__double_as_longlong(fabs(beta[i * nhist + k])) == best) p = min(p, i);
      p = __reduce_min_sync(0xffffffffu, p);
      if (best == 0ull) {
        if (lane == 0) fail = k + 1;
      } else {
        if (p != k) {
          for (int j = lane; j < nhist; j += 32) {
            const double x = beta[k * nhist + j];
            beta[k * nhist + j] = beta[p * nhist + j];
            beta[p * nhist + j] = x;
          }
          if (lane == 0) {
            const double x = cvec[k];
            cvec[k] = cvec[p];
            cvec[p] = x;
          }
          __syncwarp();
        }
        const double pivv = beta[k * nhist + k];
        for (int i = k + 1 + lane; i < nhist; i += 32) fac[i] = beta[i * nhist + k] / pivv;
      }
    }
    __syncthreads();
    if (fail) break;
    const int rem = nhist - k - 1;
    for (int t = threadIdx.x; t < rem * (rem + 1); t += blockDim.x) {
      const int i = k + 1 + t / (rem + 1), j = k + 1 + t % (rem + 1);
      if (j < nhist) beta[i * nhist + j] = fma(-fac[i], beta[k * nhist + j], beta[i * nhist + j]);
      else cvec[i] = fma(-fac[i], cvec[k], cvec[i]);
    }
    __syncthreads();
  }
  if (fail) {
    if (threadIdx.x == 0) *status = fail;
    return;
  }
  // back substitution by columns: the diagonal's reciprocals first, then one solved element at a
  // time leaves all the rows above it (ordered: row by row, one thread)
  for (int i = threadIdx.x; i < nhist; i += blockDim.x) fac[i] = 1.0 / beta[i * nhist + i];
  __syncthreads();
  if (wid == 0) {
    if (ordered && lane == 0)
      for (int i = nhist - 1; i >= 0; --i) {
        double x = cvec[i];
        for (int j = i + 1; j < nhist; ++j) x -= beta[i * nhist + j] * cvec[j];
        cvec[i] = x / beta[i * nhist + i];
      }
    __syncwarp();
    for (int i = nhist - 1; !ordered && i >= 0; --i) {
      const double x = cvec[i] * fac[i];
      for (int l = lane; l < i; l += 32) cvec[l] = fma(-beta[l * nhist + i], x, cvec[l]);
      __syncwarp();
      if (lane == 0) cvec[i] = x;
    }
    for (int ih = lane; ih < nhist; ih += 32) fac[ih] = omega[(first + ih - 1) % memory];
    __syncwarp();
    for (int ih = lane; ih < nhist; ih += 32) fac[ih] *= cvec[ih];
    if (lane == 0) *status = 0;
  }
  __syncthreads();
  double* un = u + (size_t)it1 * nd;
  for (int t = threadIdx.x; t < nd; t += blockDim.x) {
    un[t] = alpha * dfn[t] + inv * (q[t] - qlast[t]);
    dqlast[t] = dq[t];
    qlast[t] = q[t];
    double v = q[t] + alpha * dq[t];
    // (each thread reads its own element of the new history vector)
#pragma unroll 4
    for (int ih = 0; ih < nhist; ++ih)
      v = fma(-fac[ih], u[(size_t)((first + ih - 1) % memory) * nd + t], v);
    q[t] = v;
  }
}
__global__ void k_broyden(int nd, int memory, int iter, double alpha, double* q, double* qlast,
                          const double* dq, double* dqlast, double* df, double* u, double* a,
                          double* omega, double* work, int* status, bool ordered) {
  broyden_dev(nd, memory, iter, alpha, q, qlast, dq, dqlast, df, u, a, omega, work, status,
              ordered);
}

__device__ __forceinline__ void eelec_init_dev(int nat, const double* ts, const double* eband, double* eelec) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nat) eelec[i] = *ts / nat + eband[i];
}
__global__ void k_eelec_init(int nat, const double* ts, const double* eband, double* eelec) {
  eelec_init_dev(nat, ts, eband, eelec);
}

__global__ void k_collect(int nat, const double* eelec, const double* scal, const int* icount,
                          const int* status, double* out) {
  for (int t = threadIdx.x; t < nat + 5; t += blockDim.x)
    out[t] = t < nat       ? eelec[t]
             : t < nat + 2 ? scal[t - nat]
             : t < nat + 4 ? (double)icount[t - nat - 2]
                           : (double)*status;
}
void launch_collect(int nat, const double* eelec, const double* scal, const int* icount,
                    const int* status, double* out, cudaStream_t s) {
  ++g_kernel_launches;
  k_collect<<<1, one_block(nat + 5), 0, s>>>(nat, eelec, scal, icount, status, out);
}

void launch_eelec_init(int nat, const double* ts, const double* eband, double* eelec,
                       cudaStream_t s) {
  ++g_kernel_launches;
  k_eelec_init<<<(nat + 127) / 128, 128, 0, s>>>(nat, ts, eband, eelec);
}

__device__ __forceinline__ void fe_dev(int n, const double* f, const double* e, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = f[i] * e[i];
}
__global__ void k_fe(int n, const double* f, const double* e, double* out) {
  fe_dev(n, f, e, out);
}

void launch_fe(int n, const double* f, const double* e, double* out, cudaStream_t s) {
  ++g_kernel_launches;
  k_fe<<<(n + 255) / 256, 256, 0, s>>>(n, f, e, out);
}

void launch_broyden_next(BroydenState& b, cudaStream_t s) {
  b.iter += 1;
  ++g_kernel_launches;
  k_broyden<<<1, std::max(256, one_block(b.ndim)), 0, s>>>(b.ndim, b.memory, b.iter, b.damp, b.q, b.qlast, b.dq, b.dqlast,
                               b.df, b.u, b.a, b.omega, b.work, b.status, b.ordered);
}

// ------------------------------------------------------------------------------------
// Wiberg/Mayer bond orders (wavefunction/mulliken.f90:176-235): for atoms A != B
//   wbo(A, B) += scale * sum_{mu in A, nu in B} (PS)_{nu mu} (PS)_{mu nu}
// one thread per atom pair; the orbitals of an atom are contiguous
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void wbo_dev(DevMol m, const double* __restrict__ PS, double* wbo,
                                        double scale) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int nat = m.nat, n = m.nao;
  if (t >= (long long)nat * nat) return;
  const int a = (int)(t / nat), b = (int)(t % nat);
  if (a == b) return;
  const int a0 = m.sh_ao[m.at_sh[a]], a1 = m.sh_ao[m.at_sh[a + 1] - 1] + 2 * m.sh_l[m.at_sh[a + 1] - 1] + 1;
  const int b0 = m.sh_ao[m.at_sh[b]], b1 = m.sh_ao[m.at_sh[b + 1] - 1] + 2 * m.sh_l[m.at_sh[b + 1] - 1] + 1;
  double s = 0.0;
  for (int mu = a0; mu < a1; ++mu)
    for (int nu = b0; nu < b1; ++nu) s += PS[(size_t)nu * n + mu] * PS[(size_t)mu * n + nu];
  wbo[t] += scale * s;
}
__global__ void k_wbo(DevMol m, const double* __restrict__ PS, double* wbo, double scale) {
  wbo_dev(m, PS, wbo, scale);
}
void launch_wbo(const DevMol& m, const double* PS, double* wbo, double scale, cudaStream_t s) {
  const long long nn = (long long)m.nat * m.nat;
  ++g_kernel_launches;
  k_wbo<<<(unsigned)((nn + 255) / 256), 256, 0, s>>>(m, PS, wbo, scale);
}

// ------------------------------------------------------------------------------------
// Parameter gradient of the converged energy (the SCF energy is stationary in the density,
// so dE/dtheta is the explicit derivative at the final P and charges):
//   self energies   H0_{mu nu} = (e_i + e_j)/2 * G_{mu nu}  =>  dE/de_s = sum_{mu in s, nu} P G'
//                   with G' = H0 built with every self energy set to one (= 2 G)
//   hardness        E2 = 1/2 sum_st q_s q_t gamma_st, gamma = (R^2 + eta_st^-2)^-1/2,
//                   eta_st = (eta_s + eta_t)/2  =>  dgamma/deta_st = eta_st^-3 (R^2+eta_st^-2)^-3/2
//   third order     E3 = sum_s Gamma_s q_s^3 / 3
// one thread per shell
// ------------------------------------------------------------------------------------
// Hp: H0 built with unit self energies; or nullptr, and then the same elements come from H0
// and the self energies se, Hp = H0 / ((e_s + e_t) / 2) (H0 is linear in the pair's mean self
// energy, which is never zero).  cn != nullptr: also out[3 nsh + s] = dE/dkcn_s = -CN_A dE/de_s
__device__ __forceinline__ void param_grad_dev(const DevMol& m, const double* __restrict__ P,
                                               const double* __restrict__ Hp,
                                               const double* __restrict__ H,
                                               const double* __restrict__ se,
                                               const double* __restrict__ cn,
                                               const double* __restrict__ qsh, double* out,
                                               double* zgrad, int s) {
  const int n = m.nao, nsh = m.nsh;
  const int o = m.sh_ao[s], no = 2 * m.sh_l[s] + 1;
  double tr = 0.0;
  for (int mu = o; mu < o + no; ++mu) {
    const double* pr = P + (size_t)mu * n;
    if (Hp) {
      const double* hr = Hp + (size_t)mu * n;
      for (int nu = 0; nu < n; ++nu) tr += pr[nu] * hr[nu];
    } else {
      const double* hr = H + (size_t)mu * n;
      const double es = se[s];
      for (int nu = 0; nu < n; ++nu) tr += pr[nu] * hr[nu] * (2.0 / (es + se[m.ao_sh[nu]]));
    }
  }
  const double qs = qsh[s], es = m.sh_hub[s];
  const int ia = m.sh_atom[s];
  double dh = 0.5 * qs * qs;  // gamma_ss = eta_s
  for (int t = 0; t < nsh; ++t) {
    if (t == s) continue;
    const int ja = m.sh_atom[t];
    double r2 = 0.0;
    for (int k = 0; k < 3; ++k) {
      const double d = m.xyz[3 * ia + k] - m.xyz[3 * ja + k];
      r2 += d * d;
    }
    const double eta = 0.5 * (es + m.sh_hub[t]);
    const double ie2 = 1.0 / (eta * eta);
    const double den = r2 + ie2;
    const double g = ie2 / eta / (den * sqrt(den));
    dh += qs * qsh[t] * 0.5 * g;
  }
  out[s] = tr;
  out[nsh + s] = dh;
  out[2 * nsh + s] = qs * qs * qs / 3.0;
  if (cn) out[3 * nsh + s] = -cn[ia] * tr;
  if (zgrad) zgrad[s] = 0.0;  // accumulated by the Slater-exponent kernel that follows
}
__global__ void k_param_grad(DevMol m, Gfn2Scalars p, const double* __restrict__ P,
                             const double* __restrict__ Hp, const double* __restrict__ qsh,
                             double* out /* [3][nsh]: dse, dhub, dgam3 */) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= m.nsh) return;
  param_grad_dev(m, P, Hp, nullptr, nullptr, nullptr, qsh, out, nullptr, s);
  (void)p;
}
void launch_param_grad(const DevMol& m, const Gfn2Scalars& p, const double* P, const double* Hp,
                       const double* qsh, double* out, cudaStream_t s) {
  ++g_kernel_launches;
  k_param_grad<<<(m.nsh + 127) / 128, 128, 0, s>>>(m, p, P, Hp, qsh, out);
}

// ------------------------------------------------------------------------------------
// Batched launches: blockIdx.z walks the listed molecules; each block runs the same body as
// the one-molecule kernel on that molecule's slices.  Blocks past a molecule's own size exit
// through the bodies' bounds checks (or the explicit tile checks below).
// ------------------------------------------------------------------------------------
#define BMOL const MolPtrs& q = mp[list[blockIdx.z]]
#define BARGS const MolPtrs* __restrict__ mp, const int* __restrict__ list

__global__ void kb_param_grad(BARGS) {
  BMOL;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (!q.param_grad || s >= q.m.nsh) return;
  param_grad_dev(q.m, q.P, nullptr, q.H, q.se, q.cn, q.qsh_o, q.pgrad, q.zgrad, s);
}
static inline dim3 bgrid(unsigned x, const BatchLaunch& b, unsigned y = 1);
void launch_param_grad_b(const BatchLaunch& b) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_param_grad<<<bgrid((b.nsh_max + 127) / 128, b), 128, 0, b.s>>>(b.mp, b.list);
}
static inline dim3 bgrid(unsigned x, const BatchLaunch& b, unsigned y) {
  return dim3(x > 0 ? x : 1, y, (unsigned)b.count);
}

__global__ void kb_cn(BARGS, Gfn2Scalars p) {
  BMOL;
  cn_dev(q.m, p, q.cn);
}
void launch_cn_b(const BatchLaunch& b, const Gfn2Scalars& p) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_cn<<<bgrid((b.nat_max * 32 + 63) / 64, b), 64, 0, b.s>>>(b.mp, b.list, p);
}

__global__ void kb_cn_grad(BARGS, Gfn2Scalars p) {
  BMOL;
  if (q.m.nat == 1) return;
  cn_grad_dev(q.m, p, q.dEdcn, q.grad, q.sig_at);
}
void launch_cn_grad_b(const BatchLaunch& b, const Gfn2Scalars& p) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_cn_grad<<<bgrid((b.nat_max * 32 + 63) / 64, b), 64, 0, b.s>>>(b.mp, b.list, p);
}

__global__ void kb_levels(BARGS, Gfn2Scalars p) {
  BMOL;
  levels_dev(q.m, p, q.cn, q.se, q.mrad, q.dmrdcn);
}
void launch_setup_levels_b(const BatchLaunch& b, const Gfn2Scalars& p) {
  if (!b.count) return;
  const int nt = b.nsh_max > b.nat_max ? b.nsh_max : b.nat_max;
  ++g_kernel_launches;
  kb_levels<<<bgrid((nt + 127) / 128, b), 128, 0, b.s>>>(b.mp, b.list, p);
}

__global__ void kb_coulomb_table(BARGS, Gfn2Scalars p) {
  BMOL;
  coulomb_table_dev(q.m, p, q.mrad, q.ctab);
}
void launch_coulomb_table_b(const BatchLaunch& b, const Gfn2Scalars& p) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_coulomb_table<<<bgrid((b.nat_max * 32 + 63) / 64, b), 64, 0, b.s>>>(b.mp, b.list, p);
}

template <int MODE>
__global__ void kb_coulomb(BARGS, Gfn2Scalars p) {
  BMOL;
  if (MODE == 0)
    coulomb_potential_dev(q.m, p, q.mrad, q.qsh, q.qat, q.dpat, q.qpat, q.vsh, q.vat, q.vdp,
                          q.vqp, q.ctab);
  else
    coulomb_energy_dev(q.m, p, q.mrad, q.qsh_o, q.qat_o, q.dpat_o, q.qpat_o, q.eelec, q.ctab);
}
void launch_coulomb_potential_b(const BatchLaunch& b, const Gfn2Scalars& p) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_coulomb<0><<<bgrid((b.nat_max * 32 + 63) / 64, b), 64, 0, b.s>>>(b.mp, b.list, p);
}
void launch_coulomb_energy_b(const BatchLaunch& b, const Gfn2Scalars& p) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_coulomb<1><<<bgrid((b.nat_max * 32 + 63) / 64, b), 64, 0, b.s>>>(b.mp, b.list, p);
}

__global__ void kb_coulomb_grad(BARGS, Gfn2Scalars p) {
  BMOL;
  if (q.m.nat == 1) return;
  coulomb_grad_dev(q.m, p, q.mrad, q.dmrdcn, q.qsh_o, q.qat_o, q.dpat_o, q.qpat_o, q.grad,
                   q.sig_at, q.dEdcn);
}
void launch_coulomb_gradient_b(const BatchLaunch& b, const Gfn2Scalars& p) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_coulomb_grad<<<bgrid((b.nat_max * 32 + 63) / 64, b), 64, 0, b.s>>>(b.mp, b.list, p);
}

__global__ void kb_repulsion(BARGS, Gfn2Scalars p) {
  BMOL;
  repulsion_dev(q.m, p, q.erep, q.grad, q.sig_at);
}
void launch_repulsion_b(const BatchLaunch& b, const Gfn2Scalars& p) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_repulsion<<<bgrid((b.nat_max * 32 + 63) / 64, b), 64, 0, b.s>>>(b.mp, b.list, p);
}

__global__ void kb_vao(BARGS) {
  BMOL;
  vao_dev(q.m, q.vsh, q.vat, q.vao);
}
void launch_vao_b(const BatchLaunch& b) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_vao<<<bgrid((b.nao_max + 255) / 256, b), 256, 0, b.s>>>(b.mp, b.list);
}

__global__ void __launch_bounds__(256) kb_fock(BARGS) {
  BMOL;
  const int n = q.m.nao;
  if ((int)blockIdx.x * 32 >= n || (int)blockIdx.y * 32 >= n) return;  // tile outside
  fock_dev(n, q.m.ao_at, q.H, q.S, q.with_mp ? q.D : nullptr, q.Q, q.vao, q.vdp, q.vqp, q.F);
}
void launch_fock_b(const BatchLaunch& b) {
  if (!b.count) return;
  const unsigned nt = (b.nao_max + 31) / 32;
  ++g_kernel_launches;
  kb_fock<<<bgrid(nt, b, nt), dim3(32, 8), 0, b.s>>>(b.mp, b.list);
}

__global__ void __launch_bounds__(128) kb_mull_partial(BARGS) {
  BMOL;
  if ((int)blockIdx.y >= q.mull_chunks) return;
  mull_partial_dev<1>(q.m.nao, mull_rows(q.m.nao), q.P, q.S, q.H, q.D, q.Q, q.mull);
}
__global__ void kb_mull_reduce(BARGS) {
  BMOL;
  mull_reduce_dev(q.m, q.mull, q.mull_chunks, q.qsh_o, q.qat_o, q.dpat_o, q.qpat_o, q.eband);
}
void launch_mulliken_b(const BatchLaunch& b) {
  if (!b.count) return;
  ++g_kernel_launches;
  // (the molecules of up to 512 orbitals in a wider bucket have the shorter chunks)
  const int chunks = std::max(mulliken_chunks(b.nao_max), mulliken_chunks(std::min(b.nao_max, 512)));
  kb_mull_partial<<<bgrid((b.nao_max + 127) / 128, b, chunks), 128, 0,
                    b.s>>>(b.mp, b.list);
  ++g_kernel_launches;
  kb_mull_reduce<<<bgrid((b.nat_max * MULL_LANES + 127) / 128, b), 128, 0, b.s>>>(b.mp, b.list);
}

__global__ void kb_fermi(BARGS) {
  BMOL;
  const int n = q.m.nao;
  fermi_dev(n, q.emo, q.nalp, q.nbet, q.kt, q.focc + n, q.focc + 2 * n, q.focc, q.scal, q.icount,
            q.nev);
  // too few levels computed for this Fermi level: the molecule leaves for the one-molecule path
  if (threadIdx.x == 0 && q.icount[1] != 0) *q.flag = -3;
}
void launch_fermi_b(const BatchLaunch& b) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_fermi<<<bgrid(1, b), one_block(b.nao_max), 0, b.s>>>(b.mp, b.list);
}

__global__ void kb_pack(BARGS, int output) {
  BMOL;
  const int nmp = q.with_mp ? q.m.nat : 0;
  if (output)
    pack_dev(q.m.nsh, nmp, q.qsh_o, q.dpat_o, q.qpat_o, q.vec_out);
  else
    pack_dev(q.m.nsh, nmp, q.qsh, q.dpat, q.qpat, q.bq);
}
void launch_pack_b(const BatchLaunch& b, bool output) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_pack<<<bgrid((b.nd_max + 255) / 256, b), 256, 0, b.s>>>(b.mp, b.list, output ? 1 : 0);
}

__global__ void kb_unpack(BARGS) {
  BMOL;
  unpack_dev(q.m, q.bq, q.qsh, q.qat, q.dpat, q.qpat, q.with_mp);
}
void launch_unpack_b(const BatchLaunch& b) {
  if (!b.count) return;
  const int nt = b.nsh_max > 6 * b.nat_max ? b.nsh_max : 6 * b.nat_max;
  ++g_kernel_launches;
  kb_unpack<<<bgrid((nt + 255) / 256, b), 256, 0, b.s>>>(b.mp, b.list);
}

__global__ void kb_diff(BARGS) {
  BMOL;
  diff_dev(q.nd, q.vec_out, q.bq, q.bdq, q.scal + 1);
}
void launch_diff_b(const BatchLaunch& b) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_diff<<<bgrid(1, b), one_block(b.nd_max), 0, b.s>>>(b.mp, b.list);
}

__global__ void kb_broyden(BARGS, int iter) {
  BMOL;
  broyden_dev(q.nd, q.memory, iter, q.damp, q.bq, q.bqlast, q.bdq, q.bdqlast, q.bdf, q.bu, q.ba,
              q.bomega, q.bwork, q.bstatus, false);
}
void launch_broyden_b(const BatchLaunch& b, int iter) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_broyden<<<bgrid(1, b), std::max(256, one_block(b.nd_max)), 0, b.s>>>(b.mp, b.list, iter);
}

__global__ void kb_eelec_init(BARGS) {
  BMOL;
  eelec_init_dev(q.m.nat, q.scal, q.eband, q.eelec);
}
void launch_eelec_init_b(const BatchLaunch& b) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_eelec_init<<<bgrid((b.nat_max + 127) / 128, b), 128, 0, b.s>>>(b.mp, b.list);
}

// convergence test of the single-point driver (xtb/singlepoint.f90:300-304), one thread per
// molecule: the electronic energy is summed in atom order, as the one-molecule driver does
__global__ void kb_converge(BARGS) {
  BMOL;
  if (threadIdx.x != 0 || *q.flag < 0) return;
  double e = 0.0;
  for (int i = 0; i < q.m.nat; ++i) e += q.eelec[i];
  const double elast = q.conv[1];
  q.conv[0] = elast;
  q.conv[1] = e;
  q.conv[2] = q.scal[1];
  if (*q.bstatus != 0) {
    *q.flag = -1;
    return;
  }
  const bool ok = fabs(e - elast) < q.econv && q.scal[1] < q.pconv;
  *q.flag = ok ? 1 : 0;
}
void launch_converge_b(const BatchLaunch& b) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_converge<<<bgrid(1, b), 32, 0, b.s>>>(b.mp, b.list);
}

__global__ void kb_fe(BARGS) {
  BMOL;
  fe_dev(q.m.nao, q.focc, q.emo, q.vec_out);
}
__global__ void kb_wbo(BARGS, int channel) {
  BMOL;
  if (q.wbo_ch <= channel) return;
  wbo_dev(q.m, q.scratch, q.wbo + (size_t)channel * q.m.nat * q.m.nat, q.wbo_ch == 2 ? 2.0 : 1.0);
}
void launch_wbo_b(const BatchLaunch& b, int channel) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_wbo<<<bgrid((unsigned)(((long long)b.nat_max * b.nat_max + 255) / 256), b), 256, 0, b.s>>>(
      b.mp, b.list, channel);
}

void launch_fe_b(const BatchLaunch& b) {
  if (!b.count) return;
  ++g_kernel_launches;
  kb_fe<<<bgrid((b.nao_max + 255) / 256, b), 256, 0, b.s>>>(b.mp, b.list);
}

#undef BMOL
#undef BARGS

}  // namespace tb
