// Pipelined FP64-accurate split GEMM on the BF16 tensor cores.
//
// Two splittings (struct Balanced, struct Magnitude).  Balanced: x = 2^e sum_p d_p 2^(-7 - 8p),
// p = 0..6, with digits d_p in [-128, 128]: seven slices in BF16, and the 28 slice products d_p d_q
// with p + q <= 6 (zero based).  Magnitude, the splitting of ozaki.cu: eight 7-bit digits of |x| with
// x's sign, 36 products with p + q <= 7.  Balanced radix-256 digits have the same magnitude bound
// (products <= 2^14, so as many of them sum exactly in FP32) and hold one bit more each, and what
// is rounded or dropped has no sign bias: 28 products instead of 36 and a smaller error (A A^T of
// 3072: 8.5e-16 against 1.2e-15).  The batch, the small products of one molecule (pgemm_pair) and
// tblite_gb300_split_gemm use Balanced.  The one-molecule projection (purify.cu) keeps Magnitude and
// with it its results: its bias loses 2e-10 electrons of 4000 (500 waters), which the dipole of a
// cluster far from the origin shows at 5e-10, so the splittings' results differ visibly there although both are within the solver's
// tolerance.  The operands are split once per matrix instead of once per tile pair, and the
// products are grouped so that each tensor-core instruction is wide (figures of Balanced;
// Magnitude in brackets where they differ):
//
//   psplit   turns a matrix into a slice image: per line (row of op(A) or column of op(B)) a
//            power-of-two exponent, and the BF16 slices laid out exactly as the tensor
//            cores read them from shared memory, K-major lines of 64 bytes with the 64-byte
//            swizzle: image[k chunk of 32][slice][line block of 64][64 x 64 bytes];
//   pgemm    (kernel k_opipe) one 128 x 64 output tile per CTA, 10 warps.  Warp 0 streams the
//            slices of each k chunk (84 KB: A 56 KB, B 28 KB) with cp.async.bulk into a
//            two-stage shared-memory ring (mbarrier complete_tx).  Warp 1 issues the MMAs: the B
//            slices of a stage lie one after another, so d_p times [d_q0 .. d_q0+3] is a single
//            M 128 x N 256 x K 16 tcgen05.mma whose four 64-column blocks land in the TMEM
//            accumulators of the levels p + q0 .. p + q0 + 3 (one accumulator of 64 columns per
//            level 0..6); 11 [12] MMAs per k step, first those of the levels below 4, then the
//            others.  Warps 2..9 drain the levels 0..4 [0..5] every 6 [5] chunks (192 [160] values
//            of k): they hold exact integers (at most 5 [6] products of <= 2^14 each per k: < 2^24)
//            that go into one int64 per element.  The levels 5..6 [6..7] (weight 2^-40 [2^-42] of
//            the leading level and a random sum of balanced digits) stay in FP32 over the whole of
//            k and are read with the output at the end.  Their rounding shows only where the digits
//            of long rows all have one sign: largest error of Balanced against |a| |b| at k = 3072
//            and 12288 4e-17 and 3e-17 for normal operands, 1.6e-16 and 2.3e-15 for constant ones
//            (Magnitude 9e-17 and 6e-17, 3.1e-16 and 1.1e-15; FP64 sums 6e-17 and 2e-17, 8e-15 and
//            9e-15).
//
// Bound by the tensor pipe (896 [1152] cycles per k step of 16) and by what does not run beside it:
// prologue, last drain and epilogue of a tile (one CTA per SM), and what is left of a window's drain
// (8 cycles per warp and conversion, about 3000 in all) when the other half's MMAs are done: the lower
// levels are drained under the window's last upper MMAs, the upper ones under the next window's
// first lower MMAs (A A^T of 3072 770 -> 697 us, a product of 3000 804 -> 668 us).  The drain's loads
// are issued one level ahead, level 0 (below 2^22) is converted by an FP32 addition instead.
//
// Every wait is bounded; a wait that runs out sets a CTA-wide abort flag, the other roles leave
// their loops, copies and MMAs still in flight are waited for (bounded), TMEM is freed and the
// status word is set.  Tiles are visited in groups of 8 row blocks so that the slices a wave of
// CTAs reads stay in L2.  Symmetric products compute the tiles on and below the diagonal and
// write each element also to its mirror position.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>
#include <type_traits>

#include "engine.h"

namespace tb {

namespace {

constexpr int PP_M = 128, PP_N = 64, PP_KC = 32, PP_THREADS = 320;
struct Balanced {
  static constexpr int SLICES = 7;  // BF16 slices of an operand
  static constexpr int LEVELS = 7;  // TMEM accumulators, one per level p + q
  static constexpr int EXACT = 5;   // levels 0 .. EXACT - 1 are drained as exact integers
  static constexpr int FLUSH = 6;   // k chunks per window
  static constexpr int BITS = 8;    // of a digit
};
struct Magnitude {
  static constexpr int SLICES = 8, LEVELS = 8, EXACT = 6, FLUSH = 5, BITS = 7;
};
// |int64 level sums| < 1.01 * 2^46 K (Balanced), 1.02 * 2^49 K (Magnitude): below 2^63
constexpr int PP_KMAX = 12288;
constexpr int PP_STAGES = 2;    // the producer's bookkeeping below assumes two
template <class Sch>
constexpr int PP_A_BYTES = Sch::SLICES * 8192;  // slices x 128 lines x 64 B
template <class Sch>
constexpr int PP_B_BYTES = Sch::SLICES * 4096;  // slices x 64 lines x 64 B
template <class Sch>
constexpr int PP_STAGE_BYTES = PP_A_BYTES<Sch> + PP_B_BYTES<Sch>;
template <class Sch>
constexpr int PP_SMEM = PP_STAGES * PP_STAGE_BYTES<Sch> + 1024;
constexpr int PP_TMEM_COLS = 512;
constexpr int PP_LOW = 4;  // levels 0 .. 3 are handed to the drain first
static_assert(Magnitude::LEVELS * PP_N <= PP_TMEM_COLS && Balanced::LEVELS * PP_N <= PP_TMEM_COLS,
              "one 64-column accumulator per level");
constexpr int PP_GROUP = 8;  // row blocks per tile group
constexpr int PP_WAIT = 1 << 22;
// polls of a pipeline wait (stage full / empty, accumulators ready / free) before it gives up
// and aborts the tile; the drains of copies and MMAs in flight after an abort always use
// PP_WAIT.  Settable for tests (tblite_gb300_set_pipeline_wait_limit) so that a wait runs out
// and the abort path, the status word and the hand-off can be checked.
__device__ int g_pipe_wait_limit = PP_WAIT;
// FP64-equivalent flop (2 m n K per output tile that ran) of the batched squarings since load
__device__ unsigned long long g_pipe_batch_flops = 0;

void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess)
    throw std::runtime_error(std::string("CUDA error '") + cudaGetErrorString(e) + "' in " + what);
}

__device__ __forceinline__ uint32_t su32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// shared-memory matrix descriptor (K-major, descriptor version 1): lines of 64 bytes (32 BF16 of
// k), 8-line atoms 512 B apart, the 16-byte chunks of line r permuted by chunk ^ ((r >> 1) & 3)
// (the 64-byte swizzle); a k step of 16 moves the start by 32 bytes
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait; gives up early once another role has aborted (abort != nullptr)
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort) {
  const int limit = abort ? g_pipe_wait_limit : PP_WAIT;
  for (int it = 0; it < limit; ++it) {
    if (try_wait(bar, parity)) return true;
    if (abort && *abort) return false;
  }
  return false;
}

// 32 consecutive TMEM columns of this thread's lane (one row of the tile) into v; tmem_wait before
// v is used
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
        "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr));
}
// waits for this thread's TMEM loads; the loaded registers pass through, so that no use of them
// moves above it
__device__ __forceinline__ void tmem_wait(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]),
                 "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]),
                 "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]), "+r"(v[17]),
                 "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]),
                 "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27])
               :
               : "memory");
  asm volatile("" : "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])::"memory");
}

// x 2^(55 - e), rounded: |x| < 2^e gives at most 2^55; zero and subnormals give zero
__device__ __forceinline__ long long fixed55(uint64_t bits, int e) {
  const int ex = (int)((bits >> 52) & 0x7FF);
  if (ex == 0) return 0ll;
  const uint64_t m = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int sh = ex - e - 1020;
  const uint64_t w = sh >= 0 ? m << sh : (sh > -64 ? ((m >> (-sh - 1)) + 1) >> 1 : 0ull);
  return (bits >> 63) ? -(long long)w : (long long)w;
}

// |x| 2^(56 - e) as an integer (< 2^56 for |x| < 2^e): zero and subnormals give zero
__device__ __forceinline__ uint64_t fixed_bits(uint64_t bits, int e) {
  const int ex = (int)((bits >> 52) & 0x7FF);
  if (ex == 0) return 0ull;
  const uint64_t m = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int sh = ex - e - 1019;
  return sh >= 0 ? m << sh : (sh > -64 ? m >> (-sh) : 0ull);
}

// a - b of two packed BF16 pairs (the bits of both), one BF16x2 instruction
__device__ __forceinline__ uint32_t bf16x2_sub(uint32_t a, uint32_t b) {
  union {
    uint32_t u;
    __nv_bfloat162 v;
  } x, y, r;
  x.u = a;
  y.u = b;
  r.v = __hsub2(x.v, y.v);
  return r.u;
}

// the balanced digits of two fixed-point values |W| <= 2^55 + 2^46 as packed BF16 pairs, w[p] =
// (digit p of W0, digit p of W1).  Adding 128 to every digit turns the digits into the bytes of one
// integer; a byte b gives the BF16 number 128 + (b & 127) by its mantissa field, and subtracting
// 128 (b >= 128) or 256 (b < 128) leaves the digit b - 128, both elements in one BF16x2 subtraction
// (exact: at most 8 significant bits).  The top digit + 128 may be 256: its lane then holds -128
// and the sign is cleared.
__device__ __forceinline__ void digits_pair(long long W0, long long W1,
                                            uint32_t (&w)[Balanced::SLICES]) {
  constexpr long long BIAS = 0x0080808080808080ll;
  const unsigned long long V0 = (unsigned long long)(W0 + BIAS), V1 = (unsigned long long)(W1 + BIAS);
  const uint32_t l0 = (uint32_t)V0, h0 = (uint32_t)(V0 >> 32), l1 = (uint32_t)V1,
                 h1 = (uint32_t)(V1 >> 32);
  // 16-bit lanes whose low byte is digit p of each element (the top digit: all 16 bits)
  const uint32_t R[Balanced::SLICES] = {__byte_perm(h0, h1, 0x7632), __byte_perm(h0, h1, 0x5511),
                                 __byte_perm(h0, h1, 0x4400), __byte_perm(l0, l1, 0x7733),
                                 __byte_perm(l0, l1, 0x6622), __byte_perm(l0, l1, 0x5511),
                                 __byte_perm(l0, l1, 0x4400)};
#pragma unroll
  for (int p = 0; p < Balanced::SLICES; ++p)
    w[p] = bf16x2_sub((R[p] & 0x007F007Fu) | 0x43004300u, (R[p] & 0x00800080u) ^ 0x43804380u);
  w[0] ^= (R[0] & 0x01000100u) << 7;
}
// the slices of two values x0, x1 (bits) of a line of exponent e: w[p] = (slice p of x0, of x1)
template <class Sch>
__device__ __forceinline__ void split_pair(uint64_t x0, uint64_t x1, int e,
                                           uint32_t (&w)[Sch::SLICES]) {
  if constexpr (Sch::SLICES == Balanced::SLICES) {
    digits_pair(fixed55(x0, e), fixed55(x1, e), w);
  } else {
    // digit p of |x| 2^(56 - e) is the 7-bit field at 49 - 7p, read from the 28-bit half that
    // holds it; 128 + digit by the mantissa field, minus 128, and the sign (a zero digit of a
    // negative element becomes -0, which adds nothing to a product)
    const uint32_t signs = (uint32_t)(x0 >> 63) << 15 | (uint32_t)(x1 >> 63) << 31;
    const uint64_t Y0 = fixed_bits(x0, e), Y1 = fixed_bits(x1, e);
    const uint32_t h0 = (uint32_t)(Y0 >> 28), l0 = (uint32_t)Y0 & 0xFFFFFFFu;
    const uint32_t h1 = (uint32_t)(Y1 >> 28), l1 = (uint32_t)Y1 & 0xFFFFFFFu;
    const uint32_t R[4] = {__byte_perm(h0 >> 14, h1 >> 14, 0x5410), __byte_perm(h0, h1, 0x5410),
                           __byte_perm(l0 >> 14, l1 >> 14, 0x5410), __byte_perm(l0, l1, 0x5410)};
#pragma unroll
    for (int p = 0; p < Sch::SLICES; ++p) {
      const uint32_t mag = ((R[p >> 1] >> ((p & 1) ? 0 : 7)) & 0x007F007Fu) | 0x43004300u;
      w[p] = bf16x2_sub(mag, 0x43004300u) | signs;
    }
  }
}

// |x| as bits: for non-negative doubles the unsigned order of the bit patterns is the numeric
// order, so line maxima are integer maxima (no FP64 instruction, which this GPU issues at 1/64
// of the FP32 rate); e = ilogb(max) + 1 is the biased exponent field minus 1022 for a normal
// maximum
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
}
__device__ __forceinline__ int exp_of_max(unsigned long long mb) {
  const int mexp = (int)(mb >> 52);
  return mb == 0ull ? 0 : mexp > 0 ? mexp - 1022 : ilogb(__longlong_as_double((long long)mb)) + 1;
}

// ---- exponents: e = ilogb(max |x|) + 1 of every line ------------------------------------------
// lines contiguous in memory (element (i, k) at M[i + k ld]): L lines per block, the T / L groups
// of threads take every (T / L)-th k (128-byte rows for L = 16), then a shared-memory reduction
template <int L, int T>
__device__ __forceinline__ void pexp_rows_dev(const double* __restrict__ M, int ld, int lines,
                                              int K, int Lp, int* e, int blk) {
  constexpr int G = T / L;
  __shared__ unsigned long long part[G][L + 1];
  const int li = threadIdx.x % L, kg = threadIdx.x / L;
  const int i = blk * L + li;
  unsigned long long mx = 0ull;
  if (i < lines) {
#pragma unroll 4
    for (int k = kg; k < K; k += G) mx = max(mx, abs_bits(M[i + (size_t)k * ld]));
  }
  part[kg][li] = mx;
  __syncthreads();
  if (kg == 0 && i < Lp) {
#pragma unroll 8
    for (int g = 1; g < G; ++g) mx = max(mx, part[g][li]);
    e[i] = exp_of_max(mx);
  }
}
// one matrix: 16 lines and 1024 threads per block keep enough loads in flight (3072 x 3072 with
// 32 lines and 256 threads took 57 us)
__global__ void __launch_bounds__(1024) k_pexp_rows(const double* __restrict__ M, int ld,
                                                   int lines, int K, int Lp, int* e) {
  pexp_rows_dev<16, 1024>(M, ld, lines, K, Lp, e, blockIdx.x);
}
// k contiguous (element (i, k) at M[k + i ld]): one warp per line
__global__ void k_pexp_cols(const double* __restrict__ M, int ld, int lines, int K, int Lp,
                            int* e) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= Lp) return;
  unsigned long long mx = 0ull;
  if (i < lines)
    for (int k = lane; k < K; k += 32) mx = max(mx, abs_bits(M[k + (size_t)i * ld]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) e[i] = exp_of_max(mx);
}

// ---- slice image: one block per (64 lines, 32 k); the FP64 tile goes through shared memory so
// both memory orders read coalesced; each thread splits 8 consecutive k of one line
template <class Sch>
__device__ __forceinline__ void psplit_dev(const double* __restrict__ M, int ld, int kcontig,
                                           int lines, int K, int nlb, int ei, uint16_t* img,
                                           int lb, int kc) {
  __shared__ double tile[64][33];
  const int t = threadIdx.x;
  const int l0 = lb * 64, k0 = kc * PP_KC;
  if (!kcontig) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int li = t & 63, kk = (t >> 6) + 4 * r;
      const int i = l0 + li, k = k0 + kk;
      tile[li][kk] = (i < lines && k < K) ? M[i + (size_t)k * ld] : 0.0;
    }
  } else {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int kk = t & 31, li = (t >> 5) + 8 * r;
      const int i = l0 + li, k = k0 + kk;
      tile[li][kk] = (i < lines && k < K) ? M[k + (size_t)i * ld] : 0.0;
    }
  }
  __syncthreads();
  const int li = t & 63, g = t >> 6;  // k group of 8: 0..3
  uint32_t w[Sch::SLICES][4];
#pragma unroll
  for (int c = 0; c < 8; c += 2) {  // two neighbouring k per step
    uint32_t g2[Sch::SLICES];
    split_pair<Sch>((uint64_t)__double_as_longlong(tile[li][8 * g + c]),
                    (uint64_t)__double_as_longlong(tile[li][8 * g + c + 1]), ei, g2);
#pragma unroll
    for (int p = 0; p < Sch::SLICES; ++p) w[p][c >> 1] = g2[p];
  }
  // [k chunk][slice][line block][64 lines x 64 B, 16-byte chunks swizzled]
#pragma unroll
  for (int p = 0; p < Sch::SLICES; ++p) {
    const size_t off = (((size_t)kc * Sch::SLICES + p) * nlb + lb) * 2048 + li * 32 +
                       ((g ^ ((li >> 1) & 3)) << 3);
    *reinterpret_cast<uint4*>(img + off) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
  }
}
template <class Sch>
__global__ void __launch_bounds__(256) k_psplit(const double* __restrict__ M, int ld, int kcontig,
                                                int lines, int K, int nlb,
                                                const int* __restrict__ e, uint16_t* img) {
  psplit_dev<Sch>(M, ld, kcontig, lines, K, nlb, e[blockIdx.x * 64 + (threadIdx.x & 63)], img,
                  blockIdx.x, blockIdx.y);
}

struct PipeArgs {
  const uint16_t* A;  // slice image of op(A) (lines = rows, nlbA line blocks of 64)
  const uint16_t* B;  // slice image of op(B) (lines = columns)
  const int* eA;
  const int* eB;
  int eshiftA;  // added to every exponent of A (scaling A by a power of two)
  int nlbA, nlbB;
  int M, N, nkc;  // nkc: k chunks of 32
  double* C;
  int ldc;
  int sym;
  int* status;
  // the projection iterate (opipe_tile<true>): C holds signed 64-bit fixed-point values in units
  // of 2^-SP2_FRAC instead of doubles (|D_ij| <= 1); sub2: C <- 2 C - product (the old element
  // read first), which turns D^2 into 2D - D^2 in place
  int sub2;
  // the slice image of the new iterate (lines_padded(N) lines, exponent SP2_E), the tile's partial
  // sums of it (three words) and the mark of an element out of range
  uint16_t* img;
  unsigned long long* part;
  int* bad;
};

// line exponent of every projection iterate: the spectrum of D stays in [0, 1], so every element
// has |x| <= 1 = 2^SP2_E (up to rounding) and the slices hold x to an absolute 2^-55 (an FP64
// iterate's own rounding is 2^-53 relative to its O(1) diagonal); an element at or above
// SP2_LIMIT stops the molecule.  During the projection the iterate lives in Y as signed 64-bit
// integers W = x 2^55 (SP2_FRAC fractional bits), which are the digits' source directly.
constexpr int SP2_E = 0;
constexpr int SP2_FRAC = 55 - SP2_E;
constexpr long long SP2_LIMIT = (1ll << 55) + (1ll << 46);           // the top digit reaches 128
constexpr long long SP2_BAD = (long long)0x8000000000000000ull;  // an element out of range

__device__ __forceinline__ int slice_off(int line, int k, int nlb) {
  // image[k chunk][slice][line block][64 lines x 32 k], 16-byte groups swizzled (slice 0)
  const int li = line & 63, g = (k >> 3) & 3;
  return (((k >> 5) * Balanced::SLICES) * nlb + (line >> 6)) * 2048 + li * 32 + ((g ^ ((li >> 1) & 3)) << 3) +
         (k & 7);
}


// C element (i, j) of a finished tile from the exact levels T (units of the last one, E), the two
// FP32 levels va and vb and the scale 2^sc: C = (T + F) 2^(sc - BITS E), F = va 2^-BITS + vb
// 2^(-2 BITS); the power of two goes into the exponent field by an integer add where the result
// stays normal: three FP64 operations per element (two conversions and an add)
template <class Sch>
__device__ __forceinline__ float low_levels(uint32_t va, uint32_t vb) {
  constexpr float f = 1.0f / (1 << Sch::BITS);
  return fmaf(__uint_as_float(vb), f, __uint_as_float(va)) * f;
}
template <class Sch>
__device__ __forceinline__ double tile_value(long long T, uint32_t va, uint32_t vb, int sc) {
  constexpr int U = Sch::BITS * (Sch::EXACT - 1);
  const double sum = (double)T + (double)low_levels<Sch>(va, vb);
  const long long sb = __double_as_longlong(sum);
  const int se = (int)((sb >> 52) & 0x7FF);
  if (sum == 0.0) return 0.0;
  if (se > 0 && se + (sc - U) > 0 && se + (sc - U) < 2047)
    return __longlong_as_double(sb + ((long long)(sc - U) << 52));
  return ldexp(sum, sc - U);  // subnormal or out-of-range result: the general path
}
// T + iv 2^sh for a level's integer sum
__device__ __forceinline__ long long add_level(long long T, int iv, int mul) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(iv), "r"(mul), "l"(T));
  return r;
}

// the squares of Y < 2^56 as a (2^56, 2^28, 1) limb triple: Y = h 2^28 + l, Y^2 = h^2 2^56 +
// 2 h l 2^28 + l^2 (every partial product below 2^56, so per-lane sums of up to 256 stay exact)
struct Sq3 {
  unsigned long long hh = 0ull, hl = 0ull, ll = 0ull;
  __device__ __forceinline__ void add(uint32_t h, uint32_t l) {
    hh += (unsigned long long)h * h;
    hl += (unsigned long long)h * l;
    ll += (unsigned long long)l * l;
  }
  // the 128-bit value hh 2^56 + hl 2^29 + ll
  __device__ __forceinline__ void value(unsigned long long& lo, unsigned long long& hi) const {
    lo = hh << 56;
    hi = hh >> 8;
    const unsigned long long m = hl << 29, mh = hl >> 35;
    lo += m;
    hi += mh + (lo < m ? 1ull : 0ull);
    lo += ll;
    hi += (lo < ll ? 1ull : 0ull);
  }
};
__device__ __forceinline__ void add128(unsigned long long& lo, unsigned long long& hi,
                                       unsigned long long l, unsigned long long h) {
  lo += l;
  hi += h + (lo < l ? 1ull : 0ull);
}

// the iterate's element W for its image: zero if it is out of range, and its square
__device__ __forceinline__ long long sp2_element(long long w, Sq3& sq, bool& over) {
  // magnitudes (an out-of-range element, including the marker, counts as zero and stops the
  // molecule) and their 28-bit halves
  const unsigned long long a = w < 0 ? 0ull - (unsigned long long)w : (unsigned long long)w;
  const bool bad = a >= (unsigned long long)SP2_LIMIT;
  over = over || bad;
  const unsigned long long m = bad ? 0ull : a;
  sq.add((uint32_t)(m >> 28), (uint32_t)m & 0xFFFFFFFu);
  return bad ? 0 : w;
}
// exact sums over the warp
__device__ __forceinline__ void sp2_warp_sums(long long& tr, unsigned long long& lo,
                                              unsigned long long& hi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    tr += __shfl_xor_sync(0xffffffffu, tr, o);
    add128(lo, hi, __shfl_xor_sync(0xffffffffu, lo, o), __shfl_xor_sync(0xffffffffu, hi, o));
  }
}

// rows and columns of tile b: groups of PP_GROUP row blocks, column blocks inside a group
__device__ __forceinline__ void tile_origin(int M, int N, int b, int& i0, int& j0) {
  const int mt = (M + PP_M - 1) / PP_M, nt = (N + PP_N - 1) / PP_N;
  const int gid = b / (PP_GROUP * nt);
  const int first = gid * PP_GROUP;
  const int gsize = min(mt - first, PP_GROUP);
  const int inner = b - gid * PP_GROUP * nt;
  i0 = (first + inner % gsize) * PP_M;
  j0 = (inner / gsize) * PP_N;
}
// a symmetric product skips the tiles strictly above the diagonal (mirrored from below it)
__device__ __forceinline__ bool tile_above(int i0, int j0) { return i0 + PP_M - 1 < j0; }

// one 128 x 64 output tile (number b in the grouped order) of the product a (FIXED: the
// projection's fixed-point epilogue, a.fixed set)
template <class Sch, bool FIXED = false>
__device__ __forceinline__ void opipe_tile(const PipeArgs& a, int b) {
  int i0, j0;
  tile_origin(a.M, a.N, b, i0, j0);
  if (a.sym && tile_above(i0, j0)) return;

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem =
      smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);  // 1 KB aligned stages
  __shared__ __align__(8) uint64_t full[PP_STAGES], empty[PP_STAGES], accf[2], accfree[2], fin;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  __shared__ long long s_tr[8];
  __shared__ unsigned long long s_lo[8], s_hi[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* abort = &abort_flag;

  if (tid == 0) {
    for (int s = 0; s < PP_STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&full[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&empty[s])));
    }
    for (int h = 0; h < 2; ++h) {  // 0: levels below PP_LOW, 1: the others
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&accf[h])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 256;" ::"r"(su32(&accfree[h])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&fin)));
    asm volatile("fence.mbarrier_init.release.cluster;");
    abort_flag = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(su32(&tmem_base)), "r"(PP_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  const int nkc = a.nkc;
  const int nwin = (nkc + Sch::FLUSH - 1) / Sch::FLUSH;

  if (warp == 0) {
    // ---- producer: one elected lane streams the slices of every k chunk
    if (lane == 0) {
      const int lbA = i0 / 64, lbB = j0 / 64;
      int last0 = -1, last1 = -1;  // last chunk issued into stage 0 / 1
      for (int c = 0; c < nkc; ++c) {
        const int s = c % PP_STAGES;
        if (c >= PP_STAGES &&
            !wait_bar(su32(&empty[s]), (uint32_t)(((c - PP_STAGES) / PP_STAGES) & 1), abort)) {
          if (!*abort) atomicExch(&abort_flag, 1);
          break;
        }
        const uint32_t bar = su32(&full[s]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"(PP_STAGE_BYTES<Sch>)
                     : "memory");
        unsigned char* st = smem + (size_t)s * PP_STAGE_BYTES<Sch>;
        {  // per slice: A 8 KB (two line blocks), B 4 KB
#pragma unroll 1
          for (int p = 0; p < Sch::SLICES; ++p) {
            const size_t blk = (size_t)c * Sch::SLICES + p;
            const uint16_t* srcA = a.A + (blk * a.nlbA + lbA) * 2048;
            const uint16_t* srcB = a.B + (blk * a.nlbB + lbB) * 2048;
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], "
                "%2, [%3];" ::"r"(su32(st + p * 8192)),
                "l"(srcA), "r"(8192), "r"(bar)
                : "memory");
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], "
                "%2, [%3];" ::"r"(su32(st + PP_A_BYTES<Sch> + p * 4096)),
                "l"(srcB), "r"(4096), "r"(bar)
                : "memory");
          }
        }
        if (s == 0) last0 = c;
        else last1 = c;
      }
      // copies still in flight complete on their own; wait for them before the CTA ends
      if (last0 >= 0) wait_bar(su32(&full[0]), (uint32_t)((last0 / PP_STAGES) & 1), nullptr);
      if (last1 >= 0) wait_bar(su32(&full[1]), (uint32_t)((last1 / PP_STAGES) & 1), nullptr);
    }
  } else if (warp == 1) {
    // ---- MMA issuer
    if (lane == 0) {
      // instruction descriptor: FP32 accumulator, BF16 A and B (K-major), M 128, N set below
      const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(PP_M >> 4) << 24);
      for (int c = 0; c < nkc; ++c) {
        const int s = c % PP_STAGES;
        const int win = c / Sch::FLUSH;
        const bool win_start = (c % Sch::FLUSH) == 0;
        const bool win_end = (c % Sch::FLUSH) == Sch::FLUSH - 1 || c == nkc - 1;
        if (!wait_bar(su32(&full[s]), (uint32_t)((c / PP_STAGES) & 1), abort) ||
            (win_start && win > 0 &&
             !wait_bar(su32(&accfree[0]), (uint32_t)((win - 1) & 1), abort))) {
          atomicExch(&abort_flag, 1);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t stA = su32(smem + (size_t)s * PP_STAGE_BYTES<Sch>);
        const uint32_t stB = stA + PP_A_BYTES<Sch>;
        // groups (A slice p, first B slice q0, B slices nq), first those of the levels below
        // PP_LOW, then the others: the drain of either half runs under the MMAs of the other.  At
        // the start of a window slice 0, which covers every level, overwrites the exact levels;
        // the FP32 levels go on (overwritten only by the very first MMA of the tile).  The groups
        // are known at compile time, so the issue is a straight sequence: descriptors
        // are the stage's base descriptors plus constants (the start-address field holds
        // address / 16; every address stays inside the stage)
        const uint64_t dA = sdesc_sw64(stA), dB = sdesc_sw64(stB);
        auto mma = [&](int ks, int pg, int q0, int nq, uint32_t acc) {
          const uint32_t idesc = idesc0 | ((uint32_t)((nq * PP_N) >> 3) << 17);
          const uint64_t da = dA + (uint64_t)((pg * 8192 + ks * 32) >> 4);
          const uint64_t db = dB + (uint64_t)((q0 * 4096 + ks * 32) >> 4);
          asm volatile(
              "{\n\t.reg .pred pd;\n\tsetp.ne.b32 pd, %4, 0;\n\t"
              "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, pd;\n\t}" ::"r"(
                  tmem + (uint32_t)((pg + q0) * PP_N)),
              "l"(da), "l"(db), "r"(idesc), "r"(acc));
        };
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
#pragma unroll
          for (int p = 0; p < PP_LOW; ++p)
            mma(ks, p, 0, PP_LOW - p, p == 0 && ks == 0 && win_start ? 0u : 1u);
        }
        auto commit = [&](uint64_t* bar) {
          asm volatile(
              "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                  su32(bar))
              : "memory");
        };
        if (win_end) commit(&accf[0]);
        if (win_start && win > 0) {
          if (!wait_bar(su32(&accfree[1]), (uint32_t)((win - 1) & 1), abort)) {
            atomicExch(&abort_flag, 1);
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
        }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
          if (ks == 0 && win_start) {
            mma(ks, 0, PP_LOW, Sch::EXACT - PP_LOW, 0u);
            mma(ks, 0, Sch::EXACT, Sch::LEVELS - Sch::EXACT, c == 0 ? 0u : 1u);
          } else {
            mma(ks, 0, PP_LOW, Sch::LEVELS - PP_LOW, 1u);
          }
#pragma unroll
          for (int p = 1; p < Sch::SLICES; ++p) {
            const int q = p < PP_LOW ? PP_LOW - p : 0;
            mma(ks, p, q, Sch::LEVELS - p - q, 1u);
          }
        }
        commit(&empty[s]);
        if (win_end) commit(&accf[1]);
      }
      // every MMA issued so far has completed before TMEM is read for the last time or freed
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
              su32(&fin))
          : "memory");
      wait_bar(su32(&fin), 0u, nullptr);
    }
  } else {
    // ---- epilogue warps 2..9: TMEM lane quarter warp % 4, column half (warp - 2) / 4
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int row = 32 * quarter + lane;
    long long T[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) T[c] = 0;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(32 * half);
    bool ok = true, mirror = false;
    // the exact levels LO .. HI - 1 of a window into T; the next level's load is in flight while a
    // level is converted
    auto drain = [&](auto lo, auto hi) {
      constexpr int LO = decltype(lo)::value, HI = decltype(hi)::value;
      asm volatile("tcgen05.fence::after_thread_sync;");
      uint32_t va[32], vb[32];
      tmem_ld32(lane_base + (uint32_t)(LO * PP_N), va);
      tmem_wait(va);
#pragma unroll
      for (int lv = LO; lv < HI; ++lv) {
        uint32_t(&v)[32] = ((lv - LO) & 1) ? vb : va;
        uint32_t(&vn)[32] = ((lv - LO) & 1) ? va : vb;
        if (lv + 1 < HI) tmem_ld32(lane_base + (uint32_t)((lv + 1) * PP_N), vn);
#pragma unroll
        for (int t = 0; t < 32; ++t) {
          const float f = __uint_as_float(v[t]);
          if (lv == 0) {  // |f| <= 192 * 2^14 < 2^22: read off the sum with 1.5 * 2^23
            const int iv = (int)(__float_as_uint(f + 12582912.f) - 0x4B400000u);
            T[t] = (long long)((unsigned long long)T[t] +
                               ((unsigned long long)(long long)iv << (Sch::BITS * (Sch::EXACT - 1))));
          } else {
            T[t] = add_level(T[t], __float2int_rn(f), 1 << (Sch::BITS * (Sch::EXACT - 1 - lv)));
          }
        }
        if (lv + 1 < HI) tmem_wait(vn);
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
    };
    for (int w = 0; w < nwin && ok; ++w) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        // warp-uniform decision: the TMEM loads are .sync.aligned
        const bool got = wait_bar(su32(&accf[h]), (uint32_t)(w & 1), abort);
        if (!__all_sync(0xffffffffu, got ? 1 : 0)) {
          atomicExch(&abort_flag, 1);
          ok = false;
          break;
        }
        if (h == 0) drain(std::integral_constant<int, 0>(), std::integral_constant<int, PP_LOW>());
        else drain(std::integral_constant<int, PP_LOW>(), std::integral_constant<int, Sch::EXACT>());
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(&accfree[h])) : "memory");
      }
    }
    if (__all_sync(0xffffffffu, (ok && !*abort) ? 1 : 0)) {
      // C = 2^(eA + eB - 14) (T + F) 2^(-BITS (EXACT - 1)).  A symmetric product's mirror image
      // goes through shared memory (the stages are free: every copy and MMA of the tile has
      // completed), so that both triangles are written in full sectors
      const int i = i0 + row;
      const int ei = i < a.M ? a.eA[i] + a.eshiftA : 0;
      long long* mir = reinterpret_cast<long long*>(smem);  // [PP_N][PP_M + 1]
      uint32_t v5[32], v6[32];
      tmem_ld32(lane_base + (uint32_t)(Sch::EXACT * PP_N), v5);
      tmem_ld32(lane_base + (uint32_t)((Sch::EXACT + 1) * PP_N), v6);
      tmem_wait(v5);
      tmem_wait(v6);
      if constexpr (FIXED) {
        // the projection iterate in fixed point: the product is (T + F) 2^(sc - 32) with
        // sc = 2 SP2_E - 14, i.e. W = (T + F) 2^9 in units of 2^-55 (F rounded to an
        // integer there: an absolute 2^-56); |T| < 2^53 keeps T 2^9 exact, else the element is
        // marked out of range
        long long* W = reinterpret_cast<long long*>(a.C);
        static_assert(2 * SP2_E - 14 - Sch::BITS * (Sch::EXACT - 1) + SP2_FRAC == 9,
                      "fixed-point scale of the product");
#pragma unroll
        for (int t8 = 0; t8 < 32; t8 += 8) {
          long long old[8];
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const int j = j0 + 32 * half + t8 + t;
            old[t] = (a.sub2 && j < a.N && i < a.M && i >= j) ? W[i + (size_t)j * a.ldc] : 0ll;
          }
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            const int jl = 32 * half + t8 + t, j = j0 + jl;
            const long long tv = T[t8 + t];
            const float ff = low_levels<Sch>(v5[t8 + t], v6[t8 + t]) * 0x1p9f;
            // unsigned arithmetic: wrap-around instead of undefined overflow, and the
            // out-of-range cases are replaced below
            unsigned long long w =
                ((unsigned long long)tv << 9) + (unsigned long long)(long long)__float2int_rn(ff);
            if (a.sub2) w = 2ull * (unsigned long long)old[t] - w;
            if (tv >= (1ll << 53) || tv <= -(1ll << 53) || fabsf(ff) >= 0x1p30f ||
                old[t] == SP2_BAD)
              w = (unsigned long long)SP2_BAD;
            if (i < a.M && j < a.N && i >= j) W[i + (size_t)j * a.ldc] = (long long)w;
            mir[jl * (PP_M + 1) + row] = (long long)w;
          }
        }
      } else {
#pragma unroll
        for (int t = 0; t < 32; ++t) {
          const int jl = 32 * half + t, j = j0 + jl;
          const bool in = i < a.M && j < a.N;
          const double val = in ? tile_value<Sch>(T[t], v5[t], v6[t], ei + a.eB[j] - 14) : 0.0;
          if (in && !(a.sym && i < j)) a.C[i + (size_t)j * a.ldc] = val;
          if (a.sym) mir[jl * (PP_M + 1) + row] = __double_as_longlong(val);
        }
      }
      if (FIXED || a.sym) {
        // rows of the mirror image: 16 per warp, two columns of the tile per lane.  All eight
        // epilogue warps take this branch or none does, unless a wait ran out in one of them:
        // the abort flag is read again behind a barrier that every one of them passes
        mirror = true;
      }
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (!FIXED && __all_sync(0xffffffffu, (mirror && !*abort) ? 1 : 0)) {
      const long long* mir = reinterpret_cast<const long long*>(smem);
      long long* W = reinterpret_cast<long long*>(a.C);
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const int r = (warp - 2) * 16 + k, i = i0 + r;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int jl = lane + 32 * h, j = j0 + jl;
          if (i < a.M && j < a.N && i > j) W[j + (size_t)i * a.ldc] = mir[jl * (PP_M + 1) + r];
        }
      }
    }
    if constexpr (FIXED) {
      // The slice image of the new iterate, from the tile in shared memory: the lines i of the tile
      // (k = its columns) and, for the blocks of 64 strictly below the diagonal, the lines j (k =
      // its rows); of the block on the diagonal the elements on and below it, and their mirror
      // images.  A block above the diagonal belongs to another tile.  Four lanes per line and
      // chunk of 32, eight elements each, so that a warp writes eight whole lines.  A separate
      // kernel read the iterate back for this: 24 of 224 ms of a 1024-molecule ensemble, and a
      // launch per step (243 -> 237 ms in all, the squarings with the slices taking longer).
      long long tr = 0;
      Sq3 sq;
      bool over = false;
      if (__all_sync(0xffffffffu, (mirror && !*abort) ? 1 : 0)) {
        const long long* mir = reinterpret_cast<const long long*>(smem);
        const int g = lane & 3, cb = j0 / 64;
        auto piece = [&](int line, int kc, auto element) {
          const int k0 = 32 * kc + 8 * g;
          uint32_t w[Sch::SLICES][4];
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
            long long x[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              x[e] = sp2_element(element(k0 + c + e), sq, over);
              if (k0 + c + e == line) tr = x[e];  // (one line per lane holds its diagonal here)
            }
            uint32_t t[Sch::SLICES];
            digits_pair(x[0], x[1], t);
#pragma unroll
            for (int p = 0; p < Sch::SLICES; ++p) w[p][c >> 1] = t[p];
          }
          const int li = line & 63;
#pragma unroll
          for (int p = 0; p < Sch::SLICES; ++p)
            *reinterpret_cast<uint4*>(
                a.img + (((size_t)kc * Sch::SLICES + p) * a.nlbA + (line >> 6)) * 2048 + li * 32 +
                ((g ^ ((li >> 1) & 3)) << 3)) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
        };
#pragma unroll 1
        for (int u = (warp - 2) * 8 + (lane >> 2); u < 2 * PP_M; u += 64) {  // lines of rows
          const int r = u & (PP_M - 1), i = i0 + r, kc = j0 / 32 + u / PP_M, rb = i >> 6;
          if (rb < cb || kc >= nkc) continue;
          piece(i, kc, [&](int k) {
            // on the diagonal block an element above the diagonal is the one below it
            return rb == cb && k > i ? mir[(i - j0) * (PP_M + 1) + (k - i0)]
                                     : mir[(k - j0) * (PP_M + 1) + r];
          });
        }
#pragma unroll 1
        for (int u = (warp - 2) * 8 + (lane >> 2); u < 4 * PP_N; u += 64) {  // lines of columns
          const int jl = u & (PP_N - 1), j = j0 + jl, kc = i0 / 32 + u / PP_N;
          if ((kc >> 1) <= cb || kc >= nkc) continue;
          piece(j, kc, [&](int k) { return mir[jl * (PP_M + 1) + (k - i0)]; });
        }
      }
      unsigned long long lo, hi;
      sq.value(lo, hi);
      sp2_warp_sums(tr, lo, hi);
      if (__any_sync(0xffffffffu, over ? 1 : 0) && lane == 0) *a.bad = 1;
      if (lane == 0) {
        s_tr[warp - 2] = tr;
        s_lo[warp - 2] = lo;
        s_hi[warp - 2] = hi;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (tid == 0 && abort_flag) atomicExch(a.status, 1);
  if constexpr (FIXED) {
    if (tid == 0) {  // exact integers
      long long t = 0;
      unsigned long long lo = 0ull, hi = 0ull;
      for (int u = 0; u < 8; ++u) {
        t += s_tr[u];
        add128(lo, hi, s_lo[u], s_hi[u]);
      }
      a.part[0] = (unsigned long long)t;
      a.part[1] = lo;
      a.part[2] = hi;
    }
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(PP_TMEM_COLS));
}
template <class Sch>
__global__ void __launch_bounds__(PP_THREADS, 1) k_opipe(PipeArgs a) {
  opipe_tile<Sch>(a, blockIdx.x);
}

// ---- batched spectral projection on the pipe, one launch per step for every molecule of the
// list still iterating (blockIdx.y / blockIdx.z walks the molecules): kb_opipe_sq squares the
// iterate D_k from its slice image and writes D_(k+1) = D_k^2, or 2 D_k - D_k^2 (the old element
// read first), over D_k in Y (on and below the diagonal), and the slice image of D_(k+1) (every line exponent SP2_E) into the
// other of the molecule's two images, with the tile's partial sums of its trace and of its squared
// elements; its last block takes the next decision.  Molecules that left the batch or whose
// projection has converged (sp2i[0] != 0) launch nothing.
__device__ __forceinline__ int lines_padded(int n) { return ((n + PP_M - 1) / PP_M) * PP_M; }
__device__ __forceinline__ int sq_tiles(int n) {
  return ((n + PP_M - 1) / PP_M) * ((n + PP_N - 1) / PP_N);
}
// partial-sum slots of a molecule: one per block of kb_sp2_init (8 lines) and one per tile
__host__ __device__ __forceinline__ int sp2_slots(int n) {
  const int mt = (n + PP_M - 1) / PP_M, nt = (n + PP_N - 1) / PP_N;
  return mt * (nt > PP_M / 8 ? nt : PP_M / 8);
}
// the image that holds the iterate after `steps` steps
__device__ __forceinline__ uint16_t* sp2_image(const MolPtrs& q, int steps) {
  return (steps & 1) ? q.img2 : q.img;
}

// The decision at a new iterate D, taken by one warp after every partial sum of D is written (the
// slots 0 .. nslots - 1, without those of the tiles above the diagonal if they are tiles): tr D
// and tr D^2 = sum of the squares of D's elements (D is symmetric) exactly in 128-bit integers,
// read past L1 since other CTAs wrote them; then the idempotency error
// tr(D - D^2), the stop test (the error no longer falls over two steps, Kruchinin, Rubensson,
// Niklasson 2016, or reaches the rounding floor) and the update D^2 or 2D - D^2 whose trace is
// closer to the occupied count (Niklasson 2002).  State: sp2i[0] converged, [1] steps taken,
// [2] update of the next step (1 square, 0 2D - D^2, -1 none), [3] pipeline status; sp2s[2..4]
// the last three idempotency errors, [4] set by a block that met an element outside the
// fixed-point range (the molecule leaves).
__device__ void sp2_decide(const MolPtrs& q, int nslots, bool tiles) {
  // tr D 2^55 as a signed 128-bit sum of the blocks' int64 sums, tr D^2 2^110 unsigned
  const int lane = threadIdx.x & 31;
  unsigned long long tlo = 0ull, thi_ = 0ull, slo = 0ull, shi = 0ull;
  for (int t = lane; t < nslots; t += 32) {
    if (tiles) {
      int i0, j0;
      tile_origin(q.m.nao, q.m.nao, t, i0, j0);
      if (tile_above(i0, j0)) continue;
    }
    const unsigned long long* pt = q.sp2p + 3 * t;
    const long long tv = (long long)__ldcg(pt);
    add128(tlo, thi_, (unsigned long long)tv, tv < 0 ? ~0ull : 0ull);
    add128(slo, shi, __ldcg(pt + 1), __ldcg(pt + 2));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    add128(tlo, thi_, __shfl_xor_sync(0xffffffffu, tlo, o), __shfl_xor_sync(0xffffffffu, thi_, o));
    add128(slo, shi, __shfl_xor_sync(0xffffffffu, slo, o), __shfl_xor_sync(0xffffffffu, shi, o));
  }
  if (lane != 0) return;
  const long long thi = (long long)thi_;
  const double tx = ((double)thi * 0x1p64 + (double)tlo) * 0x1p-55;
  const double tx2 = ((double)shi * 0x1p64 + (double)slo) * 0x1p-110;
  const int n = q.m.nao;
  if (q.sp2i[3] != 0) {  // a tensor-core wait ran out: the molecule takes the one-molecule path
    *q.flag = -5;
    return;
  }
  if (q.sp2i[4] != 0) {  // an element outside the fixed-point range
    *q.flag = -6;
    return;
  }
  const double e = tx - tx2;
  const int k = q.sp2i[1];
  const double ekm2 = q.sp2s[3];  // after the shift below: e(k-2)
  q.sp2s[2] = q.sp2s[3];
  q.sp2s[3] = q.sp2s[4];
  q.sp2s[4] = e;
  const bool done = (k >= 2 && ekm2 < 1e-4 * n && e >= ekm2) || e <= 1e-15 * n;
  if (done) {
    q.sp2i[0] = 1;
    q.sp2i[2] = -1;
    return;
  }
  const double nocc = q.nalp;
  q.sp2i[2] = fabs(tx2 - nocc) <= fabs(2.0 * tx - tx2 - nocc) ? 1 : 0;
  q.sp2i[1] = k + 1;
}
// the last of `units` CTAs of a molecule to finish takes the decision (no separate launch):
// after the CTA's barrier one thread fences (cumulatively, the stores its barrier ordered before
// it) and counts the finished units; the CTA that completes the count decides and resets it
__device__ __forceinline__ void sp2_last_decides(const MolPtrs& q, int units, int nslots,
                                                 bool tiles) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(q.sp2i + 5, 1) == units - 1;
  }
  __syncthreads();
  if (!last || threadIdx.x >= 32) return;
  __threadfence();
  sp2_decide(q, nslots, tiles);
  if (threadIdx.x == 0) q.sp2i[5] = 0;
}
__device__ __forceinline__ bool sq_skip(const MolPtrs& q) {
  return *q.flag < 0 || q.sp2i[0] != 0;
}
__global__ void __launch_bounds__(PP_THREADS, 1) kb_opipe_sq(const MolPtrs* __restrict__ mp,
                                                            const int* __restrict__ list) {
  const MolPtrs& q = mp[list[blockIdx.y]];
  const int n = q.m.nao;
  const int tiles = sq_tiles(n);
  if (sq_skip(q) || (int)blockIdx.x >= tiles) return;
  int i0, j0;
  tile_origin(n, n, blockIdx.x, i0, j0);
  if (tile_above(i0, j0)) return;
  // read by every tile before the last one to finish changes them
  const int steps = q.sp2i[1] - 1;  // of the iterate to be squared (the decision counted this one)
  PipeArgs a{};
  a.A = a.B = sp2_image(q, steps);  // a symmetric matrix: its rows are its columns
  a.eA = a.eB = q.iexp;
  a.eshiftA = 0;
  a.nlbA = a.nlbB = lines_padded(n) / 64;
  a.M = a.N = n;
  a.nkc = (n + PP_KC - 1) / PP_KC;
  a.C = q.Y;  // D_(k+1) over D_k, fixed point
  a.ldc = n;
  a.sym = 1;
  a.status = q.sp2i + 3;
  a.sub2 = q.sp2i[2] == 0 ? 1 : 0;
  a.img = sp2_image(q, steps + 1);
  a.part = q.sp2p + 3 * blockIdx.x;
  a.bad = q.sp2i + 4;
  if (threadIdx.x == 0)  // the tile's useful area
    atomicAdd(&g_pipe_batch_flops, 2ull * (unsigned long long)min(PP_M, n - i0) *
                                       (unsigned long long)min(PP_N, n - j0) * (unsigned)n);
  opipe_tile<Balanced, true>(a, blockIdx.x);
  int units = 0;  // tiles on and below the diagonal: row block t has 2 t + 2 of them at most
  const int mt = (n + PP_M - 1) / PP_M, nt = (n + PP_N - 1) / PP_N;
  for (int t = 0; t < mt; ++t) units += min(2 * t + 2, nt);
  sp2_last_decides(q, units, tiles, true);
}

// ---- the first iterate and its decision: each warp owns one line i of D (column i in memory, which
// equals row i), D0 = (emax I - A) / (emax - emin), computed in FP64 and written to Y in fixed point
// (W = x 2^55).  Its slices (exponent SP2_E) go to img, and the line's diagonal element and the
// exact squares of its elements to the block's partial sums (exact integers); the last block of the
// molecule takes the decision.  A lane holds two neighbouring elements k, k + 1 of a 64-element
// segment (coalesced loads), so each slice plane gets one 32-bit word per lane.  Padding lines and
// positions get zero slices.
__global__ void __launch_bounds__(256) kb_sp2_init(const MolPtrs* __restrict__ mp,
                                                   const int* __restrict__ list) {
  const MolPtrs& q = mp[list[blockIdx.z]];
  const int n = q.m.nao, lp = lines_padded(n);
  if ((int)blockIdx.x * 8 >= lp || *q.flag < 0) return;  // uniform over the block
  const int i = (int)blockIdx.x * 8 + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const double emax = q.sp2s[1], f = 1.0 / (emax - q.sp2s[0]);
  const int nkc = (n + PP_KC - 1) / PP_KC, nlb = lp / 64;
  const size_t plane = (size_t)nlb * 2048;
  long long dw = 0;  // the line's diagonal element (an integer select per element)
  Sq3 sq;
  bool over = false;
  const double* __restrict__ am = q.A + (size_t)i * n;
  long long* __restrict__ y = reinterpret_cast<long long*>(q.Y) + (size_t)i * n;
  const bool real = i < n;
  for (int seg = 0; seg * 64 < nkc * PP_KC; ++seg) {
    const int k = seg * 64 + 2 * lane;
    if ((k >> 5) >= nkc) continue;  // the last segment may hold one chunk only
    long long w0 = 0, w1 = 0;
    if (real) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (k + e >= n) continue;
        const double x = ((k + e == i ? emax : 0.0) - am[k + e]) * f;
        const uint64_t bits = (uint64_t)__double_as_longlong(x);
        const long long w =
            ((bits >> 52) & 0x7FF) > (uint64_t)(1023 + SP2_E) ? SP2_BAD : fixed55(bits, SP2_E);
        y[k + e] = w;
        (e ? w1 : w0) = w;
      }
    }
    dw = k == i ? w0 : (k + 1 == i ? w1 : dw);
    const size_t off = (size_t)slice_off(i, k, nlb);
    uint32_t w[Balanced::SLICES];
    const long long x0 = sp2_element(w0, sq, over), x1 = sp2_element(w1, sq, over);
    digits_pair(x0, x1, w);
#pragma unroll
    for (int pp = 0; pp < Balanced::SLICES; ++pp)
      *reinterpret_cast<uint32_t*>(q.img + off + pp * plane) = w[pp];
  }
  if (lane == 0) q.iexp[i] = SP2_E;
  // block partial sums (exact integers): warp trees, then the warps in order
  __shared__ long long s_tr[8];
  __shared__ unsigned long long s_lo[8], s_hi[8];
  unsigned long long flo, fhi;
  sq.value(flo, fhi);
  sp2_warp_sums(dw, flo, fhi);  // (one lane holds the diagonal, the others 0)
  over = __any_sync(0xffffffffu, over ? 1 : 0) != 0;
  if (over && lane == 0) q.sp2i[4] = 1;
  const int w = threadIdx.x >> 5;
  if (lane == 0) {
    s_tr[w] = dw;
    s_lo[w] = flo;
    s_hi[w] = fhi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long t = 0;  // 8 lines of |W| < 2^56: no overflow
    unsigned long long lo = 0ull, hi = 0ull;
    for (int u = 0; u < 8; ++u) {
      t += s_tr[u];
      add128(lo, hi, s_lo[u], s_hi[u]);
    }
    unsigned long long* pt = q.sp2p + 3 * blockIdx.x;
    pt[0] = (unsigned long long)t;
    pt[1] = lo;
    pt[2] = hi;
  }
  sp2_last_decides(q, lp / 8, lp / 8, false);
}

// after a projection: the converged iterate from fixed point back to FP64 in place (the products
// P = 2 X D X^T read it as doubles); every listed molecule of the projection bucket.  The steps keep
// the triangle on and below the diagonal: 32 x 32 tiles of it go to both places, the mirror image
// through shared memory
__global__ void __launch_bounds__(256) kb_sp2_unfix(const MolPtrs* __restrict__ mp,
                                                    const int* __restrict__ list) {
  const MolPtrs& q = mp[list[blockIdx.z]];
  if (*q.flag < 0) return;
  __shared__ double tile[32][33];
  const int n = q.m.nao, nt = (n + 31) / 32, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long* w = reinterpret_cast<const long long*>(q.Y);
  for (int t = blockIdx.x; t < nt * (nt + 1) / 2; t += gridDim.x) {
    int ti = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
    while (ti * (ti + 1) / 2 > t) --ti;
    while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
    const int tj = t - ti * (ti + 1) / 2;
    const int i = 32 * ti + lane;
    __syncthreads();
    for (int c = wid; c < 32; c += 8) {
      const int j = 32 * tj + c;
      if (i >= n || j > i) continue;
      const size_t e = i + (size_t)j * n;
      const double x = w[e] == SP2_BAD ? __longlong_as_double(0x7FF8000000000000ll)
                                       : (double)w[e] * 0x1p-55;
      q.Y[e] = x;
      tile[c][lane] = x;
    }
    __syncthreads();
    for (int r = wid; r < 32; r += 8) {
      const int row = 32 * ti + r, j = 32 * tj + lane;  // element (row, j) to (j, row)
      if (row < n && j < row) q.Y[j + (size_t)row * n] = tile[lane][r];
    }
  }
}

// ---- batched GEMM sites on the pipe (projection buckets): the rows of op(A) go into img,
// the columns of op(B) into img2, then one product per molecule
struct SiteLines {
  const double* M;
  int ld, kcontig, lines, K;
};
__device__ __forceinline__ SiteLines site_lines(const Site& s, int which) {
  if (which == 0) return {s.A, s.ld, s.ta ? 1 : 0, s.M, s.K};
  return {s.B, s.ld, s.tb ? 0 : 1, s.N, s.K};
}
// exponents of the lines: 32 lines per block (lines strided in memory) or one warp per line
// (k contiguous); grid.x covers lines_padded / 8 blocks for the widest molecule
// which operand image of a site is already split: -1 none (split it), 0 / 1 one of X's two
// cached images (rows / columns of X), 2 the image of the projection's last iterate (op(B) = D
// of X D: D is symmetric, so its columns are the lines the image holds, exact for the fixed-point D)
__host__ __device__ __forceinline__ int site_ximage(int site, int which) {
  if (site == GS_FX) return which ? 1 : -1;   // B = X: its columns
  if (site == GS_XTT) return which ? -1 : 1;  // A = X^T: rows of X^T are columns of X
  if (site == GS_XD) return which ? 2 : 0;    // A = X: its rows; B = D
  if (site == GS_PXT) return which ? 0 : -1;  // B = X^T: columns of X^T are rows of X
  return -1;
}
// xdst >= 0: the image goes to X's cached image xdst instead of img (which 0) / img2 (which 1)
__global__ void __launch_bounds__(256) kb_pexp_site(const MolPtrs* __restrict__ mp,
                                                    const int* __restrict__ list, int site,
                                                    int which, int xdst) {
  const MolPtrs& q = mp[list[blockIdx.z]];
  if (*q.flag < 0) return;
  const SiteLines L = site_lines(site_of(q, site), which);
  const int lp = lines_padded(L.lines);
  int* e = xdst >= 0 ? q.xexp[xdst] : which ? q.iexp2 : q.iexp;
  if (!L.kcontig) {
    if ((int)blockIdx.x * 32 >= lp) return;
    pexp_rows_dev<32, 256>(L.M, L.ld, L.lines, L.K, lp, e, blockIdx.x);
    return;
  }
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= lp) return;
  unsigned long long mx = 0ull;
  if (i < L.lines)
    for (int k = lane; k < L.K; k += 32) mx = max(mx, abs_bits(L.M[k + (size_t)i * L.ld]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) e[i] = exp_of_max(mx);
}
__global__ void __launch_bounds__(256) kb_psplit_site(const MolPtrs* __restrict__ mp,
                                                      const int* __restrict__ list, int site,
                                                      int which, int xdst) {
  const MolPtrs& q = mp[list[blockIdx.z]];
  if (*q.flag < 0) return;
  const SiteLines L = site_lines(site_of(q, site), which);
  const int lp = lines_padded(L.lines), nkc = (L.K + PP_KC - 1) / PP_KC;
  if ((int)blockIdx.x >= lp / 64 || (int)blockIdx.y >= nkc) return;
  const int* e = xdst >= 0 ? q.xexp[xdst] : which ? q.iexp2 : q.iexp;
  psplit_dev<Balanced>(L.M, L.ld, L.kcontig, L.lines, L.K, lp / 64,
                       e[blockIdx.x * 64 + (threadIdx.x & 63)],
                       xdst >= 0 ? q.ximg[xdst] : which ? q.img2 : q.img, blockIdx.x, blockIdx.y);
}
__global__ void __launch_bounds__(PP_THREADS, 1) kb_opipe_site(const MolPtrs* __restrict__ mp,
                                                              const int* __restrict__ list,
                                                              int site) {
  const MolPtrs& q = mp[list[blockIdx.y]];
  if (*q.flag < 0) return;
  const Site s = site_of(q, site);
  const int tiles = ((s.M + PP_M - 1) / PP_M) * ((s.N + PP_N - 1) / PP_N);
  if ((int)blockIdx.x >= tiles) return;
  PipeArgs a{};
  const int xa = site_ximage(site, 0), xb = site_ximage(site, 1);
  a.A = xa >= 0 ? q.ximg[xa] : q.img;  // (xa is never 2)
  a.B = xb == 2 ? sp2_image(q, q.sp2i[1]) : xb >= 0 ? q.ximg[xb] : q.img2;
  a.eA = xa >= 0 ? q.xexp[xa] : q.iexp;
  a.eB = xb == 2 ? q.iexp : xb >= 0 ? q.xexp[xb] : q.iexp2;
  a.eshiftA = s.alpha == 2.0 ? 1 : s.alpha == 0.5 ? -1 : 0;
  a.nlbA = lines_padded(s.M) / 64;
  a.nlbB = lines_padded(s.N) / 64;
  a.M = s.M;
  a.N = s.N;
  a.nkc = (s.K + PP_KC - 1) / PP_KC;
  a.C = s.C;
  a.ldc = s.ld;
  a.sym = s.sym ? 1 : 0;
  a.status = q.sp2i + 3;
  if (threadIdx.x == 0) {
    const int mt = (s.M + PP_M - 1) / PP_M, nt = (s.N + PP_N - 1) / PP_N;
    const int b = blockIdx.x, gid = b / (PP_GROUP * nt), first = gid * PP_GROUP;
    const int gsize = min(mt - first, PP_GROUP), inner = b - gid * PP_GROUP * nt;
    const int i0 = (first + inner % gsize) * PP_M, j0 = (inner / gsize) * PP_N;
    if (!(s.sym && i0 + PP_M - 1 < j0))
      atomicAdd(&g_pipe_batch_flops, 2ull * (unsigned long long)min(PP_M, s.M - i0) *
                                         (unsigned long long)min(PP_N, s.N - j0) * (unsigned)s.K);
  }
  opipe_tile<Balanced>(a, blockIdx.x);
}

}  // namespace

void pipe_site_b(const BatchLaunch& b, int site) {
  if (!b.count) return;
  static bool attr = false;
  if (!attr) {
    ck(cudaFuncSetAttribute(kb_opipe_site, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            PP_SMEM<Balanced>),
       "smem attr batched pipelined split gemm");
    attr = true;
  }
  const int n = b.nao_max;
  const int lp = pimage_lines(n), nkc = (n + PP_KC - 1) / PP_KC;
  const int tiles = ((n + PP_M - 1) / PP_M) * ((n + PP_N - 1) / PP_N);
  int tk = prof_kbegin(b.s);
  for (int which = 0; which < 2; ++which) {
    if (site_ximage(site, which) >= 0) continue;  // already split (X's images, the iterate)
    g_kernel_launches += 2;
    kb_pexp_site<<<dim3(lp / 8, 1, b.count), 256, 0, b.s>>>(b.mp, b.list, site, which, -1);
    kb_psplit_site<<<dim3(lp / 64, nkc, b.count), 256, 0, b.s>>>(b.mp, b.list, site, which,
                                                                   -1);
  }
  prof_kend(KS_PIPE_PREP, tk, b.s);
  ++g_kernel_launches;
  tk = prof_kbegin(b.s);
  kb_opipe_site<<<dim3(tiles, b.count), PP_THREADS, PP_SMEM<Balanced>, b.s>>>(b.mp, b.list, site);
  prof_kend(KS_PIPE, tk, b.s);
}

void pipe_x_images_b(const BatchLaunch& b) {
  if (!b.count) return;
  const int n = b.nao_max;
  const int lp = pimage_lines(n), nkc = (n + 31) / 32;  // split blocks of 32 k
  const int tk = prof_kbegin(b.s);
  // rows of X as op(A) of X D, columns of X as op(B) of F X
  const int src[2][2] = {{GS_XD, 0}, {GS_FX, 1}};
  for (int x = 0; x < 2; ++x) {
    g_kernel_launches += 2;
    kb_pexp_site<<<dim3(lp / 8, 1, b.count), 256, 0, b.s>>>(b.mp, b.list, src[x][0], src[x][1], x);
    kb_psplit_site<<<dim3(lp / 64, nkc, b.count), 256, 0, b.s>>>(b.mp, b.list, src[x][0],
                                                                   src[x][1], x);
  }
  prof_kend(KS_PIPE_PREP, tk, b.s);
}

// the first iterate D0 (from A and the Gershgorin bounds), its slice image and the first decision
void sp2_init_b(const BatchLaunch& b) {
  if (!b.count) return;
  const int lp = pimage_lines(b.nao_max);
  const int tk = prof_kbegin(b.s);
  ++g_kernel_launches;
  kb_sp2_init<<<dim3(lp / 8, 1, b.count), 256, 0, b.s>>>(b.mp, b.list);
  prof_kend(KS_PIPE_PREP, tk, b.s);
}

// the projection iterate back to FP64 for every listed molecule (after the last step)
void sp2_unfix_b(const BatchLaunch& b) {
  if (!b.count) return;
  const int nt = (b.nao_max + 31) / 32, blocks = nt * (nt + 1) / 2;
  ++g_kernel_launches;
  kb_sp2_unfix<<<dim3(blocks, 1, b.count), 256, 0, b.s>>>(b.mp, b.list);
}

// a projection step for every listed molecule still iterating: D^2 on the tensor cores from the
// iterate's slice image, the next iterate (D^2 or 2D - D^2 as decided) over D in Y, its slice
// image and the next decision
void sp2_square_b(const BatchLaunch& b) {
  if (!b.count) return;
  static bool attr = false;
  if (!attr) {
    ck(cudaFuncSetAttribute(kb_opipe_sq, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            PP_SMEM<Balanced>),
       "smem attr batched pipelined split gemm");
    attr = true;
  }
  const int n = b.nao_max;
  const int tiles = ((n + PP_M - 1) / PP_M) * ((n + PP_N - 1) / PP_N);
  const int tk = prof_kbegin(b.s);
  ++g_kernel_launches;
  kb_opipe_sq<<<dim3(tiles, b.count), PP_THREADS, PP_SMEM<Balanced>, b.s>>>(b.mp, b.list);
  prof_kend(KS_PIPE, tk, b.s);
}

size_t pimage_bytes(int lines, int K, bool balanced) {
  const size_t lp = (size_t)((lines + PP_M - 1) / PP_M) * PP_M;
  const size_t kp = (size_t)((K + PP_KC - 1) / PP_KC) * PP_KC;
  return lp * kp * (balanced ? Balanced::SLICES : Magnitude::SLICES) * sizeof(uint16_t);
}
int pimage_lines(int lines) { return ((lines + PP_M - 1) / PP_M) * PP_M; }
int sp2_slot_count(int n) { return sp2_slots(n); }

// slice image of a matrix: line i, position k is M[i + k ld] (kcontig = 0: the rows of M) or
// M[k + i ld] (kcontig = 1: the columns of M); img holds pimage_bytes(lines, K) bytes and e
// pimage_lines(lines) ints
void psplit(const double* M, int ld, int kcontig, int lines, int K, PImage& img, cudaStream_t s) {
  img.lines = lines;
  img.K = K;
  const int lp = pimage_lines(lines);
  const int nkc = (K + PP_KC - 1) / PP_KC;
  g_kernel_launches += 2;
  if (kcontig) k_pexp_cols<<<(lp * 32 + 255) / 256, 256, 0, s>>>(M, ld, lines, K, lp, img.e);
  else k_pexp_rows<<<lp / 16, 1024, 0, s>>>(M, ld, lines, K, lp, img.e);
  if (img.balanced)
    k_psplit<Balanced><<<dim3(lp / 64, nkc), 256, 0, s>>>(M, ld, kcontig, lines, K, lp / 64, img.e,
                                                          img.data);
  else
    k_psplit<Magnitude><<<dim3(lp / 64, nkc), 256, 0, s>>>(M, ld, kcontig, lines, K, lp / 64,
                                                           img.e, img.data);
}

// ---- both operands of one small product in one launch: block (line block, k chunk, operand).  A
// block finds the exponents of its 64 lines over all of k for itself (a few reads more per chunk
// instead of a launch in between), the first chunk's block writes them, and each splits its chunk.
struct SmallOperand {
  const double* M;
  int ld, kcontig, lines;
  int* e;
  uint16_t* img;
};
__global__ void __launch_bounds__(256) k_psplit_pair(SmallOperand oa, SmallOperand ob, int K) {
  const SmallOperand o = blockIdx.z ? ob : oa;
  const int lp = lines_padded(o.lines), lb = blockIdx.x, kc = blockIdx.y;
  if (lb >= lp / 64) return;
  __shared__ unsigned long long top[4][64];
  __shared__ int se[64];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (o.kcontig) {
    for (int li = wid; li < 64; li += 8) {
      const int i = lb * 64 + li;
      unsigned long long mx = 0ull;
      if (i < o.lines) {
#pragma unroll 4
        for (int k = lane; k < K; k += 32) mx = max(mx, abs_bits(o.M[k + (size_t)i * o.ld]));
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, d));
      if (lane == 0) se[li] = exp_of_max(mx);
    }
  } else {
    const int li = tid & 63, g = tid >> 6, i = lb * 64 + li;
    unsigned long long mx = 0ull;
    if (i < o.lines) {
#pragma unroll 8
      for (int k = g; k < K; k += 4) mx = max(mx, abs_bits(o.M[i + (size_t)k * o.ld]));
    }
    top[g][li] = mx;
    __syncthreads();
    if (g == 0) se[li] = exp_of_max(max(max(top[0][li], top[1][li]), max(top[2][li], top[3][li])));
  }
  __syncthreads();
  if (kc == 0 && tid < 64) o.e[lb * 64 + tid] = se[tid];
  psplit_dev<Balanced>(o.M, o.ld, o.kcontig, o.lines, K, lp / 64, se[tid & 63], o.img, lb, kc);
}

// work of pgemm_pair for orders up to n
static size_t pair_image(int n) { return (pimage_bytes(n, n, true) + 255) & ~(size_t)255; }
size_t pair_work_bytes(int n) { return 2 * (pair_image(n) + sizeof(int) * pimage_lines(n)); }

// C = op(A) op(B), column-major, all dimensions at most n: split and product in two launches
void pgemm_pair(int n, bool ta, bool tb, int M, int N, int K, const double* A, int lda,
                const double* B, int ldb, double* C, int ldc, bool sym, void* work, int* status,
                cudaStream_t s) {
  unsigned char* p = static_cast<unsigned char*>(work);
  PImage ia, ib;
  ia.balanced = ib.balanced = true;
  ia.lines = M;
  ib.lines = N;
  ia.K = ib.K = K;
  ia.data = reinterpret_cast<uint16_t*>(p);
  ib.data = reinterpret_cast<uint16_t*>(p + pair_image(n));
  ia.e = reinterpret_cast<int*>(p + 2 * pair_image(n));
  ib.e = ia.e + pimage_lines(n);
  const int lb = std::max(pimage_lines(M), pimage_lines(N)) / 64;
  ++g_kernel_launches;
  k_psplit_pair<<<dim3(lb, (K + PP_KC - 1) / PP_KC, 2), 256, 0, s>>>(
      {A, lda, ta ? 1 : 0, M, ia.e, ia.data}, {B, ldb, tb ? 0 : 1, N, ib.e, ib.data}, K);
  pgemm(ia, ib, C, ldc, sym, status, s, 0);
}

// C = 2^eshiftA op(A) op(B) from two slice images (A.K == B.K); sym: the product is symmetric
void pgemm(const PImage& A, const PImage& B, double* C, int ldc, bool sym, int* status,
           cudaStream_t s, int eshiftA) {
  if (A.lines <= 0 || B.lines <= 0) return;
  if (A.K != B.K) throw std::runtime_error("split GEMM: inner dimensions differ");
  if (A.K > PP_KMAX) throw std::runtime_error("split GEMM: inner dimension above 12288");
  if (A.balanced != B.balanced) throw std::runtime_error("split GEMM: operands split differently");
  static bool attr = false;
  if (!attr) {
    ck(cudaFuncSetAttribute(k_opipe<Balanced>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            PP_SMEM<Balanced>),
       "smem attr pipelined split gemm");
    ck(cudaFuncSetAttribute(k_opipe<Magnitude>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            PP_SMEM<Magnitude>),
       "smem attr pipelined split gemm");
    attr = true;
  }
  PipeArgs a{};
  a.A = A.data;
  a.B = B.data;
  a.eA = A.e;
  a.eB = B.e;
  a.eshiftA = eshiftA;
  a.nlbA = pimage_lines(A.lines) / 64;
  a.nlbB = pimage_lines(B.lines) / 64;
  a.M = A.lines;
  a.N = B.lines;
  a.nkc = (A.K + PP_KC - 1) / PP_KC;
  a.C = C;
  a.ldc = ldc;
  a.sym = sym ? 1 : 0;
  a.status = status;
  const int mt = (a.M + PP_M - 1) / PP_M, nt = (a.N + PP_N - 1) / PP_N;
  g_split_flops += sym ? (unsigned long long)a.N * (a.N + 1) * A.K
                       : 2ull * a.M * a.N * A.K;
  const int tk = prof_kbegin(s);
  ++g_kernel_launches;
  if (A.balanced) k_opipe<Balanced><<<mt * nt, PP_THREADS, PP_SMEM<Balanced>, s>>>(a);
  else k_opipe<Magnitude><<<mt * nt, PP_THREADS, PP_SMEM<Magnitude>, s>>>(a);
  prof_kend(KS_GEMM, tk, s);
}

}  // namespace tb

namespace tb {
extern bool g_pipe_gemm;

namespace {

// Workspace of tblite_gb300_split_gemm: a stream-ordered pool of this library's own per device, so
// that calls of any thread on any stream take and return memory in stream order (five cudaMalloc /
// cudaFree pairs and a pageable copy were 380 of the 468 us of a 1202 x 601 x 777 product).  At
// most GEMM_POOL_KEEP bytes stay with the pool between calls; what a larger product takes beyond
// that goes back to the device when its call has synchronised, and
// tblite_gb300_split_gemm_release gives back the rest.
constexpr uint64_t GEMM_POOL_KEEP = 512ull << 20;
constexpr int GEMM_MAX_DEVICES = 64;
// the current device's pool; null: it could not be made, or (make == false) no call has made it yet
cudaMemPool_t gemm_pool(bool make = true) {
  static std::mutex mutex;
  static cudaMemPool_t pools[GEMM_MAX_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= GEMM_MAX_DEVICES) return nullptr;
  std::lock_guard<std::mutex> lock(mutex);
  if (!pools[dev] && make) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
    uint64_t keep = GEMM_POOL_KEEP;
    if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return nullptr;
    }
    pools[dev] = pool;
  }
  return pools[dev];
}

// the status word of a thread's call (calls synchronise their stream, so one is enough): mapped
// host memory, written by the kernel only when a wait ran out
struct StatusWord {
  int* p = nullptr;
  ~StatusWord() {
    if (p) cudaFreeHost(p);
  }
  int* get() {
    if (!p && cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) !=
                  cudaSuccess)
      p = nullptr;
    return p;
  }
};

}  // namespace
}  // namespace tb

// C = A B on the pipelined split GEMM from device pointers (column-major: A m x k with leading
// dimension m, B k x n with leading dimension k, C m x n with leading dimension m; sym: C is
// symmetric, m == n).  The two slice images live in the library's pool for the call, which
// synchronises the stream.  0 on success, 1 if a wait of the tensor-core pipeline ran out, -1 on
// bad arguments, -2 on a CUDA error.
extern "C" int tblite_gb300_split_gemm(int m, int n, int k, const double* a, const double* b,
                                       double* c, int sym, void* stream) {
  using namespace tb;
  if (m <= 0 || n <= 0 || k <= 0 || !a || !b || !c || (sym && m != n)) return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  thread_local StatusWord word;
  int* st = word.get();
  const cudaMemPool_t pool = gemm_pool();
  if (!st || !pool) {
    cudaGetLastError();
    return -2;
  }
  *(volatile int*)st = 0;
  auto aligned = [](size_t x) { return (x + 1023) & ~(size_t)1023; };
  const size_t da = aligned(pimage_bytes(m, k, true)), db = aligned(pimage_bytes(n, k, true));
  const size_t ea = aligned(sizeof(int) * pimage_lines(m));
  char* w = nullptr;
  if (cudaMallocFromPoolAsync((void**)&w, da + db + ea + sizeof(int) * pimage_lines(n), pool, s) !=
      cudaSuccess) {
    cudaGetLastError();
    return -2;
  }
  PImage ia, ib;
  ia.balanced = ib.balanced = true;
  ia.data = reinterpret_cast<uint16_t*>(w);
  ib.data = reinterpret_cast<uint16_t*>(w + da);
  ia.e = reinterpret_cast<int*>(w + da + db);
  ib.e = reinterpret_cast<int*>(w + da + db + ea);
  int rc = 0;
  try {
    psplit(a, m, 0, m, k, ia, s);
    psplit(b, k, 1, n, k, ib, s);
    pgemm(ia, ib, c, m, sym != 0, st, s);
  } catch (...) {
    rc = -2;
  }
  if (cudaFreeAsync(w, s) != cudaSuccess) rc = -2;
  if (cudaStreamSynchronize(s) != cudaSuccess) rc = -2;
  return rc != 0 ? rc : *(volatile int*)st != 0 ? 1 : 0;
}

extern "C" int tblite_gb300_split_gemm_release(void) {
  const cudaMemPool_t pool = tb::gemm_pool(false);
  return !pool || cudaMemPoolTrimTo(pool, 0) == cudaSuccess ? 0 : -2;
}

extern "C" void tblite_gb300_set_pipelined_gemm(int enable) { tb::g_pipe_gemm = enable != 0; }

// test setting: polls of the pipelined split GEMM's pipeline waits on the current device (0:
// the default 2^22).  0 on success, -1 on a CUDA error.
extern "C" unsigned long long tblite_gb300_get_pipe_batch_flops(void) {
  unsigned long long v = 0;
  if (cudaMemcpyFromSymbol(&v, tb::g_pipe_batch_flops, sizeof(v)) != cudaSuccess) return 0;
  return v;
}

extern "C" int tblite_gb300_set_pipeline_wait_limit(int polls) {
  const int v = polls > 0 ? polls : tb::PP_WAIT;
  return cudaMemcpyToSymbol(tb::g_pipe_wait_limit, &v, sizeof(int)) == cudaSuccess ? 0 : -1;
}
