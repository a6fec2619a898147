// Sums of several FP64 numbers over a warp.
//
// What bounds them: an FP64 addition costs a warp 64 to 76 cycles, a shuffle two issue slots, and the
// butterfly of one number is five additions (580 cycles measured).  N numbers together need N - 1
// or a few more additions instead of 5 N: in the first step the lower half-warp goes on with the
// first half of the numbers and the upper half-warp with the second half, and so on.  Every number
// is summed in the same tree as by warp_sum (lane ^ 16, 8, 4, 2, 1), so the result has the same bits.
#pragma once
#include <cuda_runtime.h>

namespace tb {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

namespace wsums {
template <int N, int O>
__device__ __forceinline__ void fold(double* v, unsigned mask) {
  if constexpr (O > 0) {
    constexpr int M = (N + 1) / 2;
    const bool upper = threadIdx.x & O;
#pragma unroll
    for (int k = 0; k < M; ++k) {
      if (k + M < N) {
        const double keep = upper ? v[k + M] : v[k], send = upper ? v[k] : v[k + M];
        v[k] = keep + __shfl_xor_sync(mask, send, O);
      } else {
        v[k] += __shfl_xor_sync(mask, v[k], O);
      }
    }
    fold<M, O / 2>(v, mask);
  }
}
// where the sum of number j of n stands after the steps of a group of g lanes: lane, and place there
__host__ __device__ constexpr int place(int n, int j, int g, bool lane) {
  int l = 0;
  for (int o = g / 2; o > 0; o /= 2) {
    const int m = (n + 1) / 2;
    if (j >= m) {
      l |= o;
      j -= m;
    }
    n = m;
  }
  return lane ? l : j;
}
template <int N, int G, int J = 0>
__device__ __forceinline__ void spread(const double* t, double* v, unsigned mask) {
  if constexpr (J < N) {
    constexpr int from = place(N, J, G, true), at = place(N, J, G, false);
    v[J] = __shfl_sync(mask, t[at], from, G);
    spread<N, G, J + 1>(t, v, mask);
  }
}
}  // namespace wsums

// v[j] of every lane becomes the sum of v[j] over its group of G lanes (a power of two; mask: the
// lanes of the groups that come here)
template <int G, int N>
__device__ __forceinline__ void group_sums(double (&v)[N], unsigned mask) {
  double t[N];
#pragma unroll
  for (int j = 0; j < N; ++j) t[j] = v[j];
  wsums::fold<N, G / 2>(t, mask);
  wsums::spread<N, G>(t, v, mask);
}
// over the warp
template <int N>
__device__ __forceinline__ void warp_sums(double (&v)[N]) {
  group_sums<32>(v, 0xffffffffu);
}
// four sums, left where they arise; warp_sum4_of gives a lane the sum of number j & 3
__device__ __forceinline__ double warp_sums4(double (&v)[4]) {
  wsums::fold<4, 16>(v, 0xffffffffu);
  return v[0];
}
__device__ __forceinline__ double warp_sum4_of(double s, int j) {
  return __shfl_sync(0xffffffffu, s, (j & 2) << 3 | (j & 1) << 3);
}
// the same for a gradient, a virial and further numbers
template <class... T>
__device__ __forceinline__ void warp_sums_grad(double (&g)[3], double (&sg)[9], T&... rest) {
  double t[12 + sizeof...(T)] = {g[0],  g[1],  g[2],  sg[0], sg[1], sg[2], sg[3],
                                 sg[4], sg[5], sg[6], sg[7], sg[8], rest...};
  warp_sums(t);
#pragma unroll
  for (int k = 0; k < 3; ++k) g[k] = t[k];
#pragma unroll
  for (int k = 0; k < 9; ++k) sg[k] = t[3 + k];
  int k = 12;
  ((rest = t[k++]), ...);
}

}  // namespace tb
