// FP64 pieces shared by the assembly kernels: the points of one panel spread
// over the lanes of a warp, and the reduction of the eight sums (four
// shape-function entries each of N and D) that such a panel yields.
#pragma once
#include <cuda_runtime.h>
#include "kernels.h"

namespace wbem {

constexpr double kInv4PiPanel = 0.07957747154594766788;  // 1 / (4 pi)

// Sums v[0..7] over the 16 lanes of a half warp (FULL: over the whole warp)
// and returns to lane l the total of v[(l >> 1) & 7]. A reduce-scatter: three
// halving exchanges (4 + 2 + 1 additions) and one plain exchange, 8 additions
// per lane (FULL: 9) against 32 (40) for eight butterflies. FP64 additions
// issue at 1/64 of the FP32 rate on this GPU, so they are what the reduction
// costs.
template <bool FULL>
__device__ __forceinline__ double panel_reduce8(double v[8], int lane) {
#pragma unroll
  for (int o = 8, n = 4; o >= 2; o >>= 1, n >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i < n) {
        const double keep = up ? v[i + n] : v[i], send = up ? v[i] : v[i + n];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
  }
  double s = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
  if (FULL) s += __shfl_xor_sync(0xffffffffu, s, 16);
  return s;
}

// One vertex-singular panel of the collocation point x (source/
// bem_problem.cc:478-522), the rule's points over the lanes of a warp: every
// lane returns the sum of component (lane >> 1) & 7 (N entries 0..3, D
// entries 0..3). P: panel vertices, sp: the rule of the singular vertex.
// With the edges F0 = P1 - P0, E0 = P2 - P0 and W = P3 - P2 - F0:
//   x_q - x = (P0 - x) + s F0 + t (E0 + s W),  je = E0 + s W,  jx = F0 + t W.
__device__ __forceinline__ double singular_panel(const double P[4][3], const double x[3],
                                                 const double (*sp)[3], int nsp, int lane) {
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  double O[3], F[3], E[3], W[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    O[d] = P[0][d] - x[d];
    F[d] = P[1][d] - P[0][d];
    E[d] = P[2][d] - P[0][d];
    W[d] = (P[3][d] - P[2][d]) - F[d];
  }
  for (int q = lane; q < nsp; q += 32) {
    const double s = sp[q][0], t = sp[q][1], w = sp[q][2] * kInv4PiPanel;
    double R[3], jx[3], je[3], c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      je[d] = fma(s, W[d], E[d]);
      jx[d] = fma(t, W[d], F[d]);
      R[d] = fma(t, je[d], fma(s, F[d], O[d]));
    }
    c[0] = jx[1] * je[2] - jx[2] * je[1];
    c[1] = jx[2] * je[0] - jx[0] * je[2];
    c[2] = jx[0] * je[1] - jx[1] * je[0];
    const double det = sqrt(fma(c[0], c[0], fma(c[1], c[1], c[2] * c[2])));
    const double ri = rsqrt(fma(R[0], R[0], fma(R[1], R[1], R[2] * R[2])));
    const double u = ri * w;
    const double sq = u * det;
    const double dq = -fma(R[0], c[0], fma(R[1], c[1], R[2] * c[2])) * (u * (ri * ri));
    const double s1 = 1 - s, t1 = 1 - t;
    const double ph[4] = {s1 * t1, s * t1, s1 * t, s * t};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[j] = fma(dq, ph[j], v[j]);
      v[4 + j] = fma(sq, ph[j], v[4 + j]);
    }
  }
  return panel_reduce8<true>(v, lane);
}

}  // namespace wbem
