// Operators of the mixed Dirichlet/Neumann system and the pieces of the
// Krylov solvers.
//
// The system is never formed in full: the GMRES mat-vec streams N and D once
// and picks, per column, the block that the column's boundary condition needs
// (BEMProblem<3>::vmult, source/bem_problem.cc:620-670: A x = -D (x s) + N (x o)
// + alpha (x o)); the right-hand side uses the complementary blocks
// (compute_rhs, :673-706). Constrained rows are replaced afterwards
// (ConstrainedOperator::vmult / distribute_rhs, include/constrained_matrix.h:72-94).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <atomic>
#include "dfloat.cuh"
#include "kernels.h"
#include "../../include/wbem.h"

namespace wbem {

constexpr int kMvThreads = 256;
constexpr int kMvWarps = kMvThreads / 32;

// Sums v[0..R) over the threads of the CTA; thread r < R returns row r's
// total. Reduce-scatter inside the warps (FP64 additions issue at 1/64 of the
// FP32 rate), then the warps' sums in order.
template <int R>
__device__ __forceinline__ double cta_rows_sum(double v[R]) {
  static_assert(R == 4 || R == 8, "rows per CTA");
  __shared__ double red[kMvWarps][R];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int o = 16, n = R / 2; n > 0; o >>= 1, n >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < R / 2; ++i)
      if (i < n) {
        const double keep = up ? v[i + n] : v[i], send = up ? v[i] : v[i + n];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
  }
  constexpr int G = 32 / R;  // lanes that hold the same row now
  double s = v[0];
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane % G == 0) red[warp][lane / G] = s;
  __syncthreads();
  s = 0.0;
  if (tid < R)
    for (int w = 0; w < kMvWarps; ++w) s += red[w][tid];
  return s;
}

// y_i = sum_j sel(i,j) x_j + diag. FP64 matrices. A CTA takes 4 rows, its
// threads the columns: x_j and the column's matrix are read once for the 4
// rows, whose loads are independent. Bound by the FP64 pipe (one DFMA per 8
// bytes: 4.6 TB/s at most). With a warp per row and x staged in shared memory
// it took 46 us at N = 2,000 and 1.10 ms at N = 16,226, now 16 us and
// 0.47 ms (4.5 TB/s; 0.61 ms with the sign of x taken by an FP64 instruction).
constexpr int kMvRows64 = 4;

__global__ void __launch_bounds__(kMvThreads)
    k_matvec_fp64(int N, int mode, const double* __restrict__ Nm, const double* __restrict__ Dm,
                  const uint8_t* __restrict__ mask, const double* __restrict__ alpha,
                  const double* __restrict__ x, double* __restrict__ y) {
  constexpr int R = kMvRows64;
  const int row0 = blockIdx.x * R, tid = threadIdx.x;
  // mode 0: mask ? -D : N ; mode 1: mask ? -N : D
  const double* A0 = (mode == 0) ? Nm : Dm;  // used where mask == 0
  const double* A1 = (mode == 0) ? Dm : Nm;  // used (negated) where mask == 1
  size_t off[R];
#pragma unroll
  for (int r = 0; r < R; ++r) off[r] = (size_t)min(row0 + r, N - 1) * N;
  double acc[R] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (int j = tid; j < N; j += kMvThreads) {
    const bool m = mask[j] != 0;
    const double* A = (m ? A1 : A0) + j;
    const double xv = x[j];  // the sign by its bit: the FP64 pipe is the bound
    const double xj = __hiloint2double(__double2hiint(xv) ^ (m ? 0x80000000 : 0), __double2loint(xv));
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = fma(__ldcs(A + off[r]), xj, acc[r]);
  }
  double s = cta_rows_sum<R>(acc);
  const int row = row0 + tid;
  if (tid < R && row < N) {
    const double xi = x[row];
    if (mode == 0) {
      if (!mask[row]) s = fma(alpha[row], xi, s);
    } else {
      if (mask[row]) s = fma(-alpha[row], xi, s);
    }
    y[row] = s;
  }
}

cudaError_t launch_matvec_fp64(int N, int mode, const double* Nm, const double* Dm,
                               const uint8_t* mask, const double* alpha, const double* x,
                               double* y, cudaStream_t s) {
  k_matvec_fp64<<<(N + kMvRows64 - 1) / kMvRows64, kMvThreads, 0, s>>>(N, mode, Nm, Dm, mask, alpha,
                                                                       x, y);
  return cudaGetLastError();
}

// Same operator with (hi, lo) float pairs whose boundary-condition selection
// was applied at assembly (P = A2 for mode 0, B2 for mode 1): one contiguous
// matrix per apply. entry = hi + lo; products and sums in double-float on
// FP32 units, x given in FP64 and split into float pairs (k_split_x) first: a
// split per CTA and column would cost three FP64-rate instructions for every
// 4 entries. A CTA takes 4 rows, a thread two columns (16 bytes of each row)
// per step where N is even. HBM-bound: 285 us (4.0 TB/s) at N = 12,000 with a
// warp per row, now 182 us (6.3 TB/s); 1.55 ms at N = 32,768, now 1.21 ms.
constexpr int kMvRowsM = 4;
// Up to this size every CTA splits x itself (SPLIT): its few columns cost less
// than the launch. A vmult and a compute_rhs on host arrays, us, this way / with
// k_split_x: 600 dofs 82.5 / 86, 1,500 86 / 89, 2,000 112 / 95.
constexpr int kMvSplitCols = 1500;

__global__ void k_split_x(int N, const double* __restrict__ x, float2* __restrict__ xs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const df v = df_from_double(x[i]);
  xs[i] = make_float2(v.hi, v.lo);
}

__device__ __forceinline__ void pair_fma(df& acc, float ah, float al, float xh, float xl) {
  df p = two_prod(ah, xh);
  p.lo = __fmaf_rn(ah, xl, __fmaf_rn(al, xh, p.lo));
  acc = df_add(acc, p);
}

template <bool EVEN, bool SPLIT>
__global__ void __launch_bounds__(kMvThreads)
    k_matvec_mixed(int N, int mode, const float2* __restrict__ P, const uint8_t* __restrict__ mask,
                   const double* __restrict__ alpha, const float2* __restrict__ xs,
                   const double* __restrict__ x, double* __restrict__ y) {
  constexpr int R = kMvRowsM;
  const int row0 = blockIdx.x * R, tid = threadIdx.x;
  const float2* row[R];
#pragma unroll
  for (int r = 0; r < R; ++r) row[r] = P + (size_t)min(row0 + r, N - 1) * N;
  df acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r] = {0.f, 0.f};
  auto x_pair = [&](int j) {
    if (!SPLIT) return xs[j];
    const df v = df_from_double(x[j]);
    return make_float2(v.hi, v.lo);
  };
  if (EVEN) {
#pragma unroll 2
    for (int j = 2 * tid; j < N; j += 2 * kMvThreads) {
      float4 a[R];
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = __ldcs(reinterpret_cast<const float4*>(row[r] + j));
      float4 xv;
      if (SPLIT) {
        const float2 u = x_pair(j), v = x_pair(j + 1);
        xv = make_float4(u.x, u.y, v.x, v.y);
      } else {
        xv = *reinterpret_cast<const float4*>(xs + j);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        pair_fma(acc[r], a[r].x, a[r].y, xv.x, xv.y);
        pair_fma(acc[r], a[r].z, a[r].w, xv.z, xv.w);
      }
    }
  } else {
#pragma unroll 4
    for (int j = tid; j < N; j += kMvThreads) {
      float2 a[R];
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = __ldcs(row[r] + j);
      const float2 xv = x_pair(j);
#pragma unroll
      for (int r = 0; r < R; ++r) pair_fma(acc[r], a[r].x, a[r].y, xv.x, xv.y);
    }
  }
  double v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = df_to_double(acc[r]);
  double s = cta_rows_sum<R>(v);
  const int i = row0 + tid;
  if (tid < R && i < N) {
    const double xi = x[i];
    if (mode == 0) {
      if (!mask[i]) s = fma(alpha[i], xi, s);
    } else {
      if (mask[i]) s = fma(-alpha[i], xi, s);
    }
    y[i] = s;
  }
}

cudaError_t launch_matvec_mixed(int N, int mode, const float2* P, const uint8_t* mask,
                                const double* alpha, const double* x, float2* xs, double* y,
                                cudaStream_t s) {
  const int g = (N + kMvRowsM - 1) / kMvRowsM;
  if (N <= kMvSplitCols) {
    if (N & 1)
      k_matvec_mixed<false, true><<<g, kMvThreads, 0, s>>>(N, mode, P, mask, alpha, nullptr, x, y);
    else
      k_matvec_mixed<true, true><<<g, kMvThreads, 0, s>>>(N, mode, P, mask, alpha, nullptr, x, y);
    return cudaGetLastError();
  }
  k_split_x<<<(N + 255) / 256, 256, 0, s>>>(N, x, xs);
  if (N & 1)
    k_matvec_mixed<false, false><<<g, kMvThreads, 0, s>>>(N, mode, P, mask, alpha, xs, x, y);
  else
    k_matvec_mixed<true, false><<<g, kMvThreads, 0, s>>>(N, mode, P, mask, alpha, xs, x, y);
  return cudaGetLastError();
}

// y = S x for the FP32 system matrix S (row-major, leading dimension ld, the
// constrained operator with alpha on its diagonal): the inner operator of the
// refinement solver. A CTA takes 8 rows, a thread four columns (16 bytes) of
// each per step; products and sums in FP32, kMvFlush terms per FP32 sum and
// FP64 beyond, so the operator is S to about 1e-6 relative, at 4 bytes of HBM
// traffic per entry. Four such sums are added without rounding error in FP32
// before they go to FP64, whose pipe would hold up the stream otherwise; for
// the same reason x is rounded to FP32 once, by k_round_x.
// HBM-bound: 317 us (5.1 TB/s) at N = 20,011 with a warp per row, now 255 us.
constexpr int kMvRows32 = 8;
constexpr int kMvFlush = 16;

__global__ void k_round_x(int N, const double* __restrict__ x, float* __restrict__ xf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) xf[i] = (float)x[i];
}

__global__ void __launch_bounds__(kMvThreads, 2)
    k_matvec_s32(int N, int ld, const float* __restrict__ S, const float* __restrict__ xf,
                 double* __restrict__ y) {
  constexpr int R = kMvRows32;
  const int row0 = blockIdx.x * R, tid = threadIdx.x;
  const float* row[R];
  double acc[R];
  float a[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    row[r] = S + (size_t)min(row0 + r, N - 1) * ld;
    acc[r] = 0.0;
    a[r][0] = a[r][1] = a[r][2] = a[r][3] = 0.f;
  }
  auto flush = [&]() {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const df u = two_sum(a[r][0], a[r][1]), w = two_sum(a[r][2], a[r][3]), t = two_sum(u.hi, w.hi);
      acc[r] += (double)t.hi;
      acc[r] += widen(t.lo + (u.lo + w.lo));
      a[r][0] = a[r][1] = a[r][2] = a[r][3] = 0.f;
    }
  };
  const int nq = N & ~3;  // whole quads (row starts are 16-byte aligned)
  int n = 0;
  for (int j = 4 * tid; j < nq; j += 4 * kMvThreads) {
    float4 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = __ldcs(reinterpret_cast<const float4*>(row[r] + j));
    const float4 f = *reinterpret_cast<const float4*>(xf + j);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      a[r][0] = __fmaf_rn(v[r].x, f.x, a[r][0]);
      a[r][1] = __fmaf_rn(v[r].y, f.y, a[r][1]);
      a[r][2] = __fmaf_rn(v[r].z, f.z, a[r][2]);
      a[r][3] = __fmaf_rn(v[r].w, f.w, a[r][3]);
    }
    if (++n == kMvFlush) {
      flush();
      n = 0;
    }
  }
  flush();
  if (nq + tid < N) {  // the last one to three columns
    const float f = xf[nq + tid];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] += (double)row[r][nq + tid] * (double)f;
  }
  const double s = cta_rows_sum<R>(acc);
  if (tid < R && row0 + tid < N) y[row0 + tid] = s;
}

cudaError_t launch_matvec_s32(int N, int ld, const float* S, const double* x, float* xf, double* y,
                              cudaStream_t s) {
  k_round_x<<<(N + 255) / 256, 256, 0, s>>>(N, x, xf);
  k_matvec_s32<<<(N + kMvRows32 - 1) / kMvRows32, kMvThreads, 0, s>>>(N, ld, S, xf, y);
  return cudaGetLastError();
}

// Transposed system operator y_j = sum_i sel(i,j) x_i + (1 - mask_j) alpha_j x_j.
// Blocks own column strips of 256 columns and a slice of rows; partial sums
// go to part[slice][N] and are added in a fixed order (deterministic).
constexpr int kMvtCols = 256;
constexpr int kMvtSlices = 32;

template <typename T>
__device__ __forceinline__ double load_entry(const T* p);
template <>
__device__ __forceinline__ double load_entry<double>(const double* p) {
  return __ldcs(p);
}

// sel: the column mask that picks N or -D (NULL: Nm already holds the
// selected operator)
template <typename T>
__global__ void k_matvec_t(int N, const T* __restrict__ Nm, const T* __restrict__ Dm,
                           const uint8_t* __restrict__ sel, const double* __restrict__ x,
                           double* __restrict__ part) {
  const int col = blockIdx.x * kMvtCols + threadIdx.x;
  const int slice = blockIdx.y;
  const int rows_per = (N + kMvtSlices - 1) / kMvtSlices;
  const int r0 = slice * rows_per, r1 = min(N, r0 + rows_per);
  if (col >= N) return;
  const bool m = sel != nullptr && sel[col] != 0;
  const T* A = m ? Dm : Nm;
  double acc = 0.0;
  for (int i = r0; i < r1; ++i) acc = fma(load_entry<T>(A + (size_t)i * N + col), x[i], acc);
  part[(size_t)slice * N + col] = m ? -acc : acc;
}

__global__ void k_matvec_t_finish(int N, const uint8_t* __restrict__ mask,
                                  const double* __restrict__ alpha, const double* __restrict__ x,
                                  const double* __restrict__ part, double* __restrict__ y) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  double s = 0;
  for (int k = 0; k < kMvtSlices; ++k) s += part[(size_t)k * N + j];
  if (alpha && !mask[j]) s = fma(alpha[j], x[j], s);
  y[j] = s;
}

cudaError_t launch_matvec_t_fp64(int N, const double* Nm, const double* Dm, const uint8_t* mask,
                                 const double* alpha, const double* x, double* y, double* part,
                                 cudaStream_t s) {
  dim3 g((N + kMvtCols - 1) / kMvtCols, kMvtSlices);
  k_matvec_t<double><<<g, kMvtCols, 0, s>>>(N, Nm, Dm, mask, x, part);
  k_matvec_t_finish<<<(N + 255) / 256, 256, 0, s>>>(N, mask, alpha, x, part, y);
  return cudaGetLastError();
}

// Transposed operator with (hi, lo) float pairs (P = A2 or B2, selection
// applied at assembly): threads own columns, blocks own a column strip and a
// slice of rows; the slice's x is split into float pairs in shared memory and
// products and sums run in double-float on FP32 units, as in k_matvec_mixed.
constexpr int kMvtChunk = 256;
__global__ void __launch_bounds__(kMvtCols)
    k_matvec_t_mixed(int N, const float2* __restrict__ P, const double* __restrict__ x,
                     double* __restrict__ part) {
  __shared__ float2 xs[kMvtChunk];
  const int col = blockIdx.x * kMvtCols + threadIdx.x;
  const int slice = blockIdx.y;
  const int rows_per = (N + kMvtSlices - 1) / kMvtSlices;
  const int r0 = slice * rows_per, r1 = min(N, r0 + rows_per);
  const bool active = col < N;
  df acc = {0.f, 0.f};
  for (int i0 = r0; i0 < r1; i0 += kMvtChunk) {
    const int n = min(kMvtChunk, r1 - i0);
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += kMvtCols) {
      const df v = df_from_double(x[i0 + k]);
      xs[k] = make_float2(v.hi, v.lo);
    }
    __syncthreads();
    if (active) {
      const float2* a_col = P + (size_t)i0 * N + col;
#pragma unroll 8
      for (int k = 0; k < n; ++k) {
        const float2 a = __ldcs(a_col + (size_t)k * N);
        const float2 xv = xs[k];
        df p = two_prod(a.x, xv.x);
        p.lo = __fmaf_rn(a.x, xv.y, __fmaf_rn(a.y, xv.x, p.lo));
        acc = df_add(acc, p);
      }
    }
  }
  if (active) part[(size_t)slice * N + col] = df_to_double(acc);
}

cudaError_t launch_matvec_t_mixed(int N, const float2* P, const uint8_t* mask, const double* alpha,
                                  const double* x, double* y, double* part, cudaStream_t s) {
  dim3 g((N + kMvtCols - 1) / kMvtCols, kMvtSlices);
  k_matvec_t_mixed<<<g, kMvtCols, 0, s>>>(N, P, x, part);
  k_matvec_t_finish<<<(N + 255) / 256, 256, 0, s>>>(N, mask, alpha, x, part, y);
  return cudaGetLastError();
}

// y = S^T x for the FP32 system matrix: threads own columns, blocks own a
// column strip and a slice of rows; FP32 partial sums over 64 rows at a time,
// moved into FP64, then the slices are added in a fixed order.
__global__ void k_matvec_s32_t(int N, int ld, const float* __restrict__ S,
                               const double* __restrict__ x, double* __restrict__ part) {
  const int col = blockIdx.x * kMvtCols + threadIdx.x;
  const int slice = blockIdx.y;
  const int rows_per = (N + kMvtSlices - 1) / kMvtSlices;
  const int r0 = slice * rows_per, r1 = min(N, r0 + rows_per);
  if (col >= N) return;
  double acc = 0.0;
  for (int i0 = r0; i0 < r1; i0 += 64) {
    const int i1 = min(r1, i0 + 64);
    float a = 0.f;
    for (int i = i0; i < i1; ++i) a = __fmaf_rn(__ldcs(S + (size_t)i * ld + col), (float)x[i], a);
    acc += (double)a;
  }
  part[(size_t)slice * N + col] = acc;
}

cudaError_t launch_matvec_s32_t(int N, int ld, const float* S, const double* x, double* y,
                                double* part, cudaStream_t s) {
  dim3 g((N + kMvtCols - 1) / kMvtCols, kMvtSlices);
  k_matvec_s32_t<<<g, kMvtCols, 0, s>>>(N, ld, S, x, part);
  k_matvec_t_finish<<<(N + 255) / 256, 256, 0, s>>>(N, nullptr, nullptr, x, part, y);
  return cudaGetLastError();
}

// Constrained rows: y_i = x_i - sum_j c_ij x_j.
__global__ void k_constraint_rows(int nrows, const int* __restrict__ crow,
                                  const int* __restrict__ cptr, const int* __restrict__ ccol,
                                  const double* __restrict__ cval, const double* __restrict__ x,
                                  double* __restrict__ y) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nrows) return;
  const int i = crow[k];
  double v = x[i];
  for (int e = cptr[k]; e < cptr[k + 1]; ++e) v -= cval[e] * x[ccol[e]];
  y[i] = v;
}

cudaError_t launch_constraint_rows(int nrows, const int* crow, const int* cptr, const int* ccol,
                                   const double* cval, const double* x, double* y,
                                   cudaStream_t s) {
  if (nrows == 0) return cudaSuccess;
  k_constraint_rows<<<(nrows + 127) / 128, 128, 0, s>>>(nrows, crow, cptr, ccol, cval, x, y);
  return cudaGetLastError();
}

// Transposed constrained operator. With C the set of constrained rows,
// (A_c^T y)_j = [j in C] y_j - sum_{i in C} c_ij y_i + [j not... ] the
// unconstrained part sum_{i not in C} A_ij y_i. The caller zeroes y_i for
// i in C before the transposed mat-vec; this kernel adds the constraint
// part: out_j += [j in C] y_j - sum_{i in C, (i,j) entry} c_ij y_i, using the
// column-major (transposed) entry lists tptr/tsrc/tval.
__global__ void k_constraint_rows_t(int N, const int* __restrict__ tptr,
                                    const int* __restrict__ tsrc, const double* __restrict__ tval,
                                    const uint8_t* __restrict__ cflag,
                                    const double* __restrict__ yin, double* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  double v = out[j];
  if (cflag[j]) v += yin[j];
  for (int e = tptr[j]; e < tptr[j + 1]; ++e) v -= tval[e] * yin[tsrc[e]];
  out[j] = v;
}

cudaError_t launch_constraint_rows_t(int N, int nrows, const int* crow, const int* cptr,
                                     const int* ccol, const double* cval, const int* tptr,
                                     const int* tsrc, const double* tval, const uint8_t* cflag,
                                     const double* x, double* y, cudaStream_t s) {
  (void)nrows; (void)crow; (void)cptr; (void)ccol; (void)cval;
  k_constraint_rows_t<<<(N + 255) / 256, 256, 0, s>>>(N, tptr, tsrc, tval, cflag, x, y);
  return cudaGetLastError();
}

__global__ void k_set_rows(int nrows, const int* __restrict__ crow, const double* __restrict__ val,
                           double* __restrict__ y) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nrows) return;
  y[crow[k]] = val[k];
}

cudaError_t launch_set_rows(int nrows, const int* crow, const double* val, double* y,
                            cudaStream_t s) {
  if (nrows == 0) return cudaSuccess;
  k_set_rows<<<(nrows + 127) / 128, 128, 0, s>>>(nrows, crow, val, y);
  return cudaGetLastError();
}

// ------------------------------------------------------------ block-Jacobi
// Diagonal blocks of the constrained system, inverted by Gauss-Jordan with
// partial pivoting. binv[b] holds the inverse transposed (column k of the
// inverse contiguous) for coalesced application.
// A cluster of kBJCtas CTAs per block, 16 rows each in registers: thread (row,
// g) holds columns g, g + 16, .... Rows are never moved: a row keeps the step
// at which it was the pivot, and pos, the place that row exchanges would have
// given it (equal pivots go to the place whose lowest differing bit is 0, as in
// a halving tree over the places). Per step each CTA sends its best candidate
// row, already scaled by its pivot, to every CTA of the cluster; one cluster
// barrier later all of them take the same winner and update their rows.
// 128^3 DFMA per block: 0.46 ms for 127 blocks on every SM's FP64 pipe at the
// least. One CTA per block, with a pivot tree and seven barriers per step, took
// 2.0 ms for up to 152 blocks and 4.0 ms for 157; now 0.32 ms for 16 blocks
// (N = 2,000), 1.13 ms for 127 (N = 16,226) and 1.39 ms for 157 (N = 20,011).
constexpr int kBJCtas = 8;
constexpr int kBJRows = kBJ / kBJCtas;       // rows per CTA
constexpr int kBJGroups = 16;                // threads per row
constexpr int kBJThreads = kBJRows * kBJGroups;
constexpr int kBJPer = kBJ / kBJGroups;      // columns per thread

struct BJCand {
  unsigned long long key;  // |pivot| as an integer (the order of positive doubles)
  int pos;                 // place of the row
  int row;                 // its index in the block
};

// The lanes of a warp with the largest key and, among them, the smallest rev
// (integer reductions: comparing doubles would take the FP64 pipe).
__device__ __forceinline__ unsigned bj_first(unsigned long long key, unsigned rev) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  const bool top = hi == mh && lo == ml;
  const unsigned mr = __reduce_min_sync(0xffffffffu, top ? rev : 0xffffffffu);
  return __ballot_sync(0xffffffffu, top && rev == mr);
}

__global__ void __cluster_dims__(kBJCtas, 1, 1) __launch_bounds__(kBJThreads, 4)
    k_bj_build(int N, const double* __restrict__ Nm, const double* __restrict__ Dm,
               const float2* __restrict__ A2, const double* __restrict__ blocks,
               const uint8_t* __restrict__ mask,
               const double* __restrict__ alpha,
               const uint8_t* __restrict__ cflag, const int* __restrict__ cptr,
               const int* __restrict__ ccol, const double* __restrict__ cval,
               double* __restrict__ binv, DevErr* err) {
  __shared__ __align__(16) double cand[2][kBJCtas][kBJ];  // scaled candidate rows of the CTAs
  __shared__ BJCand cinfo[2][kBJCtas];
  __shared__ __align__(16) double own[kBJ];               // this CTA's candidate row
  __shared__ double colv[kBJRows];
  __shared__ BJCand best;
  __shared__ double pinv;
  __shared__ int piv[kBJ];  // pivot row of each step
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int b = blockIdx.x / kBJCtas, rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, rl = tid / kBJGroups, g = tid % kBJGroups;
  const int r = rank * kBJRows + rl;  // row in the block
  const int i = b * kBJ + r, c0 = b * kBJ;
  double a[kBJPer];
#pragma unroll
  for (int m = 0; m < kBJPer; ++m) {
    const int c = g + kBJGroups * m, j = c0 + c;
    double v;
    if (i >= N || j >= N || cflag[i]) {
      v = (r == c) ? 1.0 : 0.0;
    } else if (blocks) {  // the system's diagonal block, free term included
      v = blocks[((size_t)b * kBJ + r) * kBJ + c];
    } else {
      const size_t o = (size_t)i * N + j;
      if (Nm) v = mask[j] ? -Dm[o] : Nm[o];
      else v = (double)A2[o].x + (double)A2[o].y;  // selected at assembly
      if (i == j && !mask[j]) v += alpha[i];
    }
    a[m] = v;
  }
  if (i < N && cflag[i]) {
    for (int e = cptr[i]; e < cptr[i + 1]; ++e) {
      const int j = ccol[e] - c0;
#pragma unroll
      for (int m = 0; m < kBJPer; ++m)
        if (j == g + kBJGroups * m) a[m] -= cval[e];
    }
  }
  // lanes 0..15 of warp 0 keep the places of the CTA's rows; -1 - step once used
  int pos = rank * kBJRows + (tid & (kBJRows - 1));
  bool used = false;
  int mystep = 0;  // step at which this thread's row was the pivot
  cl.sync();       // every CTA of the cluster runs: its shared memory may be written
#pragma unroll
  for (int mo = 0; mo < kBJPer; ++mo) {
#pragma unroll 1
    for (int ko = 0; ko < kBJGroups; ++ko) {
      const int k = kBJGroups * mo + ko, par = k & 1;
      if (g == ko) colv[rl] = a[mo];
      __syncthreads();
      if (tid < 32) {
        unsigned long long key = 0;
        unsigned rev = 0xffffffffu;
        if (lane < kBJRows && !used) {
          key = (unsigned long long)__double_as_longlong(fabs(colv[lane]));
          rev = __brev((unsigned)pos);
        }
        // one lane writes: once all rows of the CTA have been pivots every lane
        // is in the ballot, and the candidate is none (key 0, no row)
        const unsigned top = bj_first(key, rev);
        if (lane == __ffs(top) - 1) best = {key, pos, lane & (kBJRows - 1)};
      }
      __syncthreads();
      // the candidate row scaled by its pivot, 1 / pivot in the pivot's slot:
      // one warp per scheduler scales, 32 columns each
      const bool have = best.key != 0;  // the same in the whole CTA
      if (have && rl == best.row)
#pragma unroll
        for (int m = 0; m < kBJPer; ++m) own[g + kBJGroups * m] = a[m];
      if (have && tid == 0) pinv = 1.0 / colv[best.row];
      __syncthreads();
      if (have && tid < kBJ) own[tid] = tid == k ? pinv : own[tid] * pinv;
      __syncthreads();
      {
        const int dst = tid / 32;  // one warp per destination
        if (have) {
          double2* to = reinterpret_cast<double2*>(cl.map_shared_rank(&cand[par][rank][0], dst));
          const double2* from = reinterpret_cast<const double2*>(own);
          to[lane] = from[lane];
          to[lane + 32] = from[lane + 32];
        }
        if (lane == 0) {
          BJCand* ci = cl.map_shared_rank(&cinfo[par][rank], dst);
          *ci = {best.key, best.pos, rank * kBJRows + best.row};
        }
      }
      cl.sync();
      const BJCand mine = cinfo[par][lane & (kBJCtas - 1)];
      const int win = __ffs(bj_first(mine.key, __brev((unsigned)mine.pos))) - 1;
      const BJCand w = {__shfl_sync(0xffffffffu, mine.key, win), __shfl_sync(0xffffffffu, mine.pos, win),
                        __shfl_sync(0xffffffffu, mine.row, win)};
      // zero, or not a number: the same in every CTA of the cluster
      if (w.key == 0 || w.key > 0x7ff0000000000000ull) {
        if (rank == 0 && tid == 0) dev_fail(err, WBEM_ERR_SINGULAR, 31, b, k);
        return;
      }
      if (tid < kBJRows && !used) {
        if (rank * kBJRows + tid == w.row) used = true;
        else if (pos == k) pos = w.pos;
      }
      if (tid == 0) piv[k] = w.row;
      const double* pr = cand[par][win];
      if (r == w.row) {
        mystep = k;
#pragma unroll
        for (int m = 0; m < kBJPer; ++m) a[m] = pr[g + kBJGroups * m];
      } else {
        const double f = colv[rl];
        if (__double_as_longlong(f) << 1) {  // not zero, without the FP64 pipe
#pragma unroll
          for (int m = 0; m < kBJPer; ++m) {
            const double x = pr[g + kBJGroups * m];
            a[m] = (m == mo && g == ko) ? -f * x : fma(-f, x, a[m]);
          }
        }
      }
      __syncthreads();  // colv and own are read before the next step writes them
    }
  }
  // Row r of this CTA is row mystep of inv(P A), P the row exchanges, and
  // inv(A) = inv(P A) P: column c there is column piv[c] of inv(A). Stored
  // transposed: binv[column][row].
  __syncthreads();
  double* out = binv + (size_t)b * kBJ * kBJ;
#pragma unroll
  for (int m = 0; m < kBJPer; ++m) out[(size_t)piv[g + kBJGroups * m] * kBJ + mystep] = a[m];
  cl.sync();  // no CTA leaves while another may still write its shared memory
}

cudaError_t launch_bj_build(int N, const double* Nm, const double* Dm, const float2* A2,
                            const double* blocks, const uint8_t* mask, const double* alpha,
                            const uint8_t* cflag, const int* cptr_full, const int* ccol_full,
                            const double* cval_full, double* binv, DevErr* err, cudaStream_t s) {
  const int nb = (N + kBJ - 1) / kBJ;
  k_bj_build<<<nb * kBJCtas, kBJThreads, 0, s>>>(N, Nm, Dm, A2, blocks, mask, alpha, cflag, cptr_full,
                                                 ccol_full, cval_full, binv, err);
  return cudaGetLastError();
}

// z = inverse block * x. A CTA takes 32 rows of a block, its four warps a
// quarter of the columns each: a row's 128 FP64 multiply-adds in one chain (a
// CTA per block, a thread per row) take 8,192 cycles of each FP64 pipe, 14-15
// us with the launch at 2,000 to 16,000 dofs; here 2,048, and 5.8 us.
template <bool TRANS>
__global__ void __launch_bounds__(128)
    k_bj_apply(int N, const double* __restrict__ binv, const double* __restrict__ x,
               double* __restrict__ y) {
  __shared__ double part[4][32];
  const int b = blockIdx.x / 4, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int r = (blockIdx.x % 4) * 32 + lane, k0 = 32 * w, i0 = b * kBJ + k0;
  const double* B = binv + (size_t)b * kBJ * kBJ + (TRANS ? (size_t)r * kBJ + k0 : (size_t)k0 * kBJ + r);
  double v[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = B[TRANS ? k : (size_t)k * kBJ];
  const double xl = i0 + lane < N ? x[i0 + lane] : 0.0;
  double s0 = 0.0, s1 = 0.0;
#pragma unroll
  for (int k = 0; k < 32; k += 2) {
    s0 = fma(v[k], __shfl_sync(0xffffffffu, xl, k), s0);
    s1 = fma(v[k + 1], __shfl_sync(0xffffffffu, xl, k + 1), s1);
  }
  part[w][lane] = s0 + s1;
  __syncthreads();
  const int i = b * kBJ + r;
  if (w == 0 && i < N) y[i] = (part[0][lane] + part[1][lane]) + (part[2][lane] + part[3][lane]);
}

// A row's products in one chain: the order of sums that the FMA solve, which
// repeats to 1e-8 if a last bit changes, has always had.
__global__ void __launch_bounds__(kBJ)
    k_bj_apply_ordered(int N, const double* __restrict__ binv, const double* __restrict__ x,
               double* __restrict__ y) {
  __shared__ double xs[kBJ];
  const int b = blockIdx.x, r = threadIdx.x;
  const int i = b * kBJ + r;
  xs[r] = (i < N) ? x[i] : 0.0;
  __syncthreads();
  const double* B = binv + (size_t)b * kBJ * kBJ;
  double s = 0;
  // 32 loads in flight ahead of the chain of additions
#pragma unroll
  for (int k0 = 0; k0 < kBJ; k0 += 32) {
    double v[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = B[(size_t)(k0 + k) * kBJ + r];
#pragma unroll
    for (int k = 0; k < 32; ++k) s = fma(v[k], xs[k0 + k], s);
  }
  if (i < N) y[i] = s;
}

cudaError_t launch_bj_apply(int N, const double* binv, const double* x, double* y, int transpose,
                            bool ordered, cudaStream_t s) {
  const int nb = (N + kBJ - 1) / kBJ;
  if (transpose) k_bj_apply<true><<<4 * nb, 128, 0, s>>>(N, binv, x, y);
  else if (ordered) k_bj_apply_ordered<<<nb, kBJ, 0, s>>>(N, binv, x, y);
  else k_bj_apply<false><<<4 * nb, 128, 0, s>>>(N, binv, x, y);
  return cudaGetLastError();
}

// ------------------------------------------------------------ Krylov helpers
constexpr int kRedBlocks = 120;

// One Arnoldi step: classical Gram-Schmidt of w against the k basis vectors of
// V, once more, the norm, and the next basis vector v = w / |w|. out[0..k) =
// the summed coefficients, out[k] = the norm. A cooperative launch: CTA b owns
// the rows of chunk b (of w, V and v), the dot products and the norm meet in
// grid barriers (bounded waits on a counter), and every CTA adds the partial
// sums of all CTAs itself, in the same order.
// Bound by latency: the work is 4 k N FP64 operations on a basis that sits in
// L2. As nine launches (dots, a serial sum of the CTAs' parts, update, twice,
// then norm and scaling) a step took 110 us at N = 2,000 (mean over the 34
// steps of a solve), now 25 us.
// ORDERED: every sum in the order that those launches used (kRedBlocks chunks,
// trees of 256 threads, serial sums of the chunks and over the vectors). The
// FMA product is linear to FP32 round-off only, so that an FMA solve repeats
// to 1e-8 if any sum changes in its last bit; with these orders it repeats
// exactly: 94 us at N = 32,768 (mean over 55 steps), as launches 178 us.
constexpr int kOrthoThreads = 256;
constexpr int kOrthoRows = 64;   // fewest rows per CTA
constexpr int kOrthoMaxK = 256;  // basis vectors (restart <= 250)

// Sum over rows first, first + 256, ... < end of a[i] * c[i] for "threads"
// t = 0..255 (row first + t + 256 m), then their tree sum, all by one warp:
// lane l stands for threads l, l + 32, ..., l + 224. The total is on lane 0.
__device__ __forceinline__ double tree256_dot(const double* a, const double* c, int first, int end,
                                              int stride, int lane) {
  double t[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    double s = 0.0;
    for (int i = first + lane + 32 * m; i < end; i += stride) s = fma(__ldcg(a + i), __ldcg(c + i), s);
    t[m] = s;
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int m = 0; m < 4; ++m)
      if (m < o) t[m] += t[m + o];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t[0] += __shfl_down_sync(0xffffffffu, t[0], o);
  return t[0];
}

// Sum of p[0..n) by one warp, in every lane. ORDERED: one after the other.
template <bool ORDERED>
__device__ __forceinline__ double warp_total(const double* p, int n, int lane) {
  double s = 0.0;
  if (ORDERED) {
    for (int g0 = 0; g0 < n; g0 += 32) {
      const double x = g0 + lane < n ? __ldcg(p + g0 + lane) : 0.0;
      const int m = min(32, n - g0);
      for (int u = 0; u < m; ++u) s += __shfl_sync(0xffffffffu, x, u);
    }
  } else {
    for (int g = lane; g < n; g += 32) s += __ldcg(p + g);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;
}

template <bool ORDERED>
__global__ void __launch_bounds__(kOrthoThreads)
    k_ortho(int N, int k, const double* __restrict__ V, double* w, double* __restrict__ v,
            double* part, double* __restrict__ out, unsigned* ctr, unsigned base, DevErr* err) {
  __shared__ double hs[kOrthoMaxK];
  __shared__ double red[4][kOrthoRows];
  __shared__ double wsum[kOrthoThreads / 32];
  constexpr int kWarps = kOrthoThreads / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x, b = blockIdx.x;
  // ordered: always kRedBlocks chunks of rows, however many CTAs share them
  const int CH = ORDERED ? kRedBlocks : G;
  const int per = (N + CH - 1) / CH;
  auto begin = [&](int c) { return min(N, c * per); };
  auto end = [&](int c) { return min(N, begin(c) + per); };
  // not a number as the norm: the solver stops, and finds the error word
  auto give_up = [&]() {
    if (b == 0 && tid == 0) out[k] = __longlong_as_double(0x7ff8000000000000ll);
  };
  double nrm = 0.0;
  for (int pass = 0; pass < 2; ++pass) {
    double* pp = part + (size_t)pass * kOrthoMaxK * CH;
    // this CTA's part of every dot product: a warp per basis vector
    for (int c = b; c < CH; c += G) {
      const int i0 = begin(c), i1 = end(c);
      for (int j = warp; j < k; j += kWarps) {
        const double* vj = V + (size_t)j * N;
        double s = 0.0;
        if (ORDERED) {
          s = tree256_dot(vj, w, i0, i1, 256, lane);
        } else {
#pragma unroll 4
          for (int i = i0 + lane; i < i1; i += 32) s = fma(vj[i], w[i], s);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        }
        if (lane == 0) pp[(size_t)j * CH + c] = s;
      }
    }
    if (!grid_barrier(ctr, base + (unsigned)(pass + 1) * G, 61, err)) return give_up();
    if (ORDERED) {
      // a thread per vector adds the CTAs' parts in ascending order
      for (int j = tid; j < k; j += kOrthoThreads) {
        double s = 0.0;
#pragma unroll 8
        for (int g = 0; g < CH; ++g) s += __ldcg(pp + (size_t)j * CH + g);
        hs[j] = s;
        if (b == 0) out[j] = pass == 0 ? s : out[j] + s;
      }
    } else {
      for (int j = warp; j < k; j += kWarps) {
        const double s = warp_total<false>(pp + (size_t)j * CH, CH, lane);
        if (lane == 0) {
          hs[j] = s;
          if (b == 0) out[j] = pass == 0 ? s : out[j] + s;
        }
      }
    }
    __syncthreads();
    // w -= V h on this CTA's rows
    if (ORDERED) {
      for (int c = b; c < CH; c += G)
        for (int i = begin(c) + tid; i < end(c); i += kOrthoThreads) {
          double s = 0.0;
#pragma unroll 8
          for (int j = 0; j < k; ++j) s = fma(hs[j], V[(size_t)j * N + i], s);
          w[i] -= s;
        }
      __syncthreads();
    } else {
      // 64 rows at a time, the vectors over 4 groups
      const int i0 = begin(b), i1 = end(b);
      const int r = tid & (kOrthoRows - 1), q = tid / kOrthoRows;
      for (int c0 = i0; c0 < i1; c0 += kOrthoRows) {
        const int i = c0 + r;
        double s = 0.0;
        if (i < i1)
#pragma unroll 8
          for (int j = q; j < k; j += 4) s = fma(hs[j], V[(size_t)j * N + i], s);
        red[q][r] = s;
        __syncthreads();
        if (q == 0 && i < i1) {
          const double x = w[i] - ((red[0][r] + red[1][r]) + (red[2][r] + red[3][r]));
          w[i] = x;
          if (pass == 1) nrm = fma(x, x, nrm);
        }
        __syncthreads();
      }
    }
  }
  double* pn = part + (size_t)2 * kOrthoMaxK * CH;
  unsigned target = base + 3u * G;
  if (ORDERED) {
    // the norm's rows: 256 c + t + 256 CH m, of other CTAs' chunks too
    if (!grid_barrier(ctr, target, 61, err)) return give_up();
    target += G;
    for (int c = b + warp * G; c < CH; c += kWarps * G) {
      const double s = tree256_dot(w, w, 256 * c, N, 256 * CH, lane);
      if (lane == 0) pn[c] = s;
    }
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    if (lane == 0) wsum[warp] = nrm;
    __syncthreads();
    if (tid == 0) {
      double s = 0.0;
      for (int u = 0; u < kWarps; ++u) s += wsum[u];
      pn[b] = s;
    }
  }
  if (!grid_barrier(ctr, target, 61, err)) return give_up();
  const double hn = sqrt(warp_total<ORDERED>(pn, CH, lane));
  if (b == 0 && tid == 0) out[k] = hn;
  const double inv = 1.0 / hn;
  if (hn > 0.0)
    for (int c = b; c < CH; c += G)
      for (int i = begin(c) + tid; i < end(c); i += kOrthoThreads) v[i] = inv * w[i];
}

// The same step for small N by one cluster of 16 CTAs: the parts meet in
// distributed shared memory and hardware cluster barriers. Up to 200 rows per
// CTA: beyond that sixteen FP64 pipes take longer than the barriers save. Whole
// FP64 solves, ms, this form against k_ortho: 2,000 dofs 2.35 / 2.43, 3,001 3.17
// / 3.27, 4,000 4.53 / 4.48.
constexpr int kOrthoCluster = 16;
constexpr int kOrthoClusterRows = 200;  // rows per CTA

__global__ void __launch_bounds__(kOrthoThreads)
    k_ortho_cluster(int N, int k, const double* __restrict__ V, double* __restrict__ w,
                    double* __restrict__ v, double* __restrict__ out) {
  __shared__ double dots[2][kOrthoMaxK], hs[kOrthoMaxK], ws[kOrthoClusterRows];
  __shared__ double red[4][kOrthoRows], wsum[kOrthoThreads / 32], nsum;
  constexpr int kWarps = kOrthoThreads / 32;
  static_assert(kOrthoClusterRows <= kOrthoThreads, "a thread per row");
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, b = (int)cl.block_rank();
  const int per = (N + kOrthoCluster - 1) / kOrthoCluster;
  const int i0 = min(N, b * per), n = min(N, i0 + per) - i0;
  if (tid < n) ws[tid] = w[i0 + tid];
  __syncthreads();
  double nrm = 0.0;
  for (int pass = 0; pass < 2; ++pass) {
    for (int j = warp; j < k; j += kWarps) {
      const double* vj = V + (size_t)j * N + i0;
      double s = 0.0;
#pragma unroll 4
      for (int i = lane; i < n; i += 32) s = fma(vj[i], ws[i], s);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) dots[pass][j] = s;
    }
    cl.sync();
    // two vectors per warp and step: lane 16 h + r reads rank r's part
    for (int j0 = 2 * warp; j0 < k; j0 += 2 * kWarps) {
      const int j = j0 + (lane >> 4);
      double s = j < k ? cl.map_shared_rank(dots[pass], lane & 15)[j] : 0.0;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if ((lane & 15) == 0 && j < k) {
        hs[j] = s;
        if (b == 0) out[j] = pass == 0 ? s : out[j] + s;
      }
    }
    __syncthreads();
    // 64 rows at a time, the vectors over 4 groups
    const int r = tid & (kOrthoRows - 1), q = tid / kOrthoRows;
    for (int c0 = 0; c0 < n; c0 += kOrthoRows) {
      const int i = c0 + r;
      double s = 0.0;
      if (i < n)
#pragma unroll 8
        for (int j = q; j < k; j += 4) s = fma(hs[j], V[(size_t)j * N + i0 + i], s);
      red[q][r] = s;
      __syncthreads();
      if (q == 0 && i < n) {
        const double x = ws[i] - ((red[0][r] + red[1][r]) + (red[2][r] + red[3][r]));
        ws[i] = x;
        if (pass == 1) {
          nrm = fma(x, x, nrm);
          w[i0 + i] = x;
        }
      }
      __syncthreads();
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
  if (lane == 0) wsum[warp] = nrm;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int u = 0; u < kWarps; ++u) s += wsum[u];
    nsum = s;
  }
  cl.sync();
  double s = *cl.map_shared_rank(&nsum, lane & 15);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const double hn = sqrt(s);
  if (b == 0 && tid == 0) out[k] = hn;
  const double inv = 1.0 / hn;
  if (hn > 0.0 && tid < n) v[i0 + tid] = inv * ws[tid];
  cl.sync();  // no CTA leaves while another reads its shared memory
}

static cudaLaunchConfig_t ortho_cluster_config(cudaLaunchAttribute* attr, cudaStream_t s) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = kOrthoCluster;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(kOrthoCluster);
  c.blockDim = dim3(kOrthoThreads);
  c.stream = s;
  c.attrs = attr;
  c.numAttrs = 1;
  return c;
}

// Whether this device takes a cluster of 16 CTAs (it is beyond the portable
// size); asked once per device.
static bool ortho_cluster_fits() {
  static std::atomic<int> known[kMaxDev];  // 0: not asked, 1: yes, 2: no
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= kMaxDev) return false;
  int r = known[dev].load(std::memory_order_acquire);
  if (r == 0) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t c = ortho_cluster_config(&attr, nullptr);
    int n = 0;
    const bool ok = cudaFuncSetAttribute(k_ortho_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                         1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, k_ortho_cluster, &c) == cudaSuccess && n > 0;
    if (!ok) cudaGetLastError();
    r = ok ? 1 : 2;
    known[dev].store(r, std::memory_order_release);
  }
  return r == 1;
}

size_t ortho_part_size(int n_ctas) { return (size_t)(2 * kOrthoMaxK + 1) * n_ctas; }

// CTAs of k_ortho for N rows: at most one per SM (co-resident), and no more
// than give each kOrthoRows rows (fewer arrivals per barrier at small N).
// The ordered form always has kRedBlocks chunks.
int ortho_ctas(int N, int sms, bool ordered) {
  return ordered ? kRedBlocks : std::max(1, std::min(sms, N / kOrthoRows));
}

cudaError_t launch_ortho(int N, int k, const double* V, double* w, double* v, double* part,
                         double* out, unsigned* ctr, unsigned* epoch, int n_ctas, bool ordered,
                         DevErr* err, cudaStream_t s) {
  if (!ordered && N <= kOrthoCluster * kOrthoClusterRows && ortho_cluster_fits()) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t c = ortho_cluster_config(&attr, s);
    return cudaLaunchKernelEx(&c, k_ortho_cluster, N, k, V, w, v, out);
  }
  unsigned base = *epoch;
  void* args[] = {(void*)&N, (void*)&k, (void*)&V, (void*)&w, (void*)&v, (void*)&part,
                  (void*)&out, (void*)&ctr, (void*)&base, (void*)&err};
  const void* f = ordered ? (const void*)k_ortho<true> : (const void*)k_ortho<false>;
  const cudaError_t e = launch_coresident(n_ctas, [&](int n) {
    return cudaLaunchCooperativeKernel(f, dim3(n), dim3(kOrthoThreads), args, 0, s);
  });
  *epoch += (ordered ? 4u : 3u) * (unsigned)n_ctas;
  return e;
}

__global__ void k_axpy_basis(int N, int k, const double* __restrict__ V, const double* __restrict__ h,
                             double* __restrict__ w, double sign) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double s = 0;
#pragma unroll 8
  for (int j = 0; j < k; ++j) s = fma(h[j], V[(size_t)j * N + i], s);
  w[i] = fma(sign, s, w[i]);
}

cudaError_t launch_axpy_basis(int N, int k, const double* V, const double* h, double* w,
                              double sign, cudaStream_t s) {
  k_axpy_basis<<<(N + 255) / 256, 256, 0, s>>>(N, k, V, h, w, sign);
  return cudaGetLastError();
}

__global__ void k_scale(int N, const double* __restrict__ x, double a, double* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) y[i] = a * x[i];
}
cudaError_t launch_scale(int N, const double* x, double a, double* y, cudaStream_t s) {
  k_scale<<<(N + 255) / 256, 256, 0, s>>>(N, x, a, y);
  return cudaGetLastError();
}

__global__ void k_axpby(int N, double a, const double* __restrict__ x, double b,
                        double* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) y[i] = fma(a, x[i], b * y[i]);
}
cudaError_t launch_axpby(int N, double a, const double* x, double b, double* y, cudaStream_t s) {
  k_axpby<<<(N + 255) / 256, 256, 0, s>>>(N, a, x, b, y);
  return cudaGetLastError();
}

__global__ void k_nrm2_part(int N, const double* __restrict__ x, double* __restrict__ part) {
  __shared__ double red[256];
  double s = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
    s = fma(x[i], x[i], s);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}
// one warp; the parts added in ascending order
__global__ void k_nrm2_finish(int nb, const double* __restrict__ part, double* __restrict__ out) {
  const double s = warp_total<true>(part, nb, threadIdx.x);
  if (threadIdx.x == 0) out[0] = sqrt(s);
}
cudaError_t launch_nrm2(int N, const double* x, double* part, double* out, cudaStream_t s) {
  k_nrm2_part<<<kRedBlocks, 256, 0, s>>>(N, x, part);
  k_nrm2_finish<<<1, 32, 0, s>>>(kRedBlocks, part, out);
  return cudaGetLastError();
}

__global__ void k_gather(int N, const int* __restrict__ idx, const double* __restrict__ x,
                         double* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) y[i] = x[idx[i]];
}
cudaError_t launch_gather(int N, const int* idx, const double* x, double* y, cudaStream_t s) {
  k_gather<<<(N + 255) / 256, 256, 0, s>>>(N, idx, x, y);
  return cudaGetLastError();
}
__global__ void k_scatter(int N, const int* __restrict__ idx, const double* __restrict__ x,
                          double* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) y[idx[i]] = x[i];
}
cudaError_t launch_scatter(int N, const int* idx, const double* x, double* y, cudaStream_t s) {
  k_scatter<<<(N + 255) / 256, 256, 0, s>>>(N, idx, x, y);
  return cudaGetLastError();
}

// Caller-order rows of an internal-order matrix: out[r][q] = A[ip[r0+r]][ip[q]],
// or from the selected pairs: sel_j ? -P1 : P0.
__global__ void k_gather_rows(int N, int r0, const int* __restrict__ ip, const double* __restrict__ A,
                              const float2* __restrict__ P0, const float2* __restrict__ P1,
                              const uint8_t* __restrict__ sel, double* __restrict__ out) {
  const int r = blockIdx.y;
  const size_t src = (size_t)ip[r0 + r] * N;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x) {
    const int j = ip[q];
    double v;
    if (A) {
      v = A[src + j];
    } else if (sel[j]) {
      const float2 t = P1[src + j];
      v = -((double)t.x + (double)t.y);
    } else {
      const float2 t = P0[src + j];
      v = (double)t.x + (double)t.y;
    }
    out[(size_t)r * N + q] = v;
  }
}
cudaError_t launch_gather_rows(int N, int r0, int nr, const int* ip, const double* A,
                               const float2* P0, const float2* P1, const uint8_t* sel, double* out,
                               cudaStream_t s) {
  dim3 g(std::min(64, (N + 255) / 256), nr);
  k_gather_rows<<<g, 256, 0, s>>>(N, r0, ip, A, P0, P1, sel, out);
  return cudaGetLastError();
}

// After a boundary-condition change of the columns flips[0..nflip): the
// selected pairs swap roles, A2' = sel' ? -D : N = -B2 and B2' = -A2.
__global__ void k_reselect_pairs(int N, int nflip, const int* __restrict__ flips,
                                 float2* __restrict__ A2, float2* __restrict__ B2) {
  for (int i = blockIdx.y; i < N; i += gridDim.y)
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nflip; k += gridDim.x * blockDim.x) {
      const size_t o = (size_t)i * N + flips[k];
      const float2 a = A2[o], b = B2[o];
      A2[o] = make_float2(-b.x, -b.y);
      B2[o] = make_float2(-a.x, -a.y);
    }
}
cudaError_t launch_reselect_pairs(int N, int nflip, const int* flips, float2* A2, float2* B2,
                                  cudaStream_t s) {
  if (nflip == 0) return cudaSuccess;
  dim3 g(std::min(64, (nflip + 255) / 256), std::min(N, 65535));
  k_reselect_pairs<<<g, 256, 0, s>>>(N, nflip, flips, A2, B2);
  return cudaGetLastError();
}

}  // namespace wbem
