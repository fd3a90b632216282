// Plain (FP64) assembly of the single-layer matrix D (G) and the double-layer
// matrix N (dG/dn), the vertex-singular correction and alpha.
//
// Restates BEMProblem<3>::assemble_system (source/bem_problem.cc:106-590) and
// compute_alpha (:594-618) of the reference for the GPU:
//   - per-cell quadrature data (Q1 map, normal, JxW; :133-137, :192-196) is
//     computed once per assembly into a record per cell;
//   - k_tile_far gives each CTA a tile of 64 collocation rows x 80 dofs; the
//     records of the panels that touch the tile's dofs are staged into shared
//     memory by the TMA bulk-copy engine (cp.async.bulk, double-buffered on
//     mbarriers); the 4 shape-function entries of every regular panel
//     (:241-260) are accumulated in a shared-memory tile that is written out
//     with coalesced stores (k_tile_fp64 for rules of one and two points);
//   - panels that hold a node of the row's double-node set are skipped there
//     (:223-230) and integrated by k_singular_fp64 with the vertex-singular
//     rule (:478-522);
//   - alpha = N (-1) is a row reduction (:594-618).
#include <cuda_runtime.h>
#include <stdint.h>
#include "kernels.h"
#include "dfloat.cuh"
#include "panel_fp64.cuh"
#include "../../include/wbem.h"

namespace wbem {

constexpr double kInv4Pi = 0.07957747154594766788;  // 1 / (4 pi)

__device__ __forceinline__ void q1_geometry(const double P[4][3], double xi, double eta,
                                            double x[3], double cr[3]) {
  const double a0 = (1 - xi) * (1 - eta), a1 = xi * (1 - eta), a2 = (1 - xi) * eta, a3 = xi * eta;
  double jx[3], je[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    x[d] = a0 * P[0][d] + a1 * P[1][d] + a2 * P[2][d] + a3 * P[3][d];
    jx[d] = (1 - eta) * (P[1][d] - P[0][d]) + eta * (P[3][d] - P[2][d]);
    je[d] = (1 - xi) * (P[2][d] - P[0][d]) + xi * (P[3][d] - P[1][d]);
  }
  cr[0] = jx[1] * je[2] - jx[2] * je[1];
  cr[1] = jx[2] * je[0] - jx[0] * je[2];
  cr[2] = jx[0] * je[1] - jx[1] * je[0];
}

// Per-cell record: for each regular point q: {x, y, z, JxW/(4 pi), n_x JxW/(4 pi),
// n_y JxW/(4 pi), n_z JxW/(4 pi), 0}.
__global__ void k_cell_records_fp64(int C, const double* __restrict__ X,
                                    const int4* __restrict__ cell_dofs, double* __restrict__ rec,
                                    const __grid_constant__ PanelRule c_q) {
  const int nq = c_q.q1 * c_q.q1;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = gid / nq, q = gid % nq;
  if (c >= C) return;
  int4 d = cell_dofs[c];
  double P[4][3];
  const int id[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int e = 0; e < 3; ++e) P[k][e] = X[3 * (size_t)id[k] + e];
  double x[3], cr[3];
  q1_geometry(P, c_q.gp[q][0], c_q.gp[q][1], x, cr);
  const double w = c_q.gp[q][2] * kInv4Pi;
  const double det = sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
  double* r = rec + ((size_t)c * nq + q) * 8;
  r[0] = x[0];
  r[1] = x[1];
  r[2] = x[2];
  r[3] = det * w;
  r[4] = cr[0] * w;
  r[5] = cr[1] * w;
  r[6] = cr[2] * w;
  r[7] = 0.0;
}

cudaError_t launch_cell_records_fp64(int C, const double* X, const int4* cell_dofs, double* rec,
                                     const PanelRule& rule, cudaStream_t s) {
  const long total = (long)C * rule.q1 * rule.q1;
  const int bs = 128;
  k_cell_records_fp64<<<(unsigned)((total + bs - 1) / bs), bs, 0, s>>>(C, X, cell_dofs, rec, rule);
  return cudaGetLastError();
}

__device__ __forceinline__ bool in_set(const int set[kMaxSet], int v) {
  bool r = false;
#pragma unroll
  for (int k = 0; k < kMaxSet; ++k) r |= (set[k] == v);
  return r;
}

constexpr int kChunk = 6;  // panels per staged chunk

// Two threads per row (2 * kRowsF64 threads): each takes every other
// quadrature point of a panel; the partial sums are combined through a lane
// shuffle, then one thread adds the N entries and the other the D entries.
constexpr int kF64Threads = 2 * kRowsF64;

template <int Q1>
__global__ void __launch_bounds__(kF64Threads)
    k_tile_fp64(int N, const double* __restrict__ X, const int* __restrict__ dnset,
                const int* __restrict__ tile_ptr, const int2* __restrict__ tile_ent,
                const int4* __restrict__ cell_dofs, const double* __restrict__ rec,
                double* __restrict__ Nm, double* __restrict__ Dm, DevErr* err,
                const __grid_constant__ PanelRule c_q) {
  constexpr int NQ = Q1 * Q1;
  constexpr int RECD = NQ * 8;  // doubles per panel record
  constexpr int RT = kRowsF64, CT = kColsPerTileF64, LDA = RT + 1;
  extern __shared__ __align__(128) unsigned char smem[];
  double* stage = reinterpret_cast<double*>(smem);  // [2][kChunk][RECD], 128-byte aligned
  double* accN = stage + 2 * kChunk * RECD;         // [CT][LDA]
  double* accD = accN + CT * LDA;
  ChunkMeta* meta = reinterpret_cast<ChunkMeta*>(accD + CT * LDA);
  uint64_t* bar = reinterpret_cast<uint64_t*>(meta + 2 * kChunk);

  const int tid = threadIdx.x;
  const int rt = tid >> 1, half = tid & 1;  // row in the tile, point parity
  const int tile = blockIdx.x;
  const int row0 = blockIdx.y * RT;
  const int row = row0 + rt;
  const bool active = row < N;
  double xi = 0, yi = 0, zi = 0;
  int set[kMaxSet];
#pragma unroll
  for (int k = 0; k < kMaxSet; ++k) set[k] = -2;
  if (active) {
    xi = X[3 * (size_t)row];
    yi = X[3 * (size_t)row + 1];
    zi = X[3 * (size_t)row + 2];
#pragma unroll
    for (int k = 0; k < kMaxSet; ++k) set[k] = dnset[(size_t)row * kMaxSet + k];
  }
  for (int k = tid; k < CT * LDA; k += kF64Threads) {
    accN[k] = 0.0;
    accD[k] = 0.0;
  }
  const int e0 = tile_ptr[tile], e1 = tile_ptr[tile + 1];
  const int nch = (e1 - e0 + kChunk - 1) / kChunk;
  auto load_meta = [&](int c) {
    const int k = tid - 32;
    const int base = e0 + c * kChunk;
    if (k >= 0 && k < kChunk && base + k < e1) {
      const int2 ent = tile_ent[base + k];
      ChunkMeta m;
      m.cell = ent.x & 0x7fffffff;
      m.slots = (uint32_t)ent.y;
      m.owner = ent.x < 0;
      m.pad = 0;
      m.dofs = cell_dofs[m.cell];
      m.geo = make_float4(0.f, 0.f, 0.f, 0.f);
      meta[(c & 1) * kChunk + k] = m;
    }
  };
  if (nch > 0) load_meta(0);
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();

  auto issue = [&](int c) {
    const int sidx = c & 1;
    const int base = e0 + c * kChunk;
    const int cnt = min(kChunk, e1 - base);
    mbar_arrive_expect_tx(&bar[sidx], (uint32_t)(cnt * RECD * 8));
    for (int k = 0; k < cnt; ++k) {
      const int cell = tile_ent[base + k].x & 0x7fffffff;
      bulk_g2s(stage + (size_t)(sidx * kChunk + k) * RECD, rec + (size_t)cell * RECD,
               (uint32_t)(RECD * 8), &bar[sidx]);
    }
  };
  if (tid == 0 && nch > 0) issue(0);
  bool in_flight_next = false;

  for (int c = 0; c < nch; ++c) {
    if (tid == 0 && c + 1 < nch) {
      fence_proxy_async_smem();
      issue(c + 1);
    }
    if (c + 1 < nch) load_meta(c + 1);
    in_flight_next = (c + 1 < nch);
    const bool ok = mbar_wait_bounded(&bar[c & 1], (uint32_t)((c >> 1) & 1));
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        dev_fail(err, WBEM_ERR_TIMEOUT, 11, tile, c);
        if (in_flight_next) mbar_wait_bounded(&bar[(c + 1) & 1], (uint32_t)(((c + 1) >> 1) & 1));
      }
      return;
    }
    const int base = e0 + c * kChunk;
    const int cnt = min(kChunk, e1 - base);
    for (int k = 0; k < cnt; ++k) {
      const ChunkMeta& mt = meta[(c & 1) * kChunk + k];
      const uint32_t slots = mt.slots;
      const int4 d = mt.dofs;
      const bool sing = in_set(set, d.x) || in_set(set, d.y) || in_set(set, d.z) || in_set(set, d.w);
      // a skipped row (inactive, or the panel is singular for it) runs no
      // points but still takes part in the shuffle below: every lane of the
      // warp reaches it
      const bool skip = !active || sing;
      const double* r = stage + (size_t)((c & 1) * kChunk + k) * RECD;
      double ln0 = 0, ln1 = 0, ln2 = 0, ln3 = 0, ld0 = 0, ld1 = 0, ld2 = 0, ld3 = 0;
#pragma unroll 4
      for (int q = skip ? NQ : half; q < NQ; q += 2) {
        const double2 p01 = *reinterpret_cast<const double2*>(r + q * 8);
        const double2 p23 = *reinterpret_cast<const double2*>(r + q * 8 + 2);
        const double2 p45 = *reinterpret_cast<const double2*>(r + q * 8 + 4);
        const double p6 = r[q * 8 + 6];
        const double Rx = p01.x - xi, Ry = p01.y - yi, Rz = p23.x - zi;
        const double r2 = fma(Rx, Rx, fma(Ry, Ry, Rz * Rz));
        const double ri = rsqrt(r2);
        const double sq = ri * p23.y;
        const double rn = fma(Rx, p45.x, fma(Ry, p45.y, Rz * p6));
        const double dq = -rn * (ri * ri * ri);
        ln0 = fma(dq, c_q.phi[q][0], ln0);
        ln1 = fma(dq, c_q.phi[q][1], ln1);
        ln2 = fma(dq, c_q.phi[q][2], ln2);
        ln3 = fma(dq, c_q.phi[q][3], ln3);
        ld0 = fma(sq, c_q.phi[q][0], ld0);
        ld1 = fma(sq, c_q.phi[q][1], ld1);
        ld2 = fma(sq, c_q.phi[q][2], ld2);
        ld3 = fma(sq, c_q.phi[q][3], ld3);
      }
      // the row's sums: even points + odd points (the same on both threads)
      double lnv[4] = {ln0, ln1, ln2, ln3}, ldv[4] = {ld0, ld1, ld2, ld3};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double on = __shfl_xor_sync(0xffffffffu, lnv[j], 1);
        const double od = __shfl_xor_sync(0xffffffffu, ldv[j], 1);
        lnv[j] = half ? on + lnv[j] : lnv[j] + on;
        ldv[j] = half ? od + ldv[j] : ldv[j] + od;
      }
      if (skip) continue;
      double* acc = half ? accD : accN;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t sl = (slots >> (8 * j)) & 255u;
        if (sl != 255u) acc[sl * LDA + rt] += half ? ldv[j] : lnv[j];
      }
    }
    __syncthreads();
  }

  // coalesced write-out of the tile (row-major N x N); the tile's columns:
  // tile_ptr[gridDim.x + 1 + tile] .. (+ 1)
  const int col0 = tile_ptr[gridDim.x + 1 + tile], ncol = tile_ptr[gridDim.x + 2 + tile] - col0;
  for (int idx = tid; idx < RT * CT; idx += kF64Threads) {
    const int rr = idx / CT, cc = idx % CT;
    const int gr = row0 + rr, gc = col0 + cc;
    if (gr < N && cc < ncol) {
      Nm[(size_t)gr * N + gc] = accN[cc * LDA + rr];
      Dm[(size_t)gr * N + gc] = accD[cc * LDA + rr];
    }
  }
}

// ---- the far field: 64-bit centre terms and remainders in pairs of FP32
//
// Point by point in FP64 a pair of row and panel takes 545 FP64 instructions
// at 4 x 4 points, and each occupies the FP64 pipe for 64 cycles: k_tile_fp64
// is bound by that pipe. Where the row is at least six times as far from the
// panel's centre as the panel's vertices are, an entry is one value at the
// centre plus a small remainder. With R0 = centre - row, w = 1 / |R0| and
// centred coordinates s, t in [-1/2, 1/2], a point is
//   R = R0 + d,  d = s F + t E + s t W,  its weighted normal  c = c0 + s c1 + t c2,
//   e = e1 + e2,  e1 = 2 w^2 R0 . d,  e2 = w^2 |d|^2,
//   1/|R|   = w   (1 + f),  f  = (1 + e)^(-1/2) - 1,
//   1/|R|^3 = w^3 (1 + g),  g  = (1 + e)^(-3/2) - 1 = f (3 + f (3 + f)),
//   R . c   = R0 . (c0 + s c1 + t c2) - V s t,   V = W . c0.
// The "1" terms sum over the points to one FP64 product per entry: the record
// holds the sums of J phi_v, and those of R . c phi_v are R0 . c0 / 4, R0 . c1
// / 24 and so on (the rule is exact for them). Only the f and g sums run over
// the points, in pairs of FP32 numbers (48 bits). Up to a distance ratio of 32
// (far_pair<true>) the terms of first order in e1 are summed in FP64 as well
// (from the record's sums of J phi_v {s, t, s t}, and exact integrals for N),
// and the points add what is left,
//   f + e1/2  = f^2 (3/2 + f) (1 + e) - e2/2,
//   g + 3e1/2 = f^2 (3 + f) + 3 (f + e1/2),
// which keeps its relative accuracy because f^2 is a product. The centre terms
// carry a little more than 64 bits (low parts of w, w^3, the centre, c0 and
// the sums), since no 16 points average their rounding.
// RMS error of a matrix's entries against 80-bit sums, relative to D_ij and
// D_ij / r_ij, here / point by point in FP64, units of 1e-17:
//   tank of 2,000 dofs    D 9.0 / 10.9, N 7.1 / 7.6
//   tank of 7,000         D 8.6 / 11.5, N 7.0 / 7.8
//   sphere of 5,402       D 8.3 / 11.2, N 8.1 / 8.7
// and at 300 dofs (tank; cube-sphere as it is, stretched 30:1, roughened by 6%,
// graded 1:12), sums in 113 bits: at 4 x 4 points D 0.81 to 0.92 of point by
// point, N 0.92 to 1.01; at 3, 5 and 6 points per direction D 0.80 to 0.99, N
// 0.90 to 1.16 (the sphere's; 8.9e-17 where it was 7.7e-17).
// Time of the far field (point by point before): 1.5 ms (4.2) at 2,000 dofs,
// 9.6 (32.1) at 5,402, 69.8 (283) at 16,226. Per 32 pairs: 67 FP64
// instructions (113 with first order) and 3,000 to 4,000 FP32 and integer
// ones; the FP64 pipe is still the bound (71% busy).

constexpr float kFarRatio = 6.f;       // |R0| over the panel's largest centre-vertex distance
// above this, the centre term without first order (fewer points average less)
template <int Q1>
constexpr float kFarFirstRatio = Q1 < 4 ? 64.f : 32.f;
constexpr int kFarRowThreads = 4;   // threads of a row; each takes every fourth panel of a chunk
constexpr int kFarThreads = kFarRowThreads * kRowsF64;
constexpr int kFarChunk = 16;       // panels per staged chunk

// centred 1-D rule: |node - 1/2| of the point pairs from the outside in (a
// centre point is left out), all nodes and the weights, as pairs
struct FarTables {
  float2 s[kMaxQ1 / 2], ws[kMaxQ1 / 2], wp[kMaxQ1 / 2];  // node, weight * node, weight of a pair
  float2 wc;                                             // weight of the centre point
  float2 t[kMaxQ1], w[kMaxQ1], wt[kMaxQ1];               // node, weight, weight * node
};

constexpr size_t kFarHeader = 256;  // the scale, before the records

static FarTables far_tables(const PanelRule& t) {
  const int n = t.q1;
  auto pair = [](double x) { return make_float2((float)x, (float)(x - (double)(float)x)); };
  FarTables f{};
  for (int b = 0; b < n; ++b) {
    double w = 0.0;  // the 1-D weight: the 2-D ones of a row, whose other factors add to 1
    for (int a = 0; a < n; ++a) w += t.gp[b * n + a][2];
    const double x = t.gp[b * n][1] - 0.5;
    f.t[b] = pair(x);
    f.w[b] = pair(w);
    f.wt[b] = pair(w * x);
    if (2 * b + 1 == n) f.wc = pair(w);
    if (2 * b + 1 > n) {  // the outermost pair first
      f.s[n - 1 - b] = pair(x);
      f.ws[n - 1 - b] = pair(w * x);
      f.wp[n - 1 - b] = pair(w);
    }
  }
  return f;
}

// lengths are scaled by the power of two that brings the mesh's largest
// coordinate into [2^8, 2^9), so that FP32's exponents suffice in any unit;
// D is a length (divided by the scale where it is written out), N a number
template <int Q1>
struct alignas(16) FarRecord {
  static constexpr int NC = (Q1 + 1) / 2;
  double c[3], c0[3], c1[3], c2[3];  // centre, weighted-normal coefficients / (4 pi)
  double d[3][3];                    // 2 F, 2 E, 2 W
  double M[4], V144;                 // sums of J phi_v / (4 pi), V / 144
  double Q[4][3];                    // sums of -J phi_v {s, t, s t} / 2 / (4 pi)
  double pad_;
  float cl[3], c0l[3], Ml[4];        // low parts of c, c0 and M
  float thr, thr1;                   // |R0|^2 above which the pair is far / takes far_pair<false>
  float2 V;
  float2 D1[Q1];                     // row t_b: |d|^2 = D0 + s D1 + s^2 D2
  float2 dE[Q1][NC];                 // D0 + s_a^2 D2
  float2 J[Q1][Q1];                  // J weight / (4 pi)
};

struct dd {
  double h, l;
};
__device__ __forceinline__ dd dd_sum(double a, double b) {
  const double s = __dadd_rn(a, b), bb = __dsub_rn(s, a);
  return {s, __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb))};
}
__device__ __forceinline__ dd dd_add(dd a, dd b) {
  dd s = dd_sum(a.h, b.h);
  return dd_sum(s.h, s.l + (a.l + b.l));
}
__device__ __forceinline__ dd dd_sub(dd a, dd b) { return dd_add(a, {-b.h, -b.l}); }
__device__ __forceinline__ dd dd_mul(dd a, dd b) {
  const double p = __dmul_rn(a.h, b.h);
  return dd_sum(p, fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
__device__ __forceinline__ float2 pair_of(double x) {
  const float h = (float)x;
  return make_float2(h, (float)(x - (double)h));
}

// scale[0]: the power of two that brings the largest coordinate into [2^8, 2^9);
// scale[1]: its inverse
__global__ void k_mesh_scale(int n3, const double* __restrict__ X, double* __restrict__ scale) {
  __shared__ double part[32];
  double m = 0.0;
  bool fin = true;
  for (int i = threadIdx.x; i < n3; i += blockDim.x) {
    const double a = fabs(X[i]);
    fin &= isfinite(a);
    m = fmax(m, a);
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  fin = __syncthreads_and(fin);
  if (threadIdx.x == 0) {
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k) m = fmax(m, part[k]);
    // outside 2^+-500 no panel counts as far (k_far_records)
    scale[0] = fin && m > 0.0 ? scalbn(1.0, 8 - ilogb(m)) : 1.0;
    scale[1] = 1.0 / scale[0];
  }
}

// 16 lanes per panel (a warp where the rule has more than 16 points); every
// lane computes the panel's centre terms, then its own points.
template <int Q1>
__global__ void __launch_bounds__(128)
    k_far_records(int C, const double* __restrict__ X, const int4* __restrict__ cell_dofs,
                  const double* __restrict__ scale, FarRecord<Q1>* __restrict__ out,
                  const __grid_constant__ PanelRule c_q) {
  constexpr int NQ = Q1 * Q1, G = NQ <= 16 ? 16 : 32, NC = FarRecord<Q1>::NC;
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) / G, lane = threadIdx.x % G;
  if (c - (int)(threadIdx.x % 32) / G >= C) return;  // the whole warp
  const bool on = c < C;
  const int4 id4 = cell_dofs[on ? c : C - 1];
  const int id[4] = {id4.x, id4.y, id4.z, id4.w};
  const double S = scale[0];
  double P[4][3];
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int e = 0; e < 3; ++e) P[k][e] = X[3 * (size_t)id[k] + e] * S;
  dd F[3], E[3], W[3], cen[3], c0[3];
  double c1[3], c2[3], dmax2 = 0.0;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const dd a = dd_sum(P[1][e], -P[0][e]), b = dd_sum(P[3][e], -P[2][e]);
    const dd u = dd_sum(P[2][e], -P[0][e]), v = dd_sum(P[3][e], -P[1][e]);
    const dd f = dd_add(a, b), g = dd_add(u, v);
    F[e] = {0.5 * f.h, 0.5 * f.l};
    E[e] = {0.5 * g.h, 0.5 * g.l};
    W[e] = dd_sub(b, a);
    const dd s = dd_add(dd_sum(P[0][e], P[1][e]), dd_sum(P[2][e], P[3][e]));
    cen[e] = {0.25 * s.h, 0.25 * s.l};
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    double r = 0.0;
#pragma unroll
    for (int e = 0; e < 3; ++e) r = fma(P[k][e] - cen[e].h, P[k][e] - cen[e].h, r);
    dmax2 = fmax(dmax2, r);
  }
  const dd i4 = {kInv4Pi, -4.9196691687956215e-18};
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    const int a = (e + 1) % 3, b = (e + 2) % 3;
    c0[e] = dd_mul(i4, dd_sub(dd_mul(F[a], E[b]), dd_mul(F[b], E[a])));
    c1[e] = (F[a].h * W[b].h - F[b].h * W[a].h) * kInv4Pi;
    c2[e] = (W[a].h * E[b].h - W[b].h * E[a].h) * kInv4Pi;
  }
  const double V = W[0].h * c0[0].h + W[1].h * c0[1].h + W[2].h * c0[2].h;
  // |c0| to twice 64 bits; the points add |c| - |c0|, small unless the panel is strongly skewed
  const dd n2 = dd_add(dd_add(dd_mul(c0[0], c0[0]), dd_mul(c0[1], c0[1])), dd_mul(c0[2], c0[2]));
  const double m0 = sqrt(n2.h), m0l = m0 > 0.0 ? 0.5 * (fma(-m0, m0, n2.h) + n2.l) / m0 : 0.0;
  FarRecord<Q1>* r = out + (on ? c : C - 1);
  double sum[16] = {};
  for (int q = lane; q < NQ; q += G) {
    const double s = c_q.gp[q][0] - 0.5, t = c_q.gp[q][1] - 0.5, w = c_q.gp[q][2];
    double cc = 0.0, g = 0.0;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const double k = fma(s, c1[e], t * c2[e]);
      cc = fma(k, fma(2.0, c0[e].h, k), cc);  // |c|^2 - |c0|^2
      g = fma(c0[e].h + k, c0[e].h + k, g);
    }
    const double len = sqrt(g), dev = len + m0 > 0.0 ? cc / (len + m0) * w : 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double g2 = -0.5 * len * w * c_q.phi[q][j];
      sum[j] = fma(dev, c_q.phi[q][j], sum[j]);
      sum[4 + 3 * j] = fma(g2, s, sum[4 + 3 * j]);
      sum[5 + 3 * j] = fma(g2, t, sum[5 + 3 * j]);
      sum[6 + 3 * j] = fma(g2, s * t, sum[6 + 3 * j]);
    }
    if (on) r->J[q / Q1][q % Q1] = pair_of(len * w);
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
    for (int j = 0; j < 16; ++j) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], o);
  if (!on) return;
  for (int k = lane; k < Q1 * NC; k += G) {
    const int b = k / NC, a = k % NC;
    const double t = c_q.gp[b * Q1][1] - 0.5, s = c_q.gp[Q1 - 1 - a][0] - 0.5;
    double D0 = 0.0, D1 = 0.0, D2 = 0.0;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const double g = fma(t, W[e].h, F[e].h), u = t * E[e].h;
      D0 = fma(u, u, D0);
      D1 = fma(2.0 * u, g, D1);
      D2 = fma(g, g, D2);
    }
    r->dE[b][a] = pair_of(fma(s * s, D2, D0));
    if (a == 0) r->D1[b] = pair_of(D1);
  }
  if (lane != 0) return;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    r->c[e] = cen[e].h;
    r->cl[e] = (float)cen[e].l;
    r->c0[e] = c0[e].h;
    r->c0l[e] = (float)c0[e].l;
    r->c1[e] = c1[e];
    r->c2[e] = c2[e];
    r->d[0][e] = 2.0 * F[e].h;
    r->d[1][e] = 2.0 * E[e].h;
    r->d[2][e] = 2.0 * W[e].h;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const dd m = dd_sum(0.25 * m0, fma(0.25, m0l, sum[j]));
    r->M[j] = m.h;
    r->Ml[j] = (float)m.l;
#pragma unroll
    for (int e = 0; e < 3; ++e) r->Q[j][e] = sum[4 + 3 * j + e];
  }
  r->V144 = V / 144.0;
  r->V = pair_of(V);
  r->pad_ = 0.0;
  r->thr1 = (float)(kFarFirstRatio<Q1> * kFarFirstRatio<Q1> * dmax2);
  // within these ranges the pairs keep their 48 bits (panels down to 2^-24 of
  // the mesh's size); other panels are never far
  const bool ok = dmax2 >= 0x1p-32 && dmax2 <= 0x1p+20 && m0 >= 0x1p-60 && S >= 0x1p-500 &&
                  S <= 0x1p+500;
  r->thr = ok ? (float)(kFarRatio * kFarRatio * dmax2) : __int_as_float(0x7f800000);
}

// the eight sums of a far pair: ln (N) and ld (D), R0 = centre - row
template <int Q1, bool SECOND>
__device__ __forceinline__ void far_pair(const FarRecord<Q1>& r, double Rx, double Ry, double Rz,
                                         double p, float p1, const FarTables& c_far, double ln[4],
                                         double ld[4]) {
  constexpr int NP = Q1 / 2, NC = FarRecord<Q1>::NC;
  // w = 1 / |R0| and its low part: a third-order step from the FP32 root
  float yf;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(p1));
  const double y = widen(yf), e1 = fma(-p, y * y, 1.0), ce = fma(e1, 0.375, 0.5), ye = y * e1;
  const double w = fma(ye, ce, y), wlo = fma(ye, ce, y - w);
  const double w2 = w * w, w3 = w * w2;
  const df dx = pair_split(Rx), dy = pair_split(Ry), dz = pair_split(Rz), wd = pair_split(w);
  const df W2 = pair_split(w2), W3 = pair_split(w3);
  const float wf = wd.hi, w3f = W3.hi;
  const float rc = fmaf(dx.hi, r.cl[0], fmaf(dy.hi, r.cl[1], dz.hi * r.cl[2]));
  const float wl = fmaf(-w3f, rc, cut_to_float(wlo));  // w + wl
  // w^3 (1 + w3l): from wl and the roundings of w^2 and w^3
  const float w3l = (fmaf(3.f, wl, wf * (cut_to_float(fma(w, w, -w2)) * (p1)))) * (p1 * wf) +
                    cut_to_float(fma(w, w2, -w3)) * (p1 * p1 * wf);
  const double A = fma(Rx, r.c0[0], fma(Ry, r.c0[1], Rz * r.c0[2]));
  const double B = fma(Rx, r.c1[0], fma(Ry, r.c1[1], Rz * r.c1[2]));
  const double C = fma(Rx, r.c2[0], fma(Ry, r.c2[1], Rz * r.c2[2]));
  const df Ad = pair_split(A), Bd = pair_split(B), Cd = pair_split(C), Vd = pair_load(r.V);
  // 2 w^2 R0 . {F, E, W}
  df al[3];
  double ad[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    ad[k] = fma(Rx, r.d[k][0], fma(Ry, r.d[k][1], Rz * r.d[k][2]));
    if constexpr (SECOND) {
      ad[k] *= w2;
      al[k] = pair_split(ad[k]);
    } else {
      al[k] = pair_norm(pair_mul(pair_split(ad[k]), W2));
    }
  }
  // centred moments of the remainders: sums of f, s f, t f, s t f
  df D00 = {0, 0}, D10 = {0, 0}, D01 = {0, 0}, D11 = {0, 0};
  df N00 = {0, 0}, N10 = {0, 0}, N01 = {0, 0}, N11 = {0, 0};
#pragma unroll 1
  for (int b = 0; b < Q1; ++b) {
    const df t = pair_load(c_far.t[b]);
    const df beta = pair_mul(al[1], t);
    const df D1 = pair_mul(W2, pair_load(r.D1[b]));
    const df gam = pair_norm(pair_add(pair_add(al[0], pair_mul(al[2], t)), D1));
    const df T0 = pair_norm(pair_add(Ad, pair_mul(Cd, t)));
    const df Bb = pair_norm(pair_sub(Bd, pair_mul(Vd, t)));
    df sD = {0, 0}, s1D = {0, 0}, sN = {0, 0}, s1N = {0, 0};
    auto point = [&](df e, df e2, df T, df J, df& fD, df& fN) {
      // y ~ (1 + e)^(-1/2) in FP32; z = (1 + e) y^2 - 1 in pairs; fD = y (1 - z/2 + 3 z^2 / 8) - 1
      float y0;
      asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(__fadd_rn(1.f, e.hi)));
      const df q = pair_prod(y0, y0), pe = pair_prod(e.hi, q.hi);
      const df z1 = pair_sum(__fadd_rn(__fsub_rn(q.hi, 1.f), pe.hi), q.lo);
      const float zl = __fadd_rn(z1.lo, __fmaf_rn(e.lo, q.hi, __fmaf_rn(e.hi, q.lo, pe.lo)));
      const df bz = pair_prod(y0, -0.5f * z1.hi);
      const float c2 = __fmaf_rn(0.375f * z1.hi, z1.hi, -0.5f * zl);
      df f = pair_fast(__fsub_rn(y0, 1.f), bz.hi);
      f.lo = __fadd_rn(f.lo, __fmaf_rn(y0, c2, bz.lo));
      df u = pair_fast(3.f, f.hi);
      u.lo = __fadd_rn(u.lo, f.lo);
      if constexpr (SECOND) {
        const df f2 = pair_norm(pair_mul(f, f));
        df g = pair_fast(1.f, e.hi), h = pair_fast(1.5f, f.hi);
        g.lo = __fadd_rn(g.lo, e.lo);
        h.lo = __fadd_rn(h.lo, f.lo);
        const df gD = pair_add(pair_mul(f2, pair_mul(g, h)), {-0.5f * e2.hi, -0.5f * e2.lo});
        fD = pair_mul(J, gD);
        fN = pair_mul(T, pair_add(pair_mul(f2, u), pair_mul(gD, {3.f, 0.f})));
      } else {
        const df v = pair_mul(f, u);
        df x = pair_fast(3.f, v.hi);
        x.lo = __fadd_rn(x.lo, v.lo);
        fD = pair_mul(J, f);
        fN = pair_mul(T, pair_mul(f, x));
      }
    };
#pragma unroll
    for (int a = 0; a < NP; ++a) {
      const df s = pair_load(c_far.s[a]);
      const df D0 = pair_mul(W2, pair_load(r.dE[b][a])), D1s = pair_mul(D1, s);
      const df even = pair_add(beta, D0), odd = pair_mul(gam, s);
      df ep = pair_sum(even.hi, odd.hi), em = pair_sum(even.hi, -odd.hi);
      ep = pair_fast(ep.hi, __fadd_rn(ep.lo, __fadd_rn(even.lo, odd.lo)));
      em = pair_fast(em.hi, __fadd_rn(em.lo, __fsub_rn(even.lo, odd.lo)));
      const df Ts = pair_mul(Bb, s);
      df fDp, fNp, fDm, fNm;
      point(ep, pair_add(D0, D1s), pair_add(T0, Ts), pair_load(r.J[b][Q1 - 1 - a]), fDp, fNp);
      point(em, pair_sub(D0, D1s), pair_sub(T0, Ts), pair_load(r.J[b][a]), fDm, fNm);
      const df D_ = pair_add(fDp, fDm), Dd = pair_mul(pair_sub(fDp, fDm), s);
      const df N_ = pair_mul(pair_add(fNp, fNm), pair_load(c_far.wp[a]));
      const df Nd = pair_mul(pair_sub(fNp, fNm), pair_load(c_far.ws[a]));
      sD = a ? pair_add(sD, D_) : D_;
      s1D = a ? pair_add(s1D, Dd) : Dd;
      sN = a ? pair_add(sN, N_) : N_;
      s1N = a ? pair_add(s1N, Nd) : Nd;
    }
    if constexpr (NC > NP) {
      const df D0 = pair_mul(W2, pair_load(r.dE[b][NP]));
      const df e = pair_norm(pair_add(beta, D0));
      df fD, fN;
      point(e, D0, T0, pair_load(r.J[b][NP]), fD, fN);
      sD = pair_add(sD, fD);
      sN = pair_add(sN, pair_mul(fN, pair_load(c_far.wc)));
    }
    const df wb = pair_load(c_far.w[b]), wt = pair_load(c_far.wt[b]);
    sD = pair_norm(sD);
    s1D = pair_norm(s1D);
    sN = pair_norm(sN);
    s1N = pair_norm(s1N);
    D00 = pair_add(D00, sD);
    D10 = pair_add(D10, s1D);
    D01 = pair_add(D01, pair_mul(sD, t));
    D11 = pair_add(D11, pair_mul(s1D, t));
    N00 = pair_add(N00, pair_mul(sN, wb));
    N10 = pair_add(N10, pair_mul(s1N, wb));
    N01 = pair_add(N01, pair_mul(sN, wt));
    N11 = pair_add(N11, pair_mul(s1N, wt));
  }
  // entries: phi_v = (1/2 -+ s) (1/2 -+ t)
  auto corners = [](df m00, df m10, df m01, df m11, df v[4]) {
    const df q = {0.25f * m00.hi, 0.25f * m00.lo};
    const df P = pair_add(q, m11), Q = pair_sub(q, m11);
    const df Rp = pair_half(pair_add(m10, m01)), Rm = pair_half(pair_sub(m10, m01));
    v[0] = pair_sub(P, Rp);
    v[1] = pair_add(Q, Rm);
    v[2] = pair_sub(Q, Rm);
    v[3] = pair_add(P, Rp);
  };
  df v[4];
  corners(D00, D10, D01, D11, v);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const df g = pair_mul(pair_norm(v[j]), wd);
    const float lo = fmaf(cut_to_float(r.M[j]), wl, fmaf(wf, r.Ml[j], g.lo));
    double m = r.M[j];
    if constexpr (SECOND) m = fma(ad[0], r.Q[j][0], fma(ad[1], r.Q[j][1], fma(ad[2], r.Q[j][2], m)));
    ld[j] = fma(w, m, widen(g.hi) + widen(lo));
  }
  corners(N00, N10, N01, N11, v);
  double Pd = fma(0.25, A, -r.V144), Qd = fma(0.25, A, r.V144), Kp = B + C, Km = B - C;
  if constexpr (SECOND) {
    // centred moments of -3/2 (R . c) e1, by the exact integrals of s^2 and t^2
    const double a0 = -1.5 * ad[0], a1 = -1.5 * ad[1], a2 = -1.5 * ad[2];
    const double A12 = A * (1.0 / 12.0), A144 = A * (1.0 / 144.0), B144 = B * (1.0 / 144.0), C144 = C * (1.0 / 144.0);
    const double n00 = fma(12.0, fma(B144, a0, C144 * a1), -r.V144 * a2);
    const double n10 = fma(A12, a0, fma(C144, a2, -r.V144 * a1));
    const double n01 = fma(A12, a1, fma(B144, a2, -r.V144 * a0));
    const double n11 = fma(A144, a2, fma(B144, a1, C144 * a0));
    Pd = fma(0.25, n00, Pd + n11);
    Qd = fma(0.25, n00, Qd - n11);
    Kp = fma(12.0, n10 + n01, Kp);
    Km = fma(12.0, n10 - n01, Km);
  }
  const double i24 = 1.0 / 24.0;
  const double dot[4] = {fma(-i24, Kp, Pd), fma(i24, Km, Qd), fma(-i24, Km, Qd), fma(i24, Kp, Pd)};
  const float k0 = fmaf(dx.hi, r.c0l[0], fmaf(dy.hi, r.c0l[1], dz.hi * r.c0l[2])) +
                   fmaf(r.cl[0], cut_to_float(r.c0[0]),
                        fmaf(r.cl[1], cut_to_float(r.c0[1]), r.cl[2] * cut_to_float(r.c0[2])));
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const df g = pair_mul(pair_norm(v[j]), W3);
    const float lo = fmaf(w3f, fmaf(0.25f, k0, cut_to_float(dot[j]) * w3l), g.lo);
    ln[j] = fma(-w3, dot[j], -(widen(g.hi) + widen(lo)));
  }
}

// One CTA per (kRowsF64 rows, column tile), four threads per row, each on its
// own panel of a staged chunk. Pairs that are not far are collected by ballot
// and integrated point by point in FP64, a half warp per pair: 21 FP64
// instructions a pair against 17 with a pair per lane, but a few near rows do
// not hold up a whole warp.
template <int Q1>
__global__ void __launch_bounds__(kFarThreads, 2)
    k_tile_far(int N, int n_tiles, const double* __restrict__ X, const double* __restrict__ scale,
               const int* __restrict__ dnset, const int* __restrict__ tile_ptr,
               const int2* __restrict__ tile_ent, const int4* __restrict__ cell_dofs,
               const FarRecord<Q1>* __restrict__ far, const double* __restrict__ rec,
               double* __restrict__ Nm, double* __restrict__ Dm, DevErr* err,
               const __grid_constant__ PanelRule c_q, const __grid_constant__ FarTables c_far) {
  using Rec = FarRecord<Q1>;
  constexpr int NQ = Q1 * Q1;
  constexpr int RT = kRowsF64, CT = kColsPerTileF64, LDA = RT + 1;
  static_assert(kFarChunk % kFarRowThreads == 0 && sizeof(Rec) % 16 == 0, "chunk layout");
  extern __shared__ __align__(128) unsigned char smem[];
  Rec* stage = reinterpret_cast<Rec*>(smem);  // [2][kFarChunk]
  double* accN = reinterpret_cast<double*>(stage + 2 * kFarChunk);  // [CT][LDA]
  double* accD = accN + CT * LDA;
  ChunkMeta* meta = reinterpret_cast<ChunkMeta*>(accD + CT * LDA);
  uint64_t* bar = reinterpret_cast<uint64_t*>(meta + 2 * kFarChunk);

  const int tid = threadIdx.x, lane = tid & 31;
  const int rt = tid / kFarRowThreads, part = tid % kFarRowThreads;
  const int tile = blockIdx.x % n_tiles;
  const int col0 = tile_ptr[n_tiles + 1 + tile], ncol = tile_ptr[n_tiles + 2 + tile] - col0;
  // the rows around the tile's own first (0, 1, -1, 2, ... from it): their
  // near pairs make a CTA up to six times as long, which at the end of the
  // launch would leave the other SMs idle
  const int n_rt = (N + RT - 1) / RT, kth = blockIdx.x / n_tiles;
  const int row0 = (col0 / RT + n_rt + ((kth & 1) ? (kth + 1) / 2 : -(kth / 2))) % n_rt * RT;
  const int row = row0 + rt;
  const bool active = row < N;
  double xi = 0, yi = 0, zi = 0;
  int set[kMaxSet];
#pragma unroll
  for (int k = 0; k < kMaxSet; ++k) set[k] = -2;
  const double S = scale[0], inv_S = scale[1];
  if (active) {
    xi = X[3 * (size_t)row] * S;
    yi = X[3 * (size_t)row + 1] * S;
    zi = X[3 * (size_t)row + 2] * S;
#pragma unroll
    for (int k = 0; k < kMaxSet; ++k) set[k] = dnset[(size_t)row * kMaxSet + k];
  }
  for (int k = tid; k < CT * LDA; k += kFarThreads) {
    accN[k] = 0.0;
    accD[k] = 0.0;
  }
  const int e0 = tile_ptr[tile], e1 = tile_ptr[tile + 1];
  const int nch = (e1 - e0 + kFarChunk - 1) / kFarChunk;
  auto load_meta = [&](int c) {
    const int k = tid - 32;
    const int base = e0 + c * kFarChunk;
    if (k >= 0 && k < kFarChunk && base + k < e1) {
      const int2 ent = tile_ent[base + k];
      ChunkMeta m;
      m.cell = ent.x & 0x7fffffff;
      m.slots = (uint32_t)ent.y;
      m.owner = ent.x < 0;
      // does it share a column with an earlier panel of its group?
      m.pad = 0;
      for (int j = k % kFarRowThreads; j > 0; --j) {
        const uint32_t mine = m.slots, other = (uint32_t)tile_ent[base + k - j].y;
        const uint32_t in = ~__vcmpeq4(mine, 0xffffffffu);
        m.pad |= ((__vcmpeq4(mine, other) | __vcmpeq4(mine, __byte_perm(other, 0, 0x0321)) |
                   __vcmpeq4(mine, __byte_perm(other, 0, 0x1032)) |
                   __vcmpeq4(mine, __byte_perm(other, 0, 0x2103))) & in) != 0;
      }
      m.dofs = cell_dofs[m.cell];
      m.geo = make_float4(0.f, 0.f, 0.f, 0.f);
      meta[(c & 1) * kFarChunk + k] = m;
    }
  };
  if (nch > 0) load_meta(0);
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();

  auto issue = [&](int c) {
    const int sidx = c & 1;
    const int base = e0 + c * kFarChunk;
    const int cnt = min(kFarChunk, e1 - base);
    mbar_arrive_expect_tx(&bar[sidx], (uint32_t)(cnt * sizeof(Rec)));
    for (int k = 0; k < cnt; ++k)
      bulk_g2s(stage + sidx * kFarChunk + k, far + (tile_ent[base + k].x & 0x7fffffff),
               (uint32_t)sizeof(Rec), &bar[sidx]);
  };
  if (tid == 0 && nch > 0) issue(0);

  for (int c = 0; c < nch; ++c) {
    if (tid == 0 && c + 1 < nch) {
      fence_proxy_async_smem();
      issue(c + 1);
    }
    if (c + 1 < nch) load_meta(c + 1);
    const bool ok = mbar_wait_bounded(&bar[c & 1], (uint32_t)((c >> 1) & 1));
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        dev_fail(err, WBEM_ERR_TIMEOUT, 11, tile, c);
        if (c + 1 < nch) mbar_wait_bounded(&bar[(c + 1) & 1], (uint32_t)(((c + 1) >> 1) & 1));
      }
      return;
    }
    const int cnt = min(kFarChunk, e1 - (e0 + c * kFarChunk));
    for (int k0 = 0; k0 < cnt; k0 += kFarRowThreads) {
      const int k = k0 + part;
      bool use = active && k < cnt;
      const int kk = (c & 1) * kFarChunk + min(k, cnt - 1);
      const ChunkMeta& mt = meta[kk];
      const Rec& r = stage[kk];
      const uint32_t slots = mt.slots;
      const int4 d = mt.dofs;
      use = use && !(in_set(set, d.x) || in_set(set, d.y) || in_set(set, d.z) || in_set(set, d.w));
      const double Rx = r.c[0] - xi, Ry = r.c[1] - yi, Rz = r.c[2] - zi;
      const double p = fma(Rx, Rx, fma(Ry, Ry, Rz * Rz));
      const float p1 = cut_to_float(p);
      const bool isfar = use && p1 > r.thr && p1 < 0x1p+30f;
      double ln[4], ld[4];
      // one form per warp: both, one after the other, would cost their sum
      const bool second = __any_sync(0xffffffffu, isfar && !(p1 > r.thr1));
      if (isfar) {
        if (second) far_pair<Q1, true>(r, Rx, Ry, Rz, p, p1, c_far, ln, ld);
        else far_pair<Q1, false>(r, Rx, Ry, Rz, p, p1, c_far, ln, ld);
      }
      // the row's four panels mostly share no column (the tile's list is in
      // that order): then all add at once
      const bool clash = __any_sync(0xffffffffu, mt.pad != 0);
#pragma unroll 1
      for (int ph = 0; ph < (clash ? kFarRowThreads : 1); ++ph) {
        if (isfar && (!clash || part == ph)) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t sl = (slots >> (8 * j)) & 255u;
            if (sl != 255u) {
              accN[sl * LDA + rt] += ln[j];
              accD[sl * LDA + rt] += ld[j];
            }
          }
        }
        __syncwarp();
      }
      // the other pairs, two at a time
      unsigned todo = __ballot_sync(0xffffffffu, use && !isfar);
      while (todo) {
        const int l0 = __ffs(todo) - 1;
        todo &= todo - 1;
        const int l1 = todo ? __ffs(todo) - 1 : -1;
        if (todo) todo &= todo - 1;
        const int src = lane < 16 ? l0 : l1;
        const int rs = (tid & ~31) / kFarRowThreads + max(src, 0) / kFarRowThreads;
        const ChunkMeta& ms = meta[(c & 1) * kFarChunk + k0 + max(src, 0) % kFarRowThreads];
        double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (src >= 0) {
          const double* xr = X + 3 * (size_t)(row0 + rs);
          const double px = xr[0], py = xr[1], pz = xr[2];
          const double* g = rec + (size_t)ms.cell * (NQ * 8);
          for (int q = lane & 15; q < NQ; q += 16) {
            const double2 p01 = *reinterpret_cast<const double2*>(g + q * 8);
            const double2 p23 = *reinterpret_cast<const double2*>(g + q * 8 + 2);
            const double2 p45 = *reinterpret_cast<const double2*>(g + q * 8 + 4);
            const double p6 = g[q * 8 + 6];
            const double qx = p01.x - px, qy = p01.y - py, qz = p23.x - pz;
            const double ri = rsqrt(fma(qx, qx, fma(qy, qy, qz * qz)));
            const double sq = ri * p23.y;
            const double dq = -fma(qx, p45.x, fma(qy, p45.y, qz * p6)) * (ri * ri * ri);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              v[j] = fma(dq, c_q.phi[q][j], v[j]);
              v[4 + j] = fma(sq, c_q.phi[q][j], v[4 + j]);
            }
          }
        }
        double s = panel_reduce8<false>(v, lane);  // component (lane >> 1) & 7
        if (lane & 8) s *= S;                      // D's, a length
        double add[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) add[j] = __shfl_sync(0xffffffffu, s, (lane & 24) + 2 * j);
#pragma unroll
        for (int ph = 0; ph < 2; ++ph) {  // both pairs may be the same row's
          if ((lane >> 4) == ph && (lane & 7) == 0 && src >= 0) {
            double* acc = (lane & 8) ? accD : accN;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t sl = (ms.slots >> (8 * j)) & 255u;
              if (sl != 255u) acc[sl * LDA + rs] += add[j];
            }
          }
          __syncwarp();
        }
      }
    }
    __syncthreads();
  }

  for (int idx = tid; idx < RT * CT; idx += kFarThreads) {
    const int rr = idx / CT, cc = idx % CT;
    const int gr = row0 + rr, gc = col0 + cc;
    if (gr < N && cc < ncol) {
      Nm[(size_t)gr * N + gc] = accN[cc * LDA + rr];
      Dm[(size_t)gr * N + gc] = accD[cc * LDA + rr] * inv_S;
    }
  }
}

template <int Q1>
static cudaError_t launch_tile_fp64_t(int N, const double* X, const int* dnset, int n_tiles,
                                      const int* tile_ptr, const int2* tile_ent,
                                      const int4* cell_dofs, const double* rec, double* Nm,
                                      double* Dm, DevErr* err, const PanelRule& rule,
                                      cudaStream_t s) {
  constexpr int RECD = Q1 * Q1 * 8;
  const size_t smem = (size_t)2 * kChunk * RECD * 8 +
                      (size_t)2 * kColsPerTileF64 * (kRowsF64 + 1) * 8 +
                      2 * kChunk * sizeof(ChunkMeta) + 2 * sizeof(uint64_t);
  cudaError_t e = cudaFuncSetAttribute(k_tile_fp64<Q1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid(n_tiles, (N + kRowsF64 - 1) / kRowsF64);
  k_tile_fp64<Q1><<<grid, kF64Threads, smem, s>>>(N, X, dnset, tile_ptr, tile_ent, cell_dofs, rec,
                                                   Nm, Dm, err, rule);
  return cudaGetLastError();
}

template <int Q1>
static cudaError_t launch_tile_far_t(int N, int C, const double* X, const int* dnset, int n_tiles,
                                     const int* tile_ptr, const int2* tile_ent,
                                     const int4* cell_dofs, const double* rec, void* far,
                                     double* Nm, double* Dm, DevErr* err, const PanelRule& rule,
                                     cudaStream_t s) {
  using Rec = FarRecord<Q1>;
  constexpr int G = Q1 * Q1 <= 16 ? 16 : 32, PB = 128 / G;
  const size_t smem = (size_t)2 * kFarChunk * sizeof(Rec) +
                      (size_t)2 * kColsPerTileF64 * (kRowsF64 + 1) * 8 +
                      2 * kFarChunk * sizeof(ChunkMeta) + 2 * sizeof(uint64_t);
  cudaError_t e = cudaFuncSetAttribute(k_tile_far<Q1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  double* scale = static_cast<double*>(far);
  Rec* recs = reinterpret_cast<Rec*>(static_cast<char*>(far) + kFarHeader);
  k_mesh_scale<<<1, 1024, 0, s>>>(3 * N, X, scale);
  k_far_records<Q1><<<(C + PB - 1) / PB, 128, 0, s>>>(C, X, cell_dofs, scale, recs, rule);
  const unsigned grid = (unsigned)n_tiles * ((N + kRowsF64 - 1) / kRowsF64);
  k_tile_far<Q1><<<grid, kFarThreads, smem, s>>>(N, n_tiles, X, scale, dnset, tile_ptr, tile_ent, cell_dofs,
                                                 recs, rec, Nm, Dm, err, rule, far_tables(rule));
  return cudaGetLastError();
}

// Rules of three and more points per direction take k_tile_far. At one and two
// points a pair has few enough that k_tile_fp64 stays: sphere of 5,402 dofs,
// k_tile_fp64 against k_tile_far, ms: two points 9.6 / 9.8, three 20.9 / 10.0,
// four 32.1 / 9.6, five 51.2 / 11.7, six 70.0 / 14.8.
size_t far_bytes(int q1, int C) {
  switch (q1) {
    case 3: return kFarHeader + sizeof(FarRecord<3>) * C;
    case 4: return kFarHeader + sizeof(FarRecord<4>) * C;
    case 5: return kFarHeader + sizeof(FarRecord<5>) * C;
    case 6: return kFarHeader + sizeof(FarRecord<6>) * C;
    default: return 0;
  }
}

cudaError_t launch_tile_fp64(int N, int C, const PanelRule& rule, const double* X, const int* dnset, int n_tiles,
                             const int* tile_ptr, const int2* tile_ent, const int4* cell_dofs,
                             const double* rec, void* far, double* Nm, double* Dm, DevErr* err,
                             cudaStream_t s) {
  switch (rule.q1) {
    case 1: return launch_tile_fp64_t<1>(N, X, dnset, n_tiles, tile_ptr, tile_ent, cell_dofs, rec, Nm, Dm, err, rule, s);
    case 2: return launch_tile_fp64_t<2>(N, X, dnset, n_tiles, tile_ptr, tile_ent, cell_dofs, rec, Nm, Dm, err, rule, s);
    case 3: return launch_tile_far_t<3>(N, C, X, dnset, n_tiles, tile_ptr, tile_ent, cell_dofs, rec, far, Nm, Dm, err, rule, s);
    case 4: return launch_tile_far_t<4>(N, C, X, dnset, n_tiles, tile_ptr, tile_ent, cell_dofs, rec, far, Nm, Dm, err, rule, s);
    case 5: return launch_tile_far_t<5>(N, C, X, dnset, n_tiles, tile_ptr, tile_ent, cell_dofs, rec, far, Nm, Dm, err, rule, s);
    case 6: return launch_tile_far_t<6>(N, C, X, dnset, n_tiles, tile_ptr, tile_ent, cell_dofs, rec, far, Nm, Dm, err, rule, s);
    default: return cudaErrorInvalidValue;
  }
}

// Vertex-singular panels: for row i, every panel holding a node of its
// double-node set; the singular vertex is the first local vertex in the set
// (source/bem_problem.cc:223-230), the rule is the polar vertex rule for that
// vertex (:478-522). One CTA per row: its four warps take every fourth panel
// with the rule's points over the lanes, then eight threads add the entries
// (panels share vertices) in ascending panel order. Bound by the latency of
// one panel's FP64 chain, not by throughput, at the sizes of the plain form:
// one thread per row (panel after panel, 50 points each) took 0.57 ms at any
// N up to 16,000; this takes 0.078 ms at N = 2,000.
constexpr int kSingWarps = 4, kSingBatch = 32;  // panels whose sums are held at a time

__global__ void __launch_bounds__(kSingWarps * 32)
    k_singular_fp64(int N, const double* __restrict__ X, const int* __restrict__ dnset,
                    const int* __restrict__ sptr, const int* __restrict__ scell,
                    const int4* __restrict__ cell_dofs, const QuadTables* __restrict__ qt,
                    double* __restrict__ Nm, double* __restrict__ Dm, DevErr* err) {
  __shared__ double sums[kSingBatch][8];
  __shared__ int ids[kSingBatch][4];
  const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double x[3] = {X[3 * (size_t)row], X[3 * (size_t)row + 1], X[3 * (size_t)row + 2]};
  int set[kMaxSet];
#pragma unroll
  for (int k = 0; k < kMaxSet; ++k) set[k] = dnset[(size_t)row * kMaxSet + k];
  const int e1 = sptr[row + 1];
  for (int e0 = sptr[row]; e0 < e1; e0 += kSingBatch) {
    const int n = min(kSingBatch, e1 - e0);
    for (int e = warp; e < n; e += kSingWarps) {
      const int4 d = cell_dofs[scell[e0 + e]];
      const int id[4] = {d.x, d.y, d.z, d.w};
      int v = -1;
#pragma unroll
      for (int j = 3; j >= 0; --j)
        if (in_set(set, id[j])) v = j;
      double val = 0.0;
      if (v < 0) {
        if (lane == 0) dev_fail(err, WBEM_ERR_ARG, 21, row, scell[e0 + e]);
      } else {
        double P[4][3];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int c = 0; c < 3; ++c) P[k][c] = X[3 * (size_t)id[k] + c];
        val = singular_panel(P, x, qt->sp[v], qt->nsp, lane);
      }
      if ((lane & 17) == 0) sums[e][(lane >> 1) & 7] = val;
      if (lane < 4) ids[e][lane] = id[lane];
    }
    __syncthreads();
    if (tid < 8) {
      double* M = (tid < 4 ? Nm : Dm) + (size_t)row * N;
      for (int e = 0; e < n; ++e) {
        M[ids[e][tid & 3]] += sums[e][tid];
        __syncwarp(0xffu);  // the next panel's shared vertex may be another thread's
      }
    }
    __syncthreads();
  }
}

cudaError_t launch_singular_fp64(int N, const double* X, const int* dnset, const int* sptr,
                                 const int* scell, const int4* cell_dofs, const QuadTables* qt,
                                 double* Nm, double* Dm, DevErr* err, cudaStream_t s) {
  k_singular_fp64<<<N, kSingWarps * 32, 0, s>>>(N, X, dnset, sptr, scell, cell_dofs, qt, Nm, Dm, err);
  return cudaGetLastError();
}

// alpha_i = - sum_j N_ij (one warp per row, FP64).
__global__ void k_alpha_rowsum(int N, const double* __restrict__ Nm, double* __restrict__ alpha) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= N) return;
  const double* r = Nm + (size_t)warp * N;
  double s = 0;
  for (int j = lane; j < N; j += 32) s += r[j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) alpha[warp] = -s;
}

cudaError_t launch_alpha_rowsum(int N, const double* Nm, double* alpha, cudaStream_t s) {
  const int bs = 256;
  k_alpha_rowsum<<<(unsigned)(((size_t)N * 32 + bs - 1) / bs), bs, 0, s>>>(N, Nm, alpha);
  return cudaGetLastError();
}

}  // namespace wbem
