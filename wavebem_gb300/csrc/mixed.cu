// Mixed-precision assembly of N (dG/dn) and D (G).
//
// Regular panels far from the collocation point are integrated with the same
// Gauss rule as the reference (source/bem_problem.cc:241-260), but evaluated as
//     k(x_q - x_i) = k(c - x_i) + [k(x_q - x_i) - k(c - x_i)]
// with c the panel centre: the panel term k(c - x_i) (and its contraction with
// the exact panel moments sum_q phi_j(q) JxW_q) is computed once per
// (row, panel) pair in double-float arithmetic on FP32 units, and the
// per-quadrature-point differences are computed in FP32 from cancellation-free
// forms (1/a - 1/b = (b^2 - a^2) / (a b (a + b)) etc.). The FP32 rounding
// then only touches the O(h/r) difference terms, which keeps entries accurate
// to about 1e-9 relative instead of the 1e-7 of plain FP32 evaluation.
// Panels within `ratio` diameters of the collocation point and the singular
// panels are integrated in FP64 (k_near_mixed, k_singular_mixed).
// Entries are stored as (hi, lo) float pairs; alpha = -sum_j N_ij is
// accumulated in FP64 from the three parts.
#include <cuda_runtime.h>
#include <stdint.h>
#include "context.h"
#include "host_util.h"
#include "packed.cuh"
#include "kernels.h"
#include "panel_fp64.cuh"

namespace wbem {

constexpr double kInv4PiM = 0.07957747154594766788;

// Panel record: 20 floats per pair of points (2 p, 2 p + 1), the nine values of
// the two points side by side: offset from the centre (3), minus its square,
// minus the normal's difference from nu (3), minus offset . normal, J weight /
// (4 pi); then 24 floats of panel data.
constexpr int kPairFloats = 20;
__host__ __device__ constexpr int mixed_rec_panel(int nq) { return (nq + 1) / 2 * kPairFloats; }
__host__ __device__ constexpr int mixed_rec_floats(int nq) { return mixed_rec_panel(nq) + 24; }

// Same near test in every kernel (no contraction: explicit round-to-nearest ops).
__device__ __forceinline__ bool near_test(float xi, float yi, float zi, float4 g) {
  const float dx = __fsub_rn(g.x, xi), dy = __fsub_rn(g.y, yi), dz = __fsub_rn(g.z, zi);
  const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
  return d2 < g.w;
}

__device__ __forceinline__ bool in_set_m(const int set[kMaxSet], int v) {
  bool r = false;
#pragma unroll
  for (int k = 0; k < kMaxSet; ++k) r |= (set[k] == v);
  return r;
}

__device__ __forceinline__ void q1_geo(const double P[4][3], double s, double t, double x[3],
                                       double cr[3]) {
  const double a0 = (1 - s) * (1 - t), a1 = s * (1 - t), a2 = (1 - s) * t, a3 = s * t;
  double jx[3], je[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    x[d] = a0 * P[0][d] + a1 * P[1][d] + a2 * P[2][d] + a3 * P[3][d];
    jx[d] = (1 - t) * (P[1][d] - P[0][d]) + t * (P[3][d] - P[2][d]);
    je[d] = (1 - s) * (P[2][d] - P[0][d]) + s * (P[3][d] - P[1][d]);
  }
  cr[0] = jx[1] * je[2] - jx[2] * je[1];
  cr[1] = jx[2] * je[0] - jx[0] * je[2];
  cr[2] = jx[0] * je[1] - jx[1] * je[0];
}

// Outputs of the mixed assembly. The entries are stored with the column's
// boundary condition already applied (sel_j = 1: Dirichlet column):
//   A2_ij = sel_j ? -D_ij : N_ij   (system operator, as vmult applies it)
//   B2_ij = sel_j ? -N_ij : D_ij   (right-hand-side operator, compute_rhs)
// as (hi, lo) float pairs, so that each mat-vec streams one matrix. Optional
// FP32 copy S_ij = hi(A2_ij) (row-major, leading dimension ld); the diagonal
// free term and the constraint rows are added at solve time.
struct SysOut {
  float* S;                  // nullptr: not written
  int ld;
  const uint8_t* sel;        // column selection of A2 / B2
};

// FP64 geometry -> mixed record + near-test data, a quadrature point per lane;
// the panel sums (normal and moments) run over the points in ascending order
// on seven lanes. HALF: two panels per warp (rules of at most 16 points).
// Latency-bound at small N and FP64-bound at large: a thread per panel took
// 0.128 ms at N = 600 as at N = 12,000, now 0.012 and 0.092 ms (a
// whole warp per 16-point panel left half the FP64 lanes idle: 0.267 ms).
constexpr int kRecWarps = 4;
constexpr int kRecPoints = 36;  // most points of the mixed form's rule (order 6)

template <bool HALF>
__global__ void __launch_bounds__(kRecWarps * 32)
    k_cell_records_mixed(int C, const double* __restrict__ X, const int4* __restrict__ cell_dofs,
                         float* __restrict__ rec, float4* __restrict__ cellgeo, float ratio,
                         const __grid_constant__ PanelRule c_q) {
  constexpr int W = HALF ? 16 : 32, kPts = HALF ? 16 : kRecPoints;
  // per panel and point: offset from the centre, cross product, its norm
  __shared__ double s_pt[kRecWarps * (32 / W)][7][kPts];
  const int slot = threadIdx.x / W, lane = threadIdx.x & (W - 1);
  const int c0 = blockIdx.x * (kRecWarps * 32 / W) + slot;
  const int c = min(c0, C - 1);  // past the last panel: its work again, not written
  double(*pt)[kPts] = s_pt[slot];
  const int nq = c_q.q1 * c_q.q1;
  const int RF = mixed_rec_floats(nq);
  const int4 d = cell_dofs[c];
  const int id[4] = {d.x, d.y, d.z, d.w};
  double P[4][3];
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int e = 0; e < 3; ++e) P[k][e] = X[3 * (size_t)id[k] + e];
  double cen[3];
#pragma unroll
  for (int e = 0; e < 3; ++e) cen[e] = 0.25 * (P[0][e] + P[1][e] + P[2][e] + P[3][e]);
  for (int q = lane; q < nq; q += W) {
    double x[3], cr[3];
    q1_geo(P, c_q.gp[q][0], c_q.gp[q][1], x, cr);
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      pt[e][q] = x[e] - cen[e];
      pt[3 + e][q] = cr[e];
    }
    pt[6][q] = sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
  }
  __syncwarp();
  // lanes 0..2: normal; lanes 3..6: moments
  double sum = 0.0;
  if (lane < 7) {
    const double* a = lane < 3 ? pt[3 + lane] : pt[6];
    for (int q = 0; q < nq; ++q) {
      const double w = c_q.gp[q][2];
      sum += lane < 3 ? a[q] * w : c_q.phi[q][max(lane - 3, 0)] * (a[q] * w * kInv4PiM);
    }
  }
  double nu[3], M[4];
#pragma unroll
  for (int e = 0; e < 3; ++e) nu[e] = __shfl_sync(0xffffffffu, sum, e, W);
#pragma unroll
  for (int j = 0; j < 4; ++j) M[j] = __shfl_sync(0xffffffffu, sum, 3 + j, W);
  const bool on = c0 < C;
  const double nl = 1.0 / sqrt(nu[0] * nu[0] + nu[1] * nu[1] + nu[2] * nu[2]);
#pragma unroll
  for (int e = 0; e < 3; ++e) nu[e] *= nl;
  float* r = rec + (size_t)c * RF;
  for (int q = lane; on && q < nq; q += W) {
    const double det = pt[6][q], rdet = 1.0 / det;
    double del[3], n[3];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      del[e] = pt[e][q];
      n[e] = pt[3 + e][q] * rdet;
    }
    const float v[10] = {(float)del[0],
                         (float)del[1],
                         (float)del[2],
                         -(float)(del[0] * del[0] + del[1] * del[1] + del[2] * del[2]),
                         -(float)(n[0] - nu[0]),
                         -(float)(n[1] - nu[1]),
                         -(float)(n[2] - nu[2]),
                         -(float)(del[0] * n[0] + del[1] * n[1] + del[2] * n[2]),
                         (float)(det * c_q.gp[q][2] * kInv4PiM),
                         0.f};
    float* rp = r + (q >> 1) * kPairFloats + (q & 1);
#pragma unroll
    for (int e = 0; e < 10; ++e) {
      rp[2 * e] = v[e];
      if (q == nq - 1 && !(q & 1)) rp[2 * e + 1] = v[e];  // a last point alone: paired with itself
    }
  }
  // panel data: lane e splits one of centre, normal, moments, moment sum
  float* cd = r + mixed_rec_panel(nq);
  if (on && lane < 11) {
    const double v = lane < 3   ? (lane == 0 ? cen[0] : lane == 1 ? cen[1] : cen[2])
                     : lane < 6 ? (lane == 3 ? nu[0] : lane == 4 ? nu[1] : nu[2])
                     : lane < 8 ? (lane == 6 ? M[0] : M[1])
                     : lane < 10 ? (lane == 8 ? M[2] : M[3])
                                 : ((M[0] + M[1]) + M[2]) + M[3];
    const df a = df_from_double(v);
    // hi at 0..2, 6..8, 12..15, 20; lo at 3..5, 9..11, 16..19, 21
    const int hi = lane < 3 ? lane : lane < 6 ? 3 + lane : lane < 10 ? 6 + lane : 20;
    const int lo = lane < 6 ? 3 + hi : lane < 10 ? 4 + hi : 21;
    cd[hi] = a.hi;
    cd[lo] = a.lo;
  } else if (on && lane == 11) {
    cd[22] = 0.f;
    cd[23] = 0.f;
  }
  // near test: centre (float) and (ratio * largest diagonal)^2, at least
  // 1.01 x the farthest vertex, so that every panel with the collocation
  // point (or a double-node partner of it) as a vertex tests near: the
  // regular far-field kernel then needs no singular test of its own.
  // Lanes 0, 1: squared diagonals; lanes 2..5: squared vertex distances.
  double d2 = 0.0;
  if (lane < 6) {
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const double a = lane == 0   ? P[3][e]
                       : lane == 1 ? P[2][e]
                       : lane == 2 ? P[0][e]
                       : lane == 3 ? P[1][e]
                       : lane == 4 ? P[2][e]
                                   : P[3][e];
      const double b = lane == 0 ? P[0][e] : lane == 1 ? P[1][e] : cen[e];
      d2 += (a - b) * (a - b);
    }
  }
  const double diag = fmax(__shfl_sync(0xffffffffu, d2, 0, W), __shfl_sync(0xffffffffu, d2, 1, W));
  const double vert = fmax(fmax(__shfl_sync(0xffffffffu, d2, 2, W), __shfl_sync(0xffffffffu, d2, 3, W)),
                           fmax(__shfl_sync(0xffffffffu, d2, 4, W), __shfl_sync(0xffffffffu, d2, 5, W)));
  if (on && lane == 0) {
    const double rad = fmax((double)ratio * sqrt(diag), 1.01 * sqrt(vert));
    cellgeo[c] = make_float4((float)cen[0], (float)cen[1], (float)cen[2], (float)(rad * rad));
  }
}

constexpr int kChunkM = 8;

// The approximate root and quotient without the steps for subnormal operands:
// the same values (1 / r^3 overflows long before r^2 is subnormal).
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float div_ftz(float x, float y) {
  float r;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
  return r;
}

template <int Q1>
__global__ void __launch_bounds__(kRowsPerTile)
    k_tile_mixed(int N, const double* __restrict__ X, const int* __restrict__ dnset,
                 const int* __restrict__ tile_ptr, const int2* __restrict__ tile_ent,
                 const int4* __restrict__ cell_dofs, const float* __restrict__ rec,
                 const float4* __restrict__ cellgeo, float2* __restrict__ A2,
                 float2* __restrict__ B2, double* __restrict__ alpha_part, SysOut so,
                 DevErr* err, const __grid_constant__ PanelRule c_q) {
  constexpr int NQ = Q1 * Q1;
  constexpr int RF = mixed_rec_floats(NQ);
  constexpr int RT = kRowsPerTile, CT = kColsPerTile, LDA = RT + 1;
  extern __shared__ __align__(128) unsigned char smem[];
  float* stage = reinterpret_cast<float*>(smem);  // [2][kChunkM][RF]
  float* aNh = stage + 2 * kChunkM * RF;          // [CT][LDA] x 4
  float* aNl = aNh + CT * LDA;
  float* aDh = aNl + CT * LDA;
  float* aDl = aDh + CT * LDA;
  ChunkMeta* meta = reinterpret_cast<ChunkMeta*>(aDl + CT * LDA + ((4 - ((CT * LDA) & 3)) & 3));
  uint64_t* bar = reinterpret_cast<uint64_t*>(meta + 2 * kChunkM);

  const int tid = threadIdx.x;
  const int tile = blockIdx.x;
  const int row0 = blockIdx.y * RT;
  const int row = row0 + tid;
  const bool active = row < N;
  df xr[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  if (active) {
#pragma unroll
    for (int d = 0; d < 3; ++d) xr[d] = df_from_double(X[3 * (size_t)row + d]);
  }
  const float xf = active ? __double2float_rn(X[3 * (size_t)row]) : 0.f;
  const float yf = active ? __double2float_rn(X[3 * (size_t)row + 1]) : 0.f;
  const float zf = active ? __double2float_rn(X[3 * (size_t)row + 2]) : 0.f;
  for (int k = tid; k < CT * LDA; k += RT) {
    aNh[k] = 0.f;
    aNl[k] = 0.f;
    aDh[k] = 0.f;
    aDl[k] = 0.f;
  }
  const int e0 = tile_ptr[tile], e1 = tile_ptr[tile + 1];
  const int nch = (e1 - e0 + kChunkM - 1) / kChunkM;
  // metadata of chunk c into meta[c & 1] (threads 32 .. 32 + kChunkM - 1)
  auto load_meta = [&](int c) {
    const int k = tid - 32;
    const int base = e0 + c * kChunkM;
    if (k >= 0 && k < kChunkM && base + k < e1) {
      const int2 ent = tile_ent[base + k];
      ChunkMeta m;
      m.cell = ent.x & 0x7fffffff;
      m.slots = (uint32_t)ent.y;
      m.owner = ent.x < 0;
      m.pad = 0;
      m.dofs = cell_dofs[m.cell];
      m.geo = cellgeo[m.cell];
      meta[(c & 1) * kChunkM + k] = m;
    }
  };
  if (nch > 0) load_meta(0);
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  df alpha_acc = {0.f, 0.f};

  auto issue = [&](int c) {
    const int sidx = c & 1;
    const int base = e0 + c * kChunkM;
    const int cnt = min(kChunkM, e1 - base);
    mbar_arrive_expect_tx(&bar[sidx], (uint32_t)(cnt * RF * 4));
    for (int k = 0; k < cnt; ++k) {
      const int cell = tile_ent[base + k].x & 0x7fffffff;
      bulk_g2s(stage + (size_t)(sidx * kChunkM + k) * RF, rec + (size_t)cell * RF,
               (uint32_t)(RF * 4), &bar[sidx]);
    }
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
        dev_fail(err, WBEM_ERR_TIMEOUT, 41, tile, c);
        if (c + 1 < nch) mbar_wait_bounded(&bar[(c + 1) & 1], (uint32_t)(((c + 1) >> 1) & 1));
      }
      return;
    }
    const int base = e0 + c * kChunkM;
    const int cnt = min(kChunkM, e1 - base);
    for (int k = 0; k < cnt; ++k) {
      const ChunkMeta& mt = meta[(c & 1) * kChunkM + k];
      const bool owner = mt.owner != 0;
      const uint32_t slots = mt.slots;
      // near (FP64 kernel) or singular (always near, see the cell records)
      if (!active || near_test(xf, yf, zf, mt.geo)) continue;
      const float* r = stage + (size_t)((c & 1) * kChunkM + k) * RF;
      const float* cd = r + mixed_rec_panel(NQ);
      // ---- panel base term in double-float
      df R[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        df s = two_sum(cd[d], -xr[d].hi);
        s.lo += cd[3 + d] - xr[d].lo;
        R[d] = fast_two_sum(s.hi, s.lo);
      }
      df r2 = two_prod(R[0].hi, R[0].hi);
      r2.lo = __fmaf_rn(2.f * R[0].hi, R[0].lo, r2.lo);
#pragma unroll
      for (int d = 1; d < 3; ++d) {
        df p = two_prod(R[d].hi, R[d].hi);
        p.lo = __fmaf_rn(2.f * R[d].hi, R[d].lo, p.lo);
        r2 = df_add_fast(r2, p);
      }
      const float y0 = rsqrtf(r2.hi);
      const df t = df_mul(r2, two_prod(y0, y0));
      const float ecor = (1.0f - t.hi) - t.lo;
      const df rinv = fast_two_sum(y0, 0.5f * y0 * ecor);
      const df ri3 = df_mul(df_mul(rinv, rinv), rinv);
      // R . nu in double-float: exact hi products, cross terms into the lo part
      df Rn;
      {
        const df p0 = two_prod(R[0].hi, cd[6]);
        const df p1 = two_prod(R[1].hi, cd[7]);
        const df p2 = two_prod(R[2].hi, cd[8]);
        df s01 = two_sum(p0.hi, p1.hi);
        df s = two_sum(s01.hi, p2.hi);
        float lo = s01.lo + s.lo + (p0.lo + p1.lo + p2.lo);
        lo = __fmaf_rn(R[0].hi, cd[9], __fmaf_rn(R[0].lo, cd[6], lo));
        lo = __fmaf_rn(R[1].hi, cd[10], __fmaf_rn(R[1].lo, cd[7], lo));
        lo = __fmaf_rn(R[2].hi, cd[11], __fmaf_rn(R[2].lo, cd[8], lo));
        Rn = fast_two_sum(s.hi, lo);
      }
      df gR = df_mul(Rn, ri3);
      gR.hi = -gR.hi;
      gR.lo = -gR.lo;
      // ---- per-point differences in FP32, two points per packed instruction: the
      // kernel is bound by issue slots (84% busy at 62% of the FP32 pipe with
      // scalar ones; 6.08 -> 5.23 ms at 12,000 dofs, the same bits)
      // with num = rc^2 - rq^2 = -(2 R_c.delta + |delta|^2):
      //   rc - rq = num / (rc + rq),  1/rq - 1/rc = (rc - rq) / (rq rc),
      //   (R.n)(-1/r^3) - (R_c.nu)(-1/rc^3)
      //     = rq^-3 [ (rc - rq)(rc^2 + rc rq + rq^2) (-(R_c.nu) / rc^3) - (R_c.(n - nu) + delta.n) ]
      const float Rcx = R[0].hi, Rcy = R[1].hi, Rcz = R[2].hi;
      const float rcinv = rinv.hi;
      const float rc2 = r2.hi;
      const float rc = rc2 * rcinv;
      const float K1 = -Rn.hi * ri3.hi;
      float ls0 = 0.f, ls1 = 0.f, ls2 = 0.f, ls3 = 0.f, ln0 = 0.f, ln1 = 0.f, ln2 = 0.f, ln3 = 0.f;
      const unsigned long long RX = pk2(Rcx, Rcx), RY = pk2(Rcy, Rcy), RZ = pk2(Rcz, Rcz);
      const unsigned long long rc_2 = pk2(rc, rc), rc2_2 = pk2(rc2, rc2), K1_2 = pk2(K1, K1);
      const unsigned long long m1 = pk2(-1.f, -1.f), m2 = pk2(-2.f, -2.f);
      // tensor-product accumulation: row sums over xi, then the two eta weights
      float st = 0.f, s1 = 0.f, nt = 0.f, n1 = 0.f;
#pragma unroll
      for (int p = 0; p < (NQ + 1) / 2; ++p) {
        const ulonglong2* g = reinterpret_cast<const ulonglong2*>(r + p * kPairFloats);
        const ulonglong2 g0 = g[0], g1 = g[1], g2 = g[2], g3 = g[3];
        const unsigned long long J = *reinterpret_cast<const unsigned long long*>(g + 4);
        const unsigned long long Rd = fma2(RX, g0.x, fma2(RY, g0.y, mul2(RZ, g1.x)));
        const unsigned long long num = fma2(m2, Rd, g1.y);
        const unsigned long long rq2 = fma2(num, m1, rc2_2);
        float a0, a1, b0, b1;
        upk2(rq2, a0, a1);
        const unsigned long long rqinv = pk2(rsqrt_ftz(a0), rsqrt_ftz(a1));
        const unsigned long long rq = mul2(rq2, rqinv);
        upk2(num, a0, a1);
        upk2(add2(rc_2, rq), b0, b1);
        const unsigned long long dr = pk2(div_ftz(a0, b0), div_ftz(a1, b1));
        const unsigned long long u = mul2(rqinv, J);
        const unsigned long long fs2 = mul2(dr, u);  // times 1/rc after the point sums
        const unsigned long long tsum = add2(fma2(rc_2, rq, rc2_2), rq2);
        const unsigned long long t2 = fma2(RX, g2.x, fma2(RY, g2.y, fma2(RZ, g3.x, g3.y)));
        const unsigned long long fn2 =
            mul2(mul2(mul2(rqinv, rqinv), u), fma2(mul2(dr, tsum), K1_2, t2));
        float fs[2], fn[2];
        upk2(fs2, fs[0], fs[1]);
        upk2(fn2, fn[0], fn[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int q = 2 * p + h;
          if (q >= NQ) break;
          const float xa = c_q.gpf[q][0];
          st = __fadd_rn(st, fs[h]);
          s1 = __fmaf_rn(fs[h], xa, s1);
          nt = __fadd_rn(nt, fn[h]);
          n1 = __fmaf_rn(fn[h], xa, n1);
          if ((q + 1) % Q1) continue;
          const float eb = c_q.gpf[q][1];
          const float s0 = st - s1, n0 = nt - n1;
          ls0 = __fmaf_rn(s0, 1.f - eb, ls0);
          ls1 = __fmaf_rn(s1, 1.f - eb, ls1);
          ls2 = __fmaf_rn(s0, eb, ls2);
          ls3 = __fmaf_rn(s1, eb, ls3);
          ln0 = __fmaf_rn(n0, 1.f - eb, ln0);
          ln1 = __fmaf_rn(n1, 1.f - eb, ln1);
          ln2 = __fmaf_rn(n0, eb, ln2);
          ln3 = __fmaf_rn(n1, eb, ln3);
          st = s1 = nt = n1 = 0.f;
        }
      }
      const float fnsum = (ln0 + ln1) + (ln2 + ln3);
      const float lsv[4] = {ls0 * rcinv, ls1 * rcinv, ls2 * rcinv, ls3 * rcinv};
      const float lnv[4] = {ln0, ln1, ln2, ln3};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t sl = (slots >> (8 * j)) & 255u;
        if (sl != 255u) {
          // acc += k(c) M_j + (FP32 point sum): exact hi product, one
          // two_sum into the accumulator, everything else into its lo part
          // (the pair is renormalised once, when it is written out)
          const float Mh = cd[12 + j], Ml = cd[16 + j];
          const int o = sl * LDA + tid;
          {
            const df p = two_prod(gR.hi, Mh);
            const float pl = __fmaf_rn(gR.hi, Ml, __fmaf_rn(gR.lo, Mh, p.lo));
            const df s2 = two_sum(aNh[o], p.hi);
            aNh[o] = s2.hi;
            aNl[o] = aNl[o] + (s2.lo + (pl + lnv[j]));
          }
          {
            const df p = two_prod(rinv.hi, Mh);
            const float pl = __fmaf_rn(rinv.hi, Ml, __fmaf_rn(rinv.lo, Mh, p.lo));
            const df s2 = two_sum(aDh[o], p.hi);
            aDh[o] = s2.hi;
            aDl[o] = aDl[o] + (s2.lo + (pl + lsv[j]));
          }
        }
      }
      if (owner) alpha_acc = df_add(alpha_acc, df_add_f(df_mul(gR, df{cd[20], cd[21]}), fnsum));
    }
    __syncthreads();
  }
  if (active) alpha_part[(size_t)tile * N + row] = df_to_double(alpha_acc);
  // the tile's columns: tile_ptr[gridDim.x + 1 + tile] .. (+ 1)
  const int col0 = tile_ptr[gridDim.x + 1 + tile], ncol = tile_ptr[gridDim.x + 2 + tile] - col0;
  for (int idx = tid; idx < RT * CT; idx += RT) {
    const int rr = idx / CT, cc = idx % CT;
    const int gr = row0 + rr, gc = col0 + cc;
    if (gr < N && cc < ncol) {
      const int o = cc * LDA + rr;
      const bool dj = so.sel[gc] != 0;
      const df en = two_sum(aNh[o], aNl[o]), ed = two_sum(aDh[o], aDl[o]);
      const float2 a = dj ? make_float2(-ed.hi, -ed.lo) : make_float2(en.hi, en.lo);
      const float2 b = dj ? make_float2(-en.hi, -en.lo) : make_float2(ed.hi, ed.lo);
      A2[(size_t)gr * N + gc] = a;
      B2[(size_t)gr * N + gc] = b;
      if (so.S) so.S[(size_t)gr * so.ld + gc] = a.x;
    }
  }
}

template <int Q1>
static cudaError_t launch_tile_mixed_t(int N, const double* X, const int* dnset, int n_tiles,
                                       const int* tile_ptr, const int2* tile_ent,
                                       const int4* cell_dofs, const float* rec,
                                       const float4* cellgeo, float2* A2, float2* B2,
                                       double* alpha_part, SysOut so, DevErr* err,
                                       const PanelRule& rule, cudaStream_t s) {
  constexpr int RF = mixed_rec_floats(Q1 * Q1);
  const size_t acc = (size_t)kColsPerTile * (kRowsPerTile + 1);
  const size_t smem = (size_t)2 * kChunkM * RF * 4 + 4 * acc * 4 + 16 +
                      2 * kChunkM * sizeof(ChunkMeta) + 2 * sizeof(uint64_t);
  cudaError_t e = cudaFuncSetAttribute(k_tile_mixed<Q1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid(n_tiles, (N + kRowsPerTile - 1) / kRowsPerTile);
  k_tile_mixed<Q1><<<grid, kRowsPerTile, smem, s>>>(N, X, dnset, tile_ptr, tile_ent, cell_dofs, rec,
                                                    cellgeo, A2, B2, alpha_part, so, err, rule);
  return cudaGetLastError();
}

// Near-field and singular contributions of a row are appended as items
// (column, dN, dD) in the order the reference adds them, so that the FP64
// kernels run beside the FP32 far-field kernel (they use different pipes)
// and k_merge_items adds them to the (hi, lo) entries afterwards.
constexpr int kNearItems = 1024;  // per row: 4 items per near panel (256 panels)
constexpr int kSingItems = 128;  // per row: 4 items per singular panel
constexpr int kItemCap = kNearItems + kSingItems;

__device__ __forceinline__ void add_entry(float2* A2, float2* B2, SysOut so, int N, int row, int col,
                                          double dn, double dd) {
  const size_t o = (size_t)row * N + col;
  const bool dj = so.sel[col] != 0;
  float2 v = A2[o];
  double s = (double)v.x + (double)v.y + (dj ? -dd : dn);
  float h = __double2float_rn(s);
  A2[o] = make_float2(h, __double2float_rn(s - (double)h));
  if (so.S) so.S[(size_t)row * so.ld + col] = h;
  v = B2[o];
  s = (double)v.x + (double)v.y + (dj ? -dn : dd);
  h = __double2float_rn(s);
  B2[o] = make_float2(h, __double2float_rn(s - (double)h));
}

// Adds a row's items to its entries, one warp per row. Each lane takes an
// item; the lane with the first item of a column sums that column's items in
// ascending order (near items, then singular ones) in FP64 and updates the
// entry once, so the updates of a row run side by side. Latency-bound: one
// thread per row (a read-modify-write after the other, about 140 per row) took
// 0.28 ms from N = 600 to 12,000, now 0.037 and 0.115 ms.
constexpr int kMergeWarps = 4;

__global__ void __launch_bounds__(kMergeWarps * 32)
    k_merge_items(int N, const int* __restrict__ cnt, const int* __restrict__ dof,
                  const double2* __restrict__ val, float2* __restrict__ A2,
                  float2* __restrict__ B2, SysOut so) {
  __shared__ int s_col[kMergeWarps][kItemCap];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * kMergeWarps + warp;
  if (row >= N) return;  // whole warps
  const size_t base = (size_t)row * kItemCap;
  const int nn = min(cnt[2 * row], kNearItems), ns = min(cnt[2 * row + 1], kSingItems);
  const int n = nn + ns;
  int* col = s_col[warp];
  // item k of the row sits at base + k (near) or in the singular part
  for (int k = lane; k < n; k += 32) col[k] = dof[base + (k < nn ? k : kNearItems + k - nn)];
  __syncwarp();
  for (int p0 = 0; p0 < n; p0 += 32) {
    const int k = p0 + lane;
    const int c = k < n ? col[k] : -1;
    bool first = k < n;
    double sn = 0.0, sd = 0.0;
    for (int q0 = 0; q0 < n; q0 += 32) {
      unsigned m = 0;
      const int qn = min(32, n - q0);
      for (int b = 0; b < qn; ++b) m |= (unsigned)(col[q0 + b] == c) << b;
      // an earlier item of the column: its lane has the column
      if (m && q0 + __ffs(m) - 1 < k) first = false;
      if (!first) m = 0;
      while (m) {
        const int e = q0 + __ffs(m) - 1;
        m &= m - 1;
        const double2 v = val[base + (e < nn ? e : kNearItems + e - nn)];
        sn += v.x;
        sd += v.y;
      }
    }
    if (first) add_entry(A2, B2, so, N, row, c, sn, sd);
  }
}

// Candidate panels of the near field per block of kNearBlock consecutive
// rows (compact surface patches, see the internal dof order): those whose near sphere can
// reach any row of the block, |centre_block - centre_panel| < r_block +
// r_panel, in ascending panel order (ballot prefix sums, deterministic). A
// list that would overflow kNearCap is marked with cnt = -1 and its rows scan
// every panel instead.
constexpr int kNearBlock = 64;
constexpr int kNearCap = 2048;

__global__ void __launch_bounds__(256)
    k_near_candidates(int N, int C, const double* __restrict__ X, const float4* __restrict__ cellgeo,
                      int* __restrict__ cnt, int* __restrict__ list) {
  __shared__ float red[6][256];
  __shared__ int woff[8];
  __shared__ int total;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.x * kNearBlock;
  // bounding box of the block's rows
  float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
  if (tid < kNearBlock && r0 + tid < N)
    for (int e = 0; e < 3; ++e) lo[e] = hi[e] = (float)X[3 * (size_t)(r0 + tid) + e];
  for (int e = 0; e < 3; ++e) {
    red[e][tid] = lo[e];
    red[3 + e][tid] = hi[e];
  }
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (tid < o)
      for (int e = 0; e < 3; ++e) {
        red[e][tid] = fminf(red[e][tid], red[e][tid + o]);
        red[3 + e][tid] = fmaxf(red[3 + e][tid], red[3 + e][tid + o]);
      }
    __syncthreads();
  }
  float cen[3], rb2 = 0.f;
  for (int e = 0; e < 3; ++e) {
    cen[e] = 0.5f * (red[e][0] + red[3 + e][0]);
    const float h = 0.5f * (red[3 + e][0] - red[e][0]);
    rb2 += h * h;
  }
  // margin for FP32 rounding of the coordinates and the radii
  const float rb = sqrtf(rb2) * 1.0001f + 1e-6f;
  if (tid == 0) total = 0;
  __syncthreads();
  for (int c0 = 0; c0 < C; c0 += 256) {
    const int c = c0 + tid;
    bool hit = false;
    if (c < C) {
      const float4 g = cellgeo[c];
      const float dx = g.x - cen[0], dy = g.y - cen[1], dz = g.z - cen[2];
      const float reach = sqrtf(g.w) * 1.0001f + rb;
      hit = dx * dx + dy * dy + dz * dz < reach * reach;
    }
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) woff[warp] = __popc(m);
    __syncthreads();
    int base = total;
    for (int w = 0; w < warp; ++w) base += woff[w];
    const int pos = base + __popc(m & ((1u << lane) - 1));
    if (hit && pos < kNearCap) list[(size_t)blockIdx.x * kNearCap + pos] = c;
    __syncthreads();
    if (tid == 0)
      for (int w = 0; w < 8; ++w) total += woff[w];
    __syncthreads();
  }
  if (tid == 0) cnt[blockIdx.x] = total <= kNearCap ? total : -1;
}

// FP64 near field: one warp per row. The lanes test 32 candidate panels at a
// time against the near criterion (same test as the tile kernel); each near,
// non-singular panel is then integrated with the regular rule in FP64, one
// quadrature point per lane, and its four contributions go to the row's items
// in ascending panel order. Bound by the FP64 pipe (and by latency at small
// N). Rules of up to 16 points take two panels at a time, one per half warp,
// and the eight sums of a panel are reduce-scattered: half the lanes no longer
// idle and the reduction's additions fall from 40 to 8 per lane. N = 12,000:
// 1.51 ms -> 0.54, N = 600: 0.205 ms -> 0.063 (kernel times).
// HALF: two panels per step (rules of at most 16 points).
template <bool HALF>
__global__ void __launch_bounds__(256)
    k_near_mixed(int N, int C, const double* __restrict__ X, const int* __restrict__ dnset,
                 const int4* __restrict__ cell_dofs, const float4* __restrict__ cellgeo,
                 const double* __restrict__ rec64, int* __restrict__ item_cnt,
                 int* __restrict__ item_dof, double2* __restrict__ item_val,
                 double* __restrict__ alpha_near, const int* __restrict__ ncnt,
                 const int* __restrict__ nlist, DevErr* err, const __grid_constant__ PanelRule c_q) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= N) return;
  const double xi = X[3 * (size_t)row], yi = X[3 * (size_t)row + 1], zi = X[3 * (size_t)row + 2];
  const float xf = __double2float_rn(xi), yf = __double2float_rn(yi), zf = __double2float_rn(zi);
  int set[kMaxSet];
#pragma unroll
  for (int k = 0; k < kMaxSet; ++k) set[k] = dnset[(size_t)row * kMaxSet + k];
  const int nq = c_q.q1 * c_q.q1;
  constexpr int W = HALF ? 16 : 32;
  const int q0 = lane & (W - 1), half = HALF ? lane >> 4 : 0;
  // the lane that holds component j of a panel's sums writes it once
  const int j = (lane >> 1) & 7;
  const bool writer = HALF ? (lane & 1) == 0 : (lane & 17) == 0;
  double ph[4] = {0, 0, 0, 0};
  if (HALF && q0 < nq)
#pragma unroll
    for (int k = 0; k < 4; ++k) ph[k] = c_q.phi[q0][k];
  double asum = 0.0;
  int nitem = 0;
  double* vals = reinterpret_cast<double*>(item_val + (size_t)row * kItemCap);
  int* dofs = item_dof + (size_t)row * kItemCap;
  // candidates of this row's block (ascending panel order), else every panel
  const int nc = ncnt[row / kNearBlock];
  const int* cl = nlist + (size_t)(row / kNearBlock) * kNearCap;
  const int ntot = nc >= 0 ? nc : C;
  for (int c0 = 0; c0 < ntot; c0 += 32) {
    const int c = c0 + lane < ntot ? (nc >= 0 ? cl[c0 + lane] : c0 + lane) : -1;
    bool nr = false;
    if (c >= 0 && near_test(xf, yf, zf, cellgeo[c])) {
      const int4 d = cell_dofs[c];
      nr = !(in_set_m(set, d.x) || in_set_m(set, d.y) || in_set_m(set, d.z) || in_set_m(set, d.w));
    }
    unsigned m = __ballot_sync(0xffffffffu, nr);
    while (m) {
      const int b0 = __ffs(m) - 1;
      m &= m - 1;
      int b1 = -1;  // the second half warp's panel, if there is one more
      if (HALF && m) {
        b1 = __ffs(m) - 1;
        m &= m - 1;
      }
      const int cell = __shfl_sync(0xffffffffu, c, half ? max(b1, 0) : b0);
      const bool on = !half || b1 >= 0;
      double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      const double2* r = reinterpret_cast<const double2*>(rec64 + (size_t)cell * nq * 8);
      for (int q = q0; on && q < nq; q += W) {
        const double2 p01 = r[4 * q], p23 = r[4 * q + 1], p45 = r[4 * q + 2], p67 = r[4 * q + 3];
        const double Rx = p01.x - xi, Ry = p01.y - yi, Rz = p23.x - zi;
        const double ri = rsqrt(fma(Rx, Rx, fma(Ry, Ry, Rz * Rz)));
        const double sq = ri * p23.y;
        const double dq = -fma(Rx, p45.x, fma(Ry, p45.y, Rz * p67.x)) * (ri * ri * ri);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (HALF) {  // one point per lane
            v[k] = dq * ph[k];
            v[4 + k] = sq * ph[k];
          } else {
            v[k] = fma(dq, c_q.phi[q][k], v[k]);
            v[4 + k] = fma(sq, c_q.phi[q][k], v[4 + k]);
          }
        }
      }
      const double s = panel_reduce8<!HALF>(v, lane);
      if (writer && on) {
        const int it = nitem + 4 * half + (j & 3);
        if (it < kNearItems) {
          if (j < 4) {
            const int4 d = cell_dofs[cell];
            dofs[it] = j < 2 ? (j == 0 ? d.x : d.y) : (j == 2 ? d.z : d.w);
          }
          vals[2 * it + (j >> 2)] = s;
        }
        if (j < 4) asum += s;
      }
      nitem += b1 >= 0 ? 8 : 4;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) asum += __shfl_xor_sync(0xffffffffu, asum, o);
  if (lane == 0) {
    alpha_near[row] = asum;
    item_cnt[2 * row] = nitem;
    if (nitem > kNearItems) dev_fail(err, WBEM_ERR_NOMEM, 43, row, nitem);
  }
}

// FP64 vertex-singular panels, appended to the row's singular items in
// ascending panel order: one CTA per row, its four warps take every fourth
// panel with the rule's points over the lanes. Bound by the FP64 pipe at large
// N, by the latency of one panel's chain at small N; one thread per row took
// 0.55 ms at N = 600 and 0.60 ms at 12,000, now 0.034 and 0.59 ms.
constexpr int kSingWarpsM = 4;

__global__ void __launch_bounds__(kSingWarpsM * 32)
    k_singular_mixed(int N, const double* __restrict__ X, const int* __restrict__ dnset,
                     const int* __restrict__ sptr, const int* __restrict__ scell,
                     const int4* __restrict__ cell_dofs, const QuadTables* __restrict__ qt,
                     int* __restrict__ item_cnt, int* __restrict__ item_dof,
                     double2* __restrict__ item_val, double* __restrict__ alpha_sing, DevErr* err) {
  __shared__ double s_alpha[kSingWarpsM];
  const int row = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double x[3] = {X[3 * (size_t)row], X[3 * (size_t)row + 1], X[3 * (size_t)row + 2]};
  int set[kMaxSet];
#pragma unroll
  for (int k = 0; k < kMaxSet; ++k) set[k] = dnset[(size_t)row * kMaxSet + k];
  const int j = (lane >> 1) & 7;
  double* vals = reinterpret_cast<double*>(item_val + (size_t)row * kItemCap + kNearItems);
  int* dofs = item_dof + (size_t)row * kItemCap + kNearItems;
  const int e0 = sptr[row], n = sptr[row + 1] - e0;
  double asum = 0.0;
  for (int e = warp; e < n; e += kSingWarpsM) {
    const int4 d = cell_dofs[scell[e0 + e]];
    const int id[4] = {d.x, d.y, d.z, d.w};
    int v = -1;
#pragma unroll
    for (int k = 3; k >= 0; --k)
      if (in_set_m(set, id[k])) v = k;
    double s = 0.0;
    if (v < 0) {
      if (lane == 0) dev_fail(err, WBEM_ERR_ARG, 42, row, scell[e0 + e]);
    } else {
      double P[4][3];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) P[k][c] = X[3 * (size_t)id[k] + c];
      s = singular_panel(P, x, qt->sp[v], qt->nsp, lane);
    }
    if ((lane & 17) == 0) {
      const int it = 4 * e + (j & 3);
      if (it < kSingItems) {
        if (j < 4) dofs[it] = j < 2 ? (j == 0 ? d.x : d.y) : (j == 2 ? d.z : d.w);
        vals[2 * it + (j >> 2)] = s;
      }
      if (j < 4) asum += s;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) asum += __shfl_xor_sync(0xffffffffu, asum, o);
  if (lane == 0) s_alpha[warp] = asum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < kSingWarpsM; ++w) s += s_alpha[w];
    alpha_sing[row] = s;
    item_cnt[2 * row + 1] = 4 * n;
    if (4 * n > kSingItems) dev_fail(err, WBEM_ERR_NOMEM, 44, row, 4 * n);
  }
}

// alpha = -(far-field partial sums of every tile + near + singular): a CTA
// takes 32 rows, its 8 warps every eighth tile (a thread per row took
// 0.23 ms at N = 32,768 for want of loads in flight).
__global__ void __launch_bounds__(256)
    k_alpha_mixed(int N, int n_tiles, const double* __restrict__ part,
                  const double* __restrict__ an, const double* __restrict__ as,
                  double* __restrict__ alpha) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  double s = 0;
  if (i < N)
#pragma unroll 4
    for (int t = warp; t < n_tiles; t += 8) s += part[(size_t)t * N + i];
  red[warp][lane] = s;
  __syncthreads();
  if (warp || i >= N) return;
  for (int w = 1; w < 8; ++w) s += red[w][lane];
  alpha[i] = -(s + an[i] + as[i]);
}

#define CUM WB_CU
#define CHKM WB_CHK

void free_mixed(wbem_context* h) {
  if (h->d_A2) { cudaFree(h->d_A2); h->d_A2 = nullptr; }
  if (h->d_B2) { cudaFree(h->d_B2); h->d_B2 = nullptr; }
  if (h->d_lu) { cudaFree(h->d_lu); h->d_lu = nullptr; }
  h->lu_elems = 0;
}

int ensure_system_buffer(wbem_context* h);
int system_ld(int N);

int assemble_mixed(wbem_context* h) {
  const int N = h->N, C = h->C;
  const wbem_options& o = h->opt;
  const int q1 = o.quadrature_order;
  if (q1 < 2 || q1 > 6) {
    h->err = "mixed form supports quadrature orders 2..6";
    return WBEM_ERR_ARG;
  }
  if (!(o.near_field_ratio >= 1.0)) {
    h->err = "near_field_ratio must be >= 1";
    return WBEM_ERR_ARG;
  }
  const size_t nn = (size_t)N * N;
  if (h->d_N) { cudaFree(h->d_N); h->d_N = nullptr; }
  if (h->d_D) { cudaFree(h->d_D); h->d_D = nullptr; }
  if (!h->d_A2 || h->mat_elems != nn) {
    CHKM(dev_alloc(h, &h->d_A2, nn));
    CHKM(dev_alloc(h, &h->d_B2, nn));
    h->mat_elems = nn;
  }
  if (!h->d_alpha) CHKM(dev_alloc(h, &h->d_alpha, (size_t)N));
  CHKM(dev_alloc(h, &h->d_alpha_part, (size_t)h->n_tiles * N));
  CHKM(dev_alloc(h, &h->d_alpha_near, (size_t)N));
  CHKM(dev_alloc(h, &h->d_alpha_sing, (size_t)N));
  const int nq = q1 * q1;
  const int RF = mixed_rec_floats(nq);
  CHKM(dev_alloc(h, &h->d_rec32, (size_t)C * RF));
  CHKM(dev_alloc(h, &h->d_cellgeo, (size_t)C * 4));
  CHKM(dev_alloc(h, &h->d_rec, (size_t)C * nq * 8));
  h->rec_cells = (size_t)C * nq;
  EvTimer tm(h->stream);
  CUM(launch_cell_records_fp64(C, h->d_X, h->d_cell_dofs, h->d_rec, h->quad, h->stream));
  float4* geo_w = reinterpret_cast<float4*>(h->d_cellgeo);
  if (nq <= 16)
    k_cell_records_mixed<true><<<(C + 2 * kRecWarps - 1) / (2 * kRecWarps), kRecWarps * 32, 0, h->stream>>>(
        C, h->d_X, h->d_cell_dofs, h->d_rec32, geo_w, (float)o.near_field_ratio, h->quad);
  else
    k_cell_records_mixed<false><<<(C + kRecWarps - 1) / kRecWarps, kRecWarps * 32, 0, h->stream>>>(
        C, h->d_X, h->d_cell_dofs, h->d_rec32, geo_w, (float)o.near_field_ratio, h->quad);
  CUM(cudaGetLastError());
  h->stats.t_geometry_ms = tm.ms();
  const float4* geo = reinterpret_cast<const float4*>(h->d_cellgeo);
  // the FP32 system copy for the solvers, written alongside N and D
  // the column selection of A2 / B2: the current mask (none yet: Neumann)
  const bool new_sel = !h->d_selmask || h->sel_mask.size() != (size_t)N;
  h->sel_mask.assign(N, 0);
  if (h->have_mask)
    for (int i = 0; i < N; ++i) h->sel_mask[i] = h->mask[h->perm[i]];
  if (new_sel) CHKM(dev_alloc(h, &h->d_selmask, (size_t)N));
  CUM(cudaMemcpyAsync(h->d_selmask, h->sel_mask.data(), (size_t)N, cudaMemcpyHostToDevice, h->stream));
  SysOut so{nullptr, 0, h->d_selmask};
  if (h->have_mask && h->d_mask) {
    CHKM(ensure_system_buffer(h));
    so.S = h->d_lu;
    so.ld = system_ld(N);
  }
  h->s32_state = 0;
  // near field and singular panels (FP64) on the auxiliary stream, beside the
  // FP32 far-field kernel; their contributions are merged afterwards
  if (!h->aux_stream) {
    // high priority: its CTAs take the free slots beside the far-field CTAs
    // first, so the FP64 work hides under the FP32 kernel
    int lo = 0, hi = 0;
    CUM(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    CUM(cudaStreamCreateWithPriority(&h->aux_stream, cudaStreamNonBlocking, hi));
    CUM(cudaEventCreateWithFlags(&h->ev_aux_fork, cudaEventDisableTiming));
    CUM(cudaEventCreateWithFlags(&h->ev_aux_join, cudaEventDisableTiming));
  }
  if (h->item_rows < (size_t)N) {
    CHKM(dev_alloc(h, &h->d_item_val, (size_t)N * kItemCap));
    CHKM(dev_alloc(h, &h->d_item_dof, (size_t)N * kItemCap));
    CHKM(dev_alloc(h, &h->d_item_cnt, (size_t)2 * N));
    h->item_rows = N;
  }
  {
    const int nblk = (N + kNearBlock - 1) / kNearBlock;
    if (h->near_cap < nblk) {
      CHKM(dev_alloc(h, &h->d_near_cnt, (size_t)nblk));
      CHKM(dev_alloc(h, &h->d_near_cells, (size_t)nblk * kNearCap));
      h->near_cap = nblk;
    }
    cudaStream_t ax = h->aux_stream;
    CUM(cudaEventRecord(h->ev_aux_fork, h->stream));
    CUM(cudaStreamWaitEvent(ax, h->ev_aux_fork, 0));
    k_near_candidates<<<nblk, 256, 0, ax>>>(N, C, h->d_X, geo, h->d_near_cnt, h->d_near_cells);
    CUM(cudaGetLastError());
    const unsigned nwb = (unsigned)(((size_t)N * 32 + 255) / 256);
    if (nq <= 16)
      k_near_mixed<true><<<nwb, 256, 0, ax>>>(N, C, h->d_X, h->d_dnset, h->d_cell_dofs, geo, h->d_rec,
                                              h->d_item_cnt, h->d_item_dof, h->d_item_val,
                                              h->d_alpha_near, h->d_near_cnt, h->d_near_cells, h->d_err, h->quad);
    else
      k_near_mixed<false><<<nwb, 256, 0, ax>>>(N, C, h->d_X, h->d_dnset, h->d_cell_dofs, geo, h->d_rec,
                                               h->d_item_cnt, h->d_item_dof, h->d_item_val,
                                               h->d_alpha_near, h->d_near_cnt, h->d_near_cells,
                                               h->d_err, h->quad);
    CUM(cudaGetLastError());
    k_singular_mixed<<<N, kSingWarpsM * 32, 0, ax>>>(N, h->d_X, h->d_dnset, h->d_sptr, h->d_scell,
                                                     h->d_cell_dofs, h->d_quad, h->d_item_cnt, h->d_item_dof,
                                                     h->d_item_val, h->d_alpha_sing, h->d_err);
    CUM(cudaGetLastError());
    CUM(cudaEventRecord(h->ev_aux_join, ax));
  }
  cudaError_t e;
  switch (q1) {
    case 2: e = launch_tile_mixed_t<2>(N, h->d_X, h->d_dnset, h->n_tiles, h->d_tile_ptr, h->d_tile_ent, h->d_cell_dofs, h->d_rec32, geo, h->d_A2, h->d_B2, h->d_alpha_part, so, h->d_err, h->quad, h->stream); break;
    case 3: e = launch_tile_mixed_t<3>(N, h->d_X, h->d_dnset, h->n_tiles, h->d_tile_ptr, h->d_tile_ent, h->d_cell_dofs, h->d_rec32, geo, h->d_A2, h->d_B2, h->d_alpha_part, so, h->d_err, h->quad, h->stream); break;
    case 4: e = launch_tile_mixed_t<4>(N, h->d_X, h->d_dnset, h->n_tiles, h->d_tile_ptr, h->d_tile_ent, h->d_cell_dofs, h->d_rec32, geo, h->d_A2, h->d_B2, h->d_alpha_part, so, h->d_err, h->quad, h->stream); break;
    case 5: e = launch_tile_mixed_t<5>(N, h->d_X, h->d_dnset, h->n_tiles, h->d_tile_ptr, h->d_tile_ent, h->d_cell_dofs, h->d_rec32, geo, h->d_A2, h->d_B2, h->d_alpha_part, so, h->d_err, h->quad, h->stream); break;
    default: e = launch_tile_mixed_t<6>(N, h->d_X, h->d_dnset, h->n_tiles, h->d_tile_ptr, h->d_tile_ent, h->d_cell_dofs, h->d_rec32, geo, h->d_A2, h->d_B2, h->d_alpha_part, so, h->d_err, h->quad, h->stream); break;
  }
  CUM(e);
  h->stats.t_assemble_ms = tm.ms();
  // join the near / singular work and add it to the far-field entries
  CUM(cudaStreamWaitEvent(h->stream, h->ev_aux_join, 0));
  k_merge_items<<<(N + kMergeWarps - 1) / kMergeWarps, kMergeWarps * 32, 0, h->stream>>>(
      N, h->d_item_cnt, h->d_item_dof,
                                                         h->d_item_val, h->d_A2, h->d_B2, so);
  CUM(cudaGetLastError());
  h->stats.t_singular_ms = tm.ms();
  k_alpha_mixed<<<(N + 31) / 32, 256, 0, h->stream>>>(N, h->n_tiles, h->d_alpha_part,
                                                         h->d_alpha_near, h->d_alpha_sing,
                                                         h->d_alpha);
  CUM(cudaGetLastError());
  h->stats.t_alpha_ms = tm.ms();
  if (so.S) h->s32_state = 1;  // entries written; free term and constraints pending
  h->launches += 8;
  return check_device_error(h, "assemble (mixed)");
}

}  // namespace wbem
