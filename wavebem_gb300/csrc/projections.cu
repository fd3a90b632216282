// L2 projections onto Q1 on the device: the node normals of
// ComputationalDomain::compute_normals (source/computational_domain.cc:
// 1525-1620), the surface gradients of BEMProblem::compute_surface_gradients
// (source/bem_problem.cc:1153-1293), and solves with their (consistent) mass
// matrix for the adjoint of the constraint lines.
//
// The mass matrix is gathered from the panels' 4 x 4 blocks through the node ->
// panel lists, and the three right-hand sides of a vector field are solved side
// by side by Jacobi-preconditioned CG in one cooperative launch. Every sum has
// a fixed order.
#include <cuda_runtime.h>
#include <algorithm>
#include <vector>
#include "context.h"
#include "host_util.h"
#include "kernels.h"

namespace wbem {

// the line rule of the regular panel rule (the panels' rule is its product)
struct LineRule {
  int n;
  double x[8], w[8];
};

constexpr int kProjWarps = 4;
constexpr int kProjPoints = 64;  // most points of a panel rule

// Per panel: the 4 x 4 mass block, and the four vertex integrals of a vector
// field: the unit normal (f == nullptr) or the surface gradient of the Q1
// interpolant of f. A warp per panel: the points over the lanes, then each of
// 22 lanes adds one integral over the points in order.
__global__ void __launch_bounds__(kProjWarps * 32)
    k_proj_panels(int C, const double* __restrict__ X, const int4* __restrict__ cell_dofs,
                  const double* __restrict__ f, double* __restrict__ mass, double* __restrict__ rhs,
                  const __grid_constant__ LineRule rule) {
  __shared__ double pt[kProjWarps][kProjPoints][8];  // shape values, area weight, field x weight
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * kProjWarps + warp;
  if (c >= C) return;  // whole warps
  const int4 d = cell_dofs[c];
  const int id[4] = {d.x, d.y, d.z, d.w};
  double P[4][3], fv[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
#pragma unroll
    for (int e = 0; e < 3; ++e) P[k][e] = X[3 * (size_t)id[k] + e];
    if (f) fv[k] = f[id[k]];
  }
  const int nq = rule.n * rule.n;
  for (int q = lane; q < nq; q += 32) {
    const int qa = q % rule.n, qb = q / rule.n;
    const double s = rule.x[qa], t = rule.x[qb], w = rule.w[qa] * rule.w[qb];
    double jx[3], je[3], cr[3];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      jx[e] = (1 - t) * (P[1][e] - P[0][e]) + t * (P[3][e] - P[2][e]);
      je[e] = (1 - s) * (P[2][e] - P[0][e]) + s * (P[3][e] - P[1][e]);
    }
    cr[0] = jx[1] * je[2] - jx[2] * je[1];
    cr[1] = jx[2] * je[0] - jx[0] * je[2];
    cr[2] = jx[0] * je[1] - jx[1] * je[0];
    const double jxw = sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]) * w;
    double* o = pt[warp][q];
    o[0] = (1 - s) * (1 - t);
    o[1] = s * (1 - t);
    o[2] = (1 - s) * t;
    o[3] = s * t;
    o[4] = jxw;
    if (f) {
      const double gx = (1 - t) * (fv[1] - fv[0]) + t * (fv[3] - fv[2]);
      const double ge = (1 - s) * (fv[2] - fv[0]) + s * (fv[3] - fv[1]);
      const double g11 = jx[0] * jx[0] + jx[1] * jx[1] + jx[2] * jx[2];
      const double g12 = jx[0] * je[0] + jx[1] * je[1] + jx[2] * je[2];
      const double g22 = je[0] * je[0] + je[1] * je[1] + je[2] * je[2];
      const double det = g11 * g22 - g12 * g12;
      const double c1 = (g22 * gx - g12 * ge) / det, c2 = (g11 * ge - g12 * gx) / det;
#pragma unroll
      for (int e = 0; e < 3; ++e) o[5 + e] = (c1 * jx[e] + c2 * je[e]) * jxw;
    } else {
#pragma unroll
      for (int e = 0; e < 3; ++e) o[5 + e] = cr[e] * w;
    }
  }
  __syncwarp();
  // lanes 0..9: mass (a, b), b <= a; lanes 10..21: vertex a, component e
  if (lane >= 22) return;
  int a, b;
  if (lane < 10) {
    a = lane < 1 ? 0 : lane < 3 ? 1 : lane < 6 ? 2 : 3;
    b = lane - a * (a + 1) / 2;
  } else {
    a = (lane - 10) / 3;
    b = 5 + (lane - 10) % 3;
  }
  double sum = 0.0;
  for (int q = 0; q < nq; ++q) {
    const double* o = pt[warp][q];
    sum += lane < 10 ? o[a] * o[b] * o[4] : o[a] * o[b];
  }
  if (lane < 10) {
    mass[16 * (size_t)c + 4 * a + b] = sum;
    mass[16 * (size_t)c + 4 * b + a] = sum;
  } else if (rhs) {
    rhs[12 * (size_t)c + 3 * a + b - 5] = sum;
  }
}

// Vectors of the solve, planar (component d of node i at d N + i): right-hand
// side b gathered from the panels (rhs) or given (in b), r = b, zp = (r / diag,
// p = 0), x = 0. The mass matrix by rows: the rcnt[i] entries (rcol, rval) of
// node i from 4 ncptr[i] on; a node of many panels keeps the entries of a column
// apart (merging them is a search per entry, by one thread).
constexpr int kProjRow = 16;    // entries of a row held in shared memory
constexpr int kProjMerge = 64;  // panels of a node whose entries are merged

struct ProjVectors {
  double *b, *dinv, *r, *x, *p, *ap;
  double2* zp;
  int *rcnt, *rcol;
  double* rval;
};

__global__ void k_proj_init(int N, const int* __restrict__ ncptr, const int* __restrict__ ncent,
                            const int4* __restrict__ cell_dofs, const double* __restrict__ mass,
                            const double* __restrict__ rhs, ProjVectors v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double m = 0.0, s[3] = {0, 0, 0};
  int* col = v.rcol + 4 * (size_t)ncptr[i];
  double* val = v.rval + 4 * (size_t)ncptr[i];
  int n = 0;
  const bool merge = ncptr[i + 1] - ncptr[i] <= kProjMerge;
  for (int e = ncptr[i]; e < ncptr[i + 1]; ++e) {
    const int c = ncent[e] >> 2, k = ncent[e] & 3;
    const double* row = mass + 16 * (size_t)c + 4 * k;
    const int4 q = cell_dofs[c];
    const int id[4] = {q.x, q.y, q.z, q.w};
    m += row[k];
    for (int u = 0; u < 4; ++u) {
      int t = merge ? 0 : n;
      while (t < n && col[t] != id[u]) ++t;
      if (t < n) {
        val[t] += row[u];
      } else {
        col[n] = id[u];
        val[n++] = row[u];
      }
    }
    if (rhs)
      for (int d = 0; d < 3; ++d) s[d] += rhs[12 * (size_t)c + 3 * k + d];
  }
  v.rcnt[i] = n;
  const double di = 1.0 / m;
  v.dinv[i] = di;
  for (int d = 0; d < 3; ++d) {
    const size_t o = (size_t)d * N + i;
    const double bi = rhs ? s[d] : v.b[o];
    v.r[o] = bi;
    v.zp[o] = make_double2(di * bi, 0.0);
    v.x[o] = 0.0;
  }
}

// Sums of a and of b over the warp, in every lane: one exchange gives each half
// of the warp one of the two, 5 FP64 additions instead of 10.
__device__ __forceinline__ void proj_warp_sum2(double& a, double& b, int lane) {
  const bool up = (lane & 16) != 0;
  double s = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  a = __shfl_sync(0xffffffffu, s, 0);
  b = __shfl_sync(0xffffffffu, s, 16);
}

// M x_d = b_d, d = 0..2, by Jacobi-preconditioned CG to a relative residual of
// 1e-15. A cooperative launch: CTA g owns the rows of chunk g; warp d holds
// component d, a row per lane (one warp per scheduler: an FP64 instruction
// takes 64 issue cycles of one). Two grid barriers per iteration (bounded
// waits): p = z + beta p_old is recomputed where a row's neighbours need it
// instead of being waited for, so that z and p_old are published together, once
// per iteration. ONE: a lane has one row at most, whose vectors stay in
// registers and whose matrix row (up to kProjRow entries) in shared memory: a
// barrier empties L1, so what is read again after it comes from L2.
// Bound by the barriers' latency and the FP64 chain between them: 0.39 ms for
// the three components at N = 2,000 (41 iterations), where the host's three
// solves, one after the other, took 2.3 ms.
constexpr int kProjRows = 32;
constexpr int kProjThreads = 3 * kProjRows;

template <bool ONE>
__global__ void __launch_bounds__(kProjThreads)
    k_proj_pcg(int N, int max_it, const int* __restrict__ ncptr, ProjVectors v, double* part,
               unsigned* ctr, DevErr* err) {
  __shared__ int scol[ONE ? kProjRow : 1][kProjRows];
  __shared__ double sval[ONE ? kProjRow : 1][kProjRows];
  const int tid = threadIdx.x, lane = tid & 31, d = tid >> 5;
  const int G = gridDim.x, g = blockIdx.x;
  const int per = (N + G - 1) / G;
  const int i0 = min(N, g * per), i1 = min(N, i0 + per);
  const size_t od = (size_t)d * N;
  unsigned target = 0;
  int slot = 0;  // the sums of successive barriers use part in turn
  // totals over all CTAs of the component's two per-thread sums
  // (false: the barrier gave up, and the kernel ends)
  auto total2 = [&](double a, double b, double* ta, double* tb) {
    proj_warp_sum2(a, b, lane);
    double* pp = part + ((size_t)slot * 6 + 2 * d) * G;
    slot ^= 1;
    if (lane < 2) pp[(size_t)lane * G + g] = lane ? b : a;
    target += (unsigned)G;
    if (!grid_barrier(ctr, target, 62, err)) return false;
    a = b = 0.0;
    for (int q = lane; q < G; q += 32) {
      a += __ldcg(pp + q);
      b += __ldcg(pp + G + q);
    }
    proj_warp_sum2(a, b, lane);
    *ta = a;
    *tb = b;
    return true;
  };
  // the lane's row in the ONE form
  const int row = i0 + lane;
  const bool on = ONE && row < i1;
  int n1 = 0;
  size_t base = 0;
  double rr = 0.0, rz1 = 0.0, rp = 0.0, rx = 0.0, rap = 0.0, rd = 0.0;
  if (on) {
    n1 = v.rcnt[row];
    base = 4 * (size_t)ncptr[row];
    if (d == 0)
      for (int e = 0; e < min(n1, kProjRow); ++e) {
        scol[e][lane] = v.rcol[base + e];
        sval[e][lane] = v.rval[base + e];
      }
    rr = v.r[od + row];
    rz1 = v.zp[od + row].x;
    rd = v.dinv[row];
  }
  __syncthreads();
  double s0 = 0.0, s1 = 0.0, bn2, rz;
  if (ONE) {
    s0 = rr * rr;
    s1 = rr * rz1;
  } else {
    for (int i = i0 + lane; i < i1; i += kProjRows) {
      const double b = v.r[od + i];
      s0 = fma(b, b, s0);
      s1 = fma(b, v.zp[od + i].x, s1);
    }
  }
  if (!total2(s0, s1, &bn2, &rz)) return;
  const double bn = sqrt(bn2);
  bool done = !(bn > 0.0);  // of this component
  double beta = 0.0;
  auto term = [&](double m, int j, double s) {
    const double2 q = __ldcg(v.zp + od + j);
    return fma(m, fma(beta, q.y, q.x), s);
  };
  for (int it = 0; it < max_it; ++it) {
    if (__syncthreads_and(done)) break;  // the same in every CTA
    double pap = 0.0;
    if (ONE) {
      double s = 0.0;
      const int ns = min(n1, kProjRow);
#pragma unroll 9
      for (int e = 0; e < ns; ++e) s = term(sval[e][lane], scol[e][lane], s);
      for (int e = kProjRow; e < n1; ++e) s = term(v.rval[base + e], v.rcol[base + e], s);
      rp = fma(beta, rp, rz1);
      rap = s;
      pap = rp * s;
    } else {
      for (int i = i0 + lane; i < i1; i += kProjRows) {
        double s = 0.0;
        const int n = v.rcnt[i];
        const size_t b = 4 * (size_t)ncptr[i];
#pragma unroll 9
        for (int e = 0; e < n; ++e) s = term(v.rval[b + e], v.rcol[b + e], s);
        const double2 q = v.zp[od + i];
        const double p = fma(beta, q.y, q.x);
        v.p[od + i] = p;
        v.ap[od + i] = s;
        pap = fma(p, s, pap);
      }
    }
    double tp, unused;
    if (!total2(pap, 0.0, &tp, &unused)) return;
    const double alpha = done ? 0.0 : rz / tp;
    double rn = 0.0, rz2 = 0.0;
    if (ONE) {
      if (!done) {
        rx = fma(alpha, rp, rx);
        rr = fma(-alpha, rap, rr);
      }
      rz1 = rd * rr;
      if (on) v.zp[od + row] = make_double2(rz1, rp);
      rn = rr * rr;
      rz2 = rr * rz1;
    } else {
      for (int i = i0 + lane; i < i1; i += kProjRows) {
        const size_t o = od + i;
        const double p = v.p[o];
        double r = v.r[o];
        if (!done) {
          v.x[o] = fma(alpha, p, v.x[o]);
          r = fma(-alpha, v.ap[o], r);
          v.r[o] = r;
        }
        const double z = v.dinv[i] * r;
        v.zp[o] = make_double2(z, p);
        rn = fma(r, r, rn);
        rz2 = fma(r, z, rz2);
      }
    }
    double trn, trz;
    if (!total2(rn, rz2, &trn, &trz)) return;
    // not a number ends the component too (the caller sees it in x)
    done = done || !(sqrt(trn) >= 1e-15 * bn);
    beta = done ? 0.0 : trz / rz;
    rz = trz;
  }
  if (on) v.x[od + row] = rx;
}

// Device buffers of the projections, kept with the mesh.
struct ProjState {
  double *mass = nullptr, *rhs = nullptr, *f = nullptr, *vec = nullptr, *part = nullptr;
  int *rcnt = nullptr, *rcol = nullptr;
  double* rval = nullptr;
  unsigned* ctr = nullptr;
  int ctas = 0;
};

void free_projections(wbem_context* h) {
  if (!h->proj_state) return;
  ProjState* P = static_cast<ProjState*>(h->proj_state);
  for (void* p : {(void*)P->mass, (void*)P->rhs, (void*)P->f, (void*)P->vec, (void*)P->part, (void*)P->rcnt, (void*)P->rcol,
                  (void*)P->rval, (void*)P->ctr})
    if (p) cudaFree(p);
  delete P;
  h->proj_state = nullptr;
}

static int proj_state(wbem_context* h, ProjState** out) {
  if (!h->proj_state) h->proj_state = new ProjState();
  ProjState* P = static_cast<ProjState*>(h->proj_state);
  *out = P;
  if (P->ctr) return WBEM_OK;
  const size_t N = h->N, C = h->C;
  int sms = 0;
  WB_CU(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device));
  P->ctas = std::max(1, std::min(sms, (h->N + kProjRows - 1) / kProjRows));
  WB_CHK(dev_alloc(h, &P->mass, 16 * C));
  WB_CHK(dev_alloc(h, &P->rhs, 12 * C));
  WB_CHK(dev_alloc(h, &P->f, N));
  WB_CHK(dev_alloc(h, &P->rcnt, N));
  WB_CHK(dev_alloc(h, &P->rcol, 16 * C));
  WB_CHK(dev_alloc(h, &P->rval, 16 * C));
  WB_CHK(dev_alloc(h, &P->vec, 22 * N));  // see project_field
  WB_CHK(dev_alloc(h, &P->part, (size_t)12 * P->ctas));
  WB_CHK(dev_alloc(h, &P->ctr, (size_t)1));
  return WBEM_OK;
}

// x = M^-1 (kind 0: integrals of the unit normals; kind 1: integrals of the
// surface gradients of f; kind 2: the given right-hand side), node-major
// 3 i + d, caller order. in: f (N) for kind 1, the right-hand side (3 N) for
// kind 2.
int project_field(wbem_context* h, int kind, const double* in, std::vector<double>& x) {
  WB_CU(cudaSetDevice(h->device));
  ProjState* P;
  WB_CHK(proj_state(h, &P));
  const int N = h->N, C = h->C;
  double* v = P->vec;
  const size_t n3 = (size_t)3 * N;
  // zp (2 x 3 N, 16-byte aligned), b, r, x, p, ap (3 N each), dinv (N)
  const ProjVectors pv{v + 2 * n3, v + 7 * n3, v + 3 * n3, v + 4 * n3, v + 5 * n3, v + 6 * n3,
                       reinterpret_cast<double2*>(v), P->rcnt, P->rcol, P->rval};
  LineRule rule{};
  rule.n = h->gauss_n;
  for (int k = 0; k < rule.n; ++k) {
    rule.x[k] = h->gauss_x[k];
    rule.w[k] = h->gauss_w[k];
  }
  std::vector<double> up;
  if (kind == 1) {
    up.resize(N);
    for (int i = 0; i < N; ++i) up[i] = in[h->perm[i]];
    WB_CU(cudaMemcpyAsync(P->f, up.data(), sizeof(double) * N, cudaMemcpyHostToDevice, h->stream));
  } else if (kind == 2) {
    up.resize(n3);
    for (int d = 0; d < 3; ++d)
      for (int i = 0; i < N; ++i) up[(size_t)d * N + i] = in[3 * (size_t)h->perm[i] + d];
    WB_CU(cudaMemcpyAsync(pv.b, up.data(), sizeof(double) * n3, cudaMemcpyHostToDevice, h->stream));
  }
  WB_CU(cudaMemsetAsync(P->ctr, 0, sizeof(unsigned), h->stream));
  double* rhs = kind == 2 ? nullptr : P->rhs;
  k_proj_panels<<<(C + kProjWarps - 1) / kProjWarps, kProjWarps * 32, 0, h->stream>>>(
      C, h->d_X, h->d_cell_dofs, kind == 1 ? P->f : nullptr, P->mass, rhs, rule);
  k_proj_init<<<(N + 127) / 128, 128, 0, h->stream>>>(N, h->d_ncptr, h->d_ncent, h->d_cell_dofs, P->mass,
                                                         rhs, pv);
  WB_CU(cudaGetLastError());
  int max_it = 10 * N + 100;
  void* args[] = {(void*)&N, (void*)&max_it, (void*)&h->d_ncptr, (void*)&pv, (void*)&P->part, (void*)&P->ctr,
                  (void*)&h->d_err};
  int ctas = P->ctas;
  WB_CU(launch_coresident(ctas, [&](int n) {
    const bool one = (N + n - 1) / n <= kProjRows;
    return cudaLaunchCooperativeKernel(one ? (const void*)k_proj_pcg<true> : (const void*)k_proj_pcg<false>,
                                       dim3(n), dim3(kProjThreads), args, 0, h->stream);
  }));
  std::vector<double> xi(n3);
  WB_CU(cudaMemcpyAsync(xi.data(), pv.x, sizeof(double) * n3, cudaMemcpyDeviceToHost, h->stream));
  WB_CHK(check_device_error(h, "L2 projection"));
  x.resize(n3);
  for (int d = 0; d < 3; ++d)
    for (int i = 0; i < N; ++i) x[3 * (size_t)h->perm[i] + d] = xi[(size_t)d * N + i];
  return WBEM_OK;
}

}  // namespace wbem
