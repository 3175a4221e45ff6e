// Euler-Bernoulli beams (body family 3).  The reference declares the family and leaves its
// routines empty (operators_struct.F90:104-106, 146-148, 171-174, 285-288, 378-381, 472-474);
// this is the library's own formulation, coupled the way the reference couples its torsional
// body (operators_struct.F90:14-505) with matrices in place of the hinge's scalars:
//   * a linear (small-deflection) beam clamped at its first point, along the line from its
//     first to its last point; nel Hermite-cubic elements with DOFs (w, dw/ds) at the nodes,
//     the clamped node's removed (ndof = 2 nel); consistent mass and stiffness;
//   * body point j moves by W q along the beam's normal, W = [-sin g Phi; cos g Phi]; point
//     forces act on the DOFs as F = (delta/dt) W^T f;
//   * trapezoidal Newmark with K_eff = 4/dt^2 M + K:
//       dq = K_eff^-1 (M a - K_eff q) + K_eff^-1 F,  a = 4/dt^2 q0 + 4/dt qd0 + qdd0;
//       compute_rhs: delta W (r - jr - qd), r = qd0 + qd + 2/dt (q0 - q),
//                    jr = 2/dt K_eff^-1 (M a - K_eff q);
//       b_times: (2 delta^2 / dt^2) W K_eff^-1 W^T x;   initial_acc: qdd = M^-1 (F - K q).
// The matrices are built on the host at context creation (the beam is linear, so they never
// change); the kernels are dense products on one CTA, which runs every beam in turn.
#include <cmath>
#include <vector>

#include "ctx.cuh"

namespace ib {

namespace {

// inverse of an SPD matrix (row-major, n x n) by Cholesky, in double
bool spd_inverse(const std::vector<double>& A, int n, std::vector<double>* out) {
  std::vector<double> L((size_t)n * n, 0.0);
  for (int j = 0; j < n; ++j) {
    double d = A[(size_t)j * n + j];
    for (int k = 0; k < j; ++k) d -= L[(size_t)j * n + k] * L[(size_t)j * n + k];
    if (!(d > 0.0)) return false;
    const double ljj = std::sqrt(d);
    L[(size_t)j * n + j] = ljj;
    for (int i = j + 1; i < n; ++i) {
      double v = A[(size_t)i * n + j];
      for (int k = 0; k < j; ++k) v -= L[(size_t)i * n + k] * L[(size_t)j * n + k];
      L[(size_t)i * n + j] = v / ljj;
    }
  }
  out->assign((size_t)n * n, 0.0);
  std::vector<double> col(n);
  for (int c = 0; c < n; ++c) {
    for (int i = 0; i < n; ++i) {   // L y = e_c
      double v = i == c ? 1.0 : 0.0;
      for (int k = 0; k < i; ++k) v -= L[(size_t)i * n + k] * col[k];
      col[i] = v / L[(size_t)i * n + i];
    }
    for (int i = n - 1; i >= 0; --i) {   // L^T x = y
      double v = col[i];
      for (int k = i + 1; k < n; ++k) v -= L[(size_t)k * n + i] * col[k];
      col[i] = v / L[(size_t)i * n + i];
    }
    for (int i = 0; i < n; ++i) (*out)[(size_t)i * n + c] = col[i];
  }
  return true;
}

}  // namespace

int beam_build(Ctx* c, const IbBody* bodies, int nbody, std::string* msg) {
  const double dt = c->p.dt;
  int off = 0;
  std::vector<BeamDev> hdev;
  for (int i = 0; i < nbody; ++i) {
    const IbBody& b = bodies[i];
    const int npts = b.npts;
    if (b.fam != 3) { off += 2 * npts; continue; }
    const int nel = b.nelem > 0 ? b.nelem : (npts - 1) / 2;
    if (nel < 1) { *msg = "a beam needs at least one element"; return IB_ERR_ARG; }
    if (!(b.itheta > 0) || !(b.ktheta > 0)) { *msg = "a beam needs mass per length (itheta) and EI (ktheta) > 0"; return IB_ERR_ARG; }
    const int nd = 2 * nel, np2 = 2 * npts;
    const double dx = b.x[npts - 1] - b.x[0], dy = b.y[npts - 1] - b.y[0];
    const double length = std::sqrt(dx * dx + dy * dy);
    const double cg = dx / length, sg = dy / length;
    const double h = length / nel, rho = b.itheta, EI = b.ktheta;
    const double kc = EI / (h * h * h), mc = rho * h / 420.0;
    const double ke[4][4] = {{12.0, 6.0 * h, -12.0, 6.0 * h}, {6.0 * h, 4.0 * h * h, -6.0 * h, 2.0 * h * h},
                             {-12.0, -6.0 * h, 12.0, -6.0 * h}, {6.0 * h, 2.0 * h * h, -6.0 * h, 4.0 * h * h}};
    const double me[4][4] = {{156.0, 22.0 * h, 54.0, -13.0 * h}, {22.0 * h, 4.0 * h * h, 13.0 * h, -3.0 * h * h},
                             {54.0, 13.0 * h, 156.0, -22.0 * h}, {-13.0 * h, -3.0 * h * h, -22.0 * h, 4.0 * h * h}};
    const int NG = 2 * (nel + 1);
    std::vector<double> KG((size_t)NG * NG, 0.0), MG((size_t)NG * NG, 0.0);
    for (int e = 0; e < nel; ++e)
      for (int a = 0; a < 4; ++a)
        for (int q = 0; q < 4; ++q) {
          KG[(size_t)(2 * e + a) * NG + 2 * e + q] += kc * ke[a][q];
          MG[(size_t)(2 * e + a) * NG + 2 * e + q] += mc * me[a][q];
        }
    std::vector<double> K((size_t)nd * nd), M((size_t)nd * nd), Ke((size_t)nd * nd);
    for (int r = 0; r < nd; ++r)
      for (int q = 0; q < nd; ++q) {
        K[(size_t)r * nd + q] = KG[(size_t)(r + 2) * NG + q + 2];
        M[(size_t)r * nd + q] = MG[(size_t)(r + 2) * NG + q + 2];
        Ke[(size_t)r * nd + q] = 4.0 / (dt * dt) * M[(size_t)r * nd + q] + K[(size_t)r * nd + q];
      }
    std::vector<double> Ki, Mi;
    if (!spd_inverse(Ke, nd, &Ki) || !spd_inverse(M, nd, &Mi)) { *msg = "beam matrices not positive definite"; return IB_ERR_ARG; }
    std::vector<double> phi((size_t)npts * nd, 0.0), W((size_t)np2 * nd);
    for (int j = 0; j < npts; ++j) {
      const int e = std::min((int)((long long)j * nel / (npts - 1)), nel - 1);
      const double xi = (double)((long long)j * nel - (long long)e * (npts - 1)) / (double)(npts - 1);
      const double xi2 = xi * xi, xi3 = xi * xi * xi;
      const double nv[4] = {1.0 - 3.0 * xi2 + 2.0 * xi3, h * (xi - 2.0 * xi2 + xi3), 3.0 * xi2 - 2.0 * xi3,
                            h * (xi3 - xi2)};
      for (int a = 0; a < 4; ++a) {
        const int dof = 2 * e + a - 2;
        if (dof >= 0) phi[(size_t)j * nd + dof] = nv[a];
      }
    }
    for (int j = 0; j < npts; ++j)
      for (int q = 0; q < nd; ++q) {
        W[(size_t)j * nd + q] = -sg * phi[(size_t)j * nd + q];
        W[(size_t)(npts + j) * nd + q] = cg * phi[(size_t)j * nd + q];
      }
    // B = W K_eff^-1 W^T
    std::vector<double> KiWt((size_t)nd * np2, 0.0), B((size_t)np2 * np2, 0.0);
    for (int r = 0; r < nd; ++r)
      for (int j = 0; j < np2; ++j) {
        double s = 0.0;
        for (int q = 0; q < nd; ++q) s += Ki[(size_t)r * nd + q] * W[(size_t)j * nd + q];
        KiWt[(size_t)r * np2 + j] = s;
      }
    for (int i2 = 0; i2 < np2; ++i2)
      for (int j = 0; j < np2; ++j) {
        double s = 0.0;
        for (int q = 0; q < nd; ++q) s += W[(size_t)i2 * nd + q] * KiWt[(size_t)q * np2 + j];
        B[(size_t)i2 * np2 + j] = s;
      }
    // device storage of this beam: matrices, reference positions, state (+ scratch)
    const size_t nmat = (size_t)5 * nd * nd + (size_t)np2 * nd + (size_t)npts * nd + (size_t)np2 * np2 + np2 + 10 * (size_t)nd;
    double* mem = nullptr;
    if (cudaMalloc(&mem, 8 * nmat) != cudaSuccess) { *msg = "beam allocation failed"; return IB_ERR_NOMEM; }
    c->beam_mem.push_back(mem);
    cudaMemset(mem, 0, 8 * nmat);
    BeamDev d;
    d.off = off; d.npts = npts; d.ndof = nd; d.sg = sg; d.cg = cg;
    double* q = mem;
    auto put = [&](const std::vector<double>& v) { double* r = q; cudaMemcpy(r, v.data(), 8 * v.size(), cudaMemcpyHostToDevice); q += v.size(); return r; };
    d.M = put(M); d.K = put(K); d.Ke = put(Ke); d.Ki = put(Ki); d.Mi = put(Mi);
    d.W = put(W); d.phi = put(phi); d.B = put(B);
    std::vector<double> xy(np2);
    for (int j = 0; j < npts; ++j) { xy[j] = b.x[j]; xy[npts + j] = b.y[j]; }
    d.xy0 = put(xy);
    d.q = q; d.qd = q + nd; d.qdd = q + 2 * nd; d.q0 = q + 3 * nd; d.qd0 = q + 4 * nd; d.qdd0 = q + 5 * nd;
    d.t1 = q + 6 * nd; d.t2 = q + 7 * nd; d.t3 = q + 8 * nd; d.t4 = q + 9 * nd;
    hdev.push_back(d);
    off += np2;
  }
  c->nbeam = (int)hdev.size();
  c->beams_h = hdev;
  if (c->nbeam > 0) {
    if (cudaMalloc(&c->beams, sizeof(BeamDev) * c->nbeam + sizeof(double)) != cudaSuccess) {
      *msg = "beam allocation failed";
      return IB_ERR_NOMEM;
    }
    c->beam_err = (double*)(c->beams + c->nbeam);
    if (cudaMemcpy(c->beams, hdev.data(), sizeof(BeamDev) * c->nbeam, cudaMemcpyHostToDevice) != cudaSuccess)
      return IB_ERR_CUDA;
    RC(wait_uploads());
  }
  return IB_OK;
}

void beam_free(Ctx* c) {
  for (double* m : c->beam_mem) cudaFree(m);
  c->beam_mem.clear();
  if (c->beams) cudaFree(c->beams);
  c->beams = nullptr;
  c->beam_err = nullptr;
  c->nbeam = 0;
}

// out[r] = sum_q A[r][q] x[q] over the CTA, one row per thread (the sum in column order)
__device__ void cta_matvec(const double* __restrict__ A, int rows, int cols, const double* x, double* out) {
  for (int r = threadIdx.x; r < rows; r += blockDim.x) {
    double s = 0.0;
    for (int q = 0; q < cols; ++q) s = fma(A[(size_t)r * cols + q], x[q], s);
    out[r] = s;
  }
  __syncthreads();
}

// The iterations' kernels (k_beam_rhs, k_beam_dx) run one CTA; what bounds them is the chain of
// dependent FP64 operations and barriers.  So every product runs over the nonzeros only where the
// matrix is sparse (M and K_eff couple a node with its neighbours, a point's rows of W and Phi the
// four DOFs of its element) and the dense K_eff^-1 spreads each row over kBeamLanes lanes.  39
// points, 38 DOFs: 7.9 us (dx) and 6.4 us (rhs); 24 and 15 us with a dense row per thread.
// The quotients come from the host (an FP64 division holds the pipe longer than a row's product),
// and a row's other terms are formed after the product by a thread per row, not by the one lane in
// eight that holds its sum.
constexpr int kBeamThreads = 512;
constexpr int kBeamLanes = 8;

struct BeamFac {
  double a2, a1, v, f, delta;   // 4/dt^2, 4/dt, 2/dt, delta/dt, delta
  BeamFac(double dt, double d) : a2(4.0 / (dt * dt)), a1(4.0 / dt), v(2.0 / dt), f(d / dt), delta(d) {}
};

// sum over a row group's lanes, valid on each of them
__device__ __forceinline__ double beam_lane_sum(double s) {
#pragma unroll
  for (int o = kBeamLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// y = A x for a dense matrix, kBeamLanes lanes a row; every thread of the CTA calls it
__device__ __forceinline__ void beam_dense(const double* __restrict__ A, int rows, int cols, const double* x,
                                           double* y) {
  const int l = threadIdx.x % kBeamLanes;
  for (int r0 = 0; r0 < rows; r0 += kBeamThreads / kBeamLanes) {
    const int r = r0 + threadIdx.x / kBeamLanes;
    double s = 0.0;
    if (r < rows) {
      const double* row = A + (size_t)r * cols;
#pragma unroll 4
      for (int q = l; q < cols; q += kBeamLanes) s = fma(row[q], x[q], s);
    }
    s = beam_lane_sum(s);
    if (r < rows && l == 0) y[r] = s;
  }
}

// Row k of M x or K x: DOFs 2n, 2n+1 (node n + 1) couple with 2n-2 .. 2n+3.
__device__ __forceinline__ double beam_band_row(const double* __restrict__ A, int nd, int k, const double* x) {
  const int c0 = (k & ~1) - 2;
  double e = 0.0, o = 0.0;
#pragma unroll
  for (int t = 0; t < 6; t += 2) {
    const int q = c0 + t;   // even, and so is nd: q and q + 1 are in range together
    if (q >= 0 && q < nd) {
      e = fma(A[(size_t)k * nd + q], x[q], e);
      o = fma(A[(size_t)k * nd + q + 1], x[q + 1], o);
    }
  }
  return e + o;
}

// First DOF (2e - 2, negative at the clamped element) of point j's element, as beam_build places it.
__device__ __forceinline__ int beam_point_dof(const BeamDev& b, int j) {
  const int nel = b.ndof / 2;
  const int e = min((int)((long long)j * nel / (b.npts - 1)), nel - 1);
  return 2 * e - 2;
}

// Row of W or Phi of a point whose element starts at DOF d, times x.
__device__ __forceinline__ double beam_point_row(const double* __restrict__ row, int nd, int d, const double* x) {
  double e = 0.0, o = 0.0;
#pragma unroll
  for (int t = 0; t < 4; t += 2)
    if (d + t >= 0 && d + t < nd) {
      e = fma(row[d + t], x[d + t], e);
      o = fma(row[d + t + 1], x[d + t + 1], o);
    }
  return e + o;
}

// a = 4/dt^2 q0 + 4/dt qd0 + qdd0 (in t1), then t3 = M a - K_eff q, a thread per row (no barrier after)
__device__ __forceinline__ void beam_residual(const BeamDev& b, const BeamFac& fc, double* t1, double* t3) {
  const int nd = b.ndof;
  for (int k = threadIdx.x; k < nd; k += kBeamThreads) t1[k] = fc.a2 * b.q0[k] + fc.a1 * b.qd0[k] + b.qdd0[k];
  __syncthreads();
  for (int k = threadIdx.x; k < nd; k += kBeamThreads)
    t3[k] = beam_band_row(b.M, nd, k, t1) - beam_band_row(b.Ke, nd, k, b.q);
}

// t2 = fac W^T f: row k sums the points of the two elements that share DOF k's node, kBeamLanes lanes a
// row, from the warps the residual's rows leave free
__device__ __forceinline__ void beam_load(const BeamDev& b, double fac, const double* __restrict__ f, double* t2) {
  const int nd = b.ndof, nel = nd / 2, np1 = b.npts - 1;
  const int l = threadIdx.x % kBeamLanes;
  for (int k0 = 0; k0 < nd; k0 += kBeamThreads / kBeamLanes) {
    // the last groups first: the first warps have the residual's rows
    const int k = k0 + (kBeamThreads - 1 - threadIdx.x) / kBeamLanes;
    double s = 0.0;
    if (k < nd) {
      const int n = k / 2 + 1;   // the node; its elements are n - 1 and n
      const int jlo = (int)(((long long)(n - 1) * np1 + nel - 1) / nel);
      const int jhi = n + 1 >= nel ? np1 : (int)(((long long)(n + 1) * np1 + nel - 1) / nel) - 1;
      for (int j = jlo + l; j <= jhi; j += kBeamLanes) {
        s = fma(b.W[(size_t)j * nd + k], f[b.off + j], s);
        s = fma(b.W[(size_t)(b.npts + j) * nd + k], f[b.off + b.npts + j], s);
      }
    }
    s = beam_lane_sum(s);
    if (k < nd && l == 0) t2[k] = fac * s;
  }
}

__global__ void __launch_bounds__(kBeamThreads) k_beam_rhs(const BeamDev* __restrict__ beams, int nbeam, BeamFac fc,
                                                           double* y) {
  IB_GRID_DEP_WAIT();
  for (int i = 0; i < nbeam; ++i) {
    const BeamDev b = beams[i];
    const int nd = b.ndof;
    beam_residual(b, fc, b.t1, b.t3);
    __syncthreads();
    beam_dense(b.Ki, nd, nd, b.t3, b.t4);   // K_eff^-1 (M a - K_eff q)
    __syncthreads();
    for (int k = threadIdx.x; k < nd; k += kBeamThreads) {
      const double r = b.qd0[k] + b.qd[k] + fc.v * (b.q0[k] - b.q[k]);
      const double jr = fc.v * b.t4[k];
      b.t1[k] = fc.delta * (r - jr - b.qd[k]);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < 2 * b.npts; j += kBeamThreads)
      y[b.off + j] = beam_point_row(b.W + (size_t)j * nd, nd, beam_point_dof(b, j < b.npts ? j : j - b.npts), b.t1);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kBeamThreads) k_beam_dx(const BeamDev* __restrict__ beams, int nbeam, BeamFac fc,
                                                          const double* __restrict__ f, double* xb, double* yb,
                                                          double* err, int fresh) {
  IB_GRID_DEP_WAIT();
  __shared__ double red[kBeamThreads / 32];
  double emax = fresh ? 0.0 : err[0];   // the torsional bodies' maximum (zero without them)
  for (int i = 0; i < nbeam; ++i) {
    const BeamDev b = beams[i];
    const int nd = b.ndof;
    beam_residual(b, fc, b.t1, b.t3);
    beam_load(b, fc.f, f, b.t2);   // F = (delta/dt) W^T f
    __syncthreads();
    for (int k = threadIdx.x; k < nd; k += kBeamThreads) b.t4[k] = b.t3[k] + b.t2[k];
    __syncthreads();
    beam_dense(b.Ki, nd, nd, b.t4, b.t1);   // dq = K_eff^-1 (M a - K_eff q + F)
    __syncthreads();
    double em = 0.0;
    for (int k = threadIdx.x; k < nd; k += kBeamThreads) {
      const double dq = b.t1[k];
      em = max_magnitude(em, dq);
      const double qn = b.q[k] + dq;
      b.q[k] = qn;
      b.qd[k] = -b.qd0[k] + fc.v * (qn - b.q0[k]);
      b.qdd[k] = -b.qdd0[k] - fc.a1 * b.qd0[k] + fc.a2 * (qn - b.q0[k]);
    }
    for (int o = 16; o > 0; o >>= 1) em = max_magnitude(em, __shfl_xor_sync(0xffffffffu, em, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = em;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < kBeamThreads / 32; ++w) emax = max_magnitude(emax, red[w]);
    // positions: x0 + (-sin g) d, y0 + cos g d, d = Phi q
    for (int j = threadIdx.x; j < b.npts; j += kBeamThreads) {
      const double d = beam_point_row(b.phi + (size_t)j * nd, nd, beam_point_dof(b, j), b.q);
      const double px = __dadd_rn(b.xy0[j], __dmul_rn(-b.sg, d));
      const double py = __dadd_rn(b.xy0[b.npts + j], __dmul_rn(b.cg, d));
      xb[b.off + j] = px; xb[b.off + b.npts + j] = px;
      yb[b.off + j] = py; yb[b.off + b.npts + j] = py;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) err[0] = emax;
}

__global__ void k_beam_btimes(const BeamDev* __restrict__ beams, int nbeam, double scale,
                              const double* __restrict__ x, double* y) {
  IB_GRID_DEP_WAIT();
  for (int i = 0; i < nbeam; ++i) {
    const BeamDev b = beams[i];
    const int np2 = 2 * b.npts;
    for (int r = threadIdx.x; r < np2; r += blockDim.x) {
      double s = 0.0;
      for (int q = 0; q < np2; ++q) s = fma(b.B[(size_t)r * np2 + q], x[b.off + q], s);
      y[b.off + r] = y[b.off + r] + s * scale;
    }
    __syncthreads();
  }
}

// St (column-major nf x nf) += scale B on each beam's block
__global__ void k_beam_add_b(const BeamDev* __restrict__ beams, int nbeam, double scale, int nf, double* St) {
  IB_GRID_DEP_WAIT();
  for (int i = 0; i < nbeam; ++i) {
    const BeamDev b = beams[i];
    const int np2 = 2 * b.npts;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < np2 * np2; t += gridDim.x * blockDim.x) {
      const int r = t / np2, q = t % np2;
      double* e = St + (size_t)(b.off + q) * nf + (b.off + r);
      *e = *e + b.B[(size_t)r * np2 + q] * scale;
    }
  }
}

__global__ void k_beam_initial_acc(const BeamDev* __restrict__ beams, int nbeam, double dt, double delta,
                                   const double* __restrict__ f) {
  IB_GRID_DEP_WAIT();
  for (int i = 0; i < nbeam; ++i) {
    const BeamDev b = beams[i];
    const int nd = b.ndof, np2 = 2 * b.npts;
    for (int k = threadIdx.x; k < nd; k += blockDim.x) {
      double s = 0.0;
      for (int j = 0; j < np2; ++j) s = fma(b.W[(size_t)j * nd + k], f[b.off + j], s);
      b.t1[k] = delta / dt * s;
    }
    __syncthreads();
    cta_matvec(b.K, nd, nd, b.q, b.t2);
    for (int k = threadIdx.x; k < nd; k += blockDim.x) b.t3[k] = b.t1[k] - b.t2[k];
    __syncthreads();
    cta_matvec(b.Mi, nd, nd, b.t3, b.qdd);
  }
}

__global__ void k_beam_save(const BeamDev* __restrict__ beams, int nbeam) {
  IB_GRID_DEP_WAIT();
  for (int i = 0; i < nbeam; ++i) {
    const BeamDev b = beams[i];
    for (int k = threadIdx.x; k < b.ndof; k += blockDim.x) {
      b.q0[k] = b.q[k];
      b.qd0[k] = b.qd[k];
      b.qdd0[k] = b.qdd[k];
    }
  }
}

static int after(int rc) { return rc == IB_OK && cudaGetLastError() == cudaSuccess ? IB_OK : IB_ERR_CUDA; }

int launch_beam_rhs(Ctx* c, double* y, cudaStream_t st) {
  if (c->nbeam == 0) return IB_OK;
  count_launch();
  k_beam_rhs<<<1, kBeamThreads, 0, st>>>(c->beams, c->nbeam, BeamFac(c->p.dt, c->delta), y);
  return after(IB_OK);
}
int launch_beam_dx(Ctx* c, const double* f, cudaStream_t st, bool own_err) {
  if (c->nbeam == 0) return IB_OK;
  count_launch();
  k_beam_dx<<<1, kBeamThreads, 0, st>>>(c->beams, c->nbeam, BeamFac(c->p.dt, c->delta), f, c->xb, c->yb,
                                        own_err ? c->beam_err : c->err_fsi, own_err ? 1 : 0);
  return after(IB_OK);
}
int launch_beam_btimes(Ctx* c, const double* x, double* y, cudaStream_t st) {
  if (c->nbeam == 0) return IB_OK;
  count_launch();
  const double dt = c->p.dt;
  k_beam_btimes<<<1, 256, 0, st>>>(c->beams, c->nbeam, 2.0 * c->delta * c->delta / (dt * dt), x, y);
  return after(IB_OK);
}
int launch_beam_add_b(Ctx* c, double* St, cudaStream_t st) {
  if (c->nbeam == 0) return IB_OK;
  count_launch();
  const double dt = c->p.dt;
  k_beam_add_b<<<64, 256, 0, st>>>(c->beams, c->nbeam, 2.0 * c->delta * c->delta / (dt * dt), c->nf, St);
  return after(IB_OK);
}
int launch_beam_initial_acc(Ctx* c, const double* f, cudaStream_t st) {
  if (c->nbeam == 0) return IB_OK;
  count_launch();
  k_beam_initial_acc<<<1, 256, 0, st>>>(c->beams, c->nbeam, c->p.dt, c->delta, f);
  return after(IB_OK);
}
int launch_beam_save(Ctx* c, cudaStream_t st) {
  if (c->nbeam == 0) return IB_OK;
  count_launch();
  k_beam_save<<<1, 256, 0, st>>>(c->beams, c->nbeam);
  return after(IB_OK);
}

}  // namespace ib
