// Device GMRES with the semantics of PETSc 3.11 KSPGMRES as the reference
// configures it (variables.F90:565-574): restart 30, classical Gram-Schmidt
// without refinement (borthog2.c), Givens-rotation least squares, nonzero initial
// guess, unpreconditioned residual norm, convergence when the rotated residual
// estimate <= max(rtol*||b||, atol) (KSPConvergedDefault).
//
// Two drivers share one arithmetic.  The graph solver runs one CTA per kernel with the
// operator (the Schur matvec) between them, reading G.xin and writing G.Av.  The cluster
// solver (k_gmres_cluster) runs a whole solve on an assembled dense operator across a
// cluster of kSlices CTAs, each owning one slice of the unknowns.  Every inner product,
// norm and Gram-Schmidt update is summed in the fixed order kernels.cuh states, which the
// graph kernels evaluate with one thread per sum and the cluster with lanes and shuffle
// trees; so both drivers produce identical iterates.
#include <cooperative_groups.h>

#include "kernels.cuh"

namespace ib {

namespace cg = cooperative_groups;

constexpr int kGmresThreads = 512;

// [lo, hi) of slice c of n unknowns
__device__ __forceinline__ int slice_size(int n) { return (n + kSlices - 1) / kSlices; }
__device__ __forceinline__ void slice_range(int n, int c, int* lo, int* hi) {
  int ns = slice_size(n);
  *lo = min(n, c * ns);
  *hi = min(n, *lo + ns);
}

static_assert(kSlices == 8, "the pairwise trees below are written for 8 slices");

// The fixed summation orders, one thread per sum (the cluster solver's lane forms match).
__device__ __forceinline__ double slice_dot_seq(const double* __restrict__ a, const double* __restrict__ b, int lo,
                                                int hi) {
  const int n = hi - lo, LP = slice_blocks_p2(n);
  // the pairwise tree over the LP block sums, streamed: merge equal-sized subtrees
  double st[32];
  int sz[32], top = 0;
  for (int k = 0; k < LP; ++k) {
    double p[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int i = lo + 4 * k + t;
      p[t] = i < hi ? a[i] * b[i] : 0.0;
    }
    double v = (p[0] + p[1]) + (p[2] + p[3]);
    int w = 1;
    while (top > 0 && sz[top - 1] == w) {
      v = st[top - 1] + v;
      w *= 2;
      --top;
    }
    st[top] = v;
    sz[top] = w;
    ++top;
  }
  return st[0];
}
__device__ __forceinline__ double tree8_seq(const double* p) {
  return ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
}
// Row i of w = Av - sum_{j<=it} h_j V_j (V with row pitch ld).
__device__ __forceinline__ double cgs_row_seq(double av, const double* __restrict__ h, const double* __restrict__ V,
                                              size_t ld, int i, int it) {
  double p[8];
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    double t = g == 0 ? av : 0.0;
    for (int j = g; j <= it; j += 8) t = fma(-h[j], V[(size_t)j * ld + i], t);
    p[g] = t;
  }
  return tree8_seq(p);
}

// Happy breakdown (KSPGMRESUpdateHessenberg): tt < min(|tt/g|, haptol = 1e-30).  The bound
// never exceeds haptol, so the quotient is formed only when tt itself is below it.
__device__ __forceinline__ bool happy_breakdown(double tt, double g) {
  if (!(tt < 1.0e-30)) return false;
  double hapbnd = fabs(tt / g);
  if (hapbnd > 1.0e-30) hapbnd = 1.0e-30;
  return tt < hapbnd;
}

// Norm of a new Krylov vector from its squared norm s: tt and the scale 1/tt applied to it
// (rsqrt and a product: a square root and a division cost about 600 cycles each here).
__device__ __forceinline__ void norm_and_scale(double s, double* tt, double* inv) {
  if (s > 0.0) {
    const double r = rsqrt(s);
    *inv = r;
    *tt = s * r;
  } else {
    *tt = sqrt(s);
    *inv = 0.0;
  }
}

// Givens update of Arnoldi step `it` (KSPGMRESUpdateHessenberg): the new Hessenberg column is
// h[0..it], tt; the previous rotations are applied with the rotated value carried in a
// register (one dependent FMA per rotation), then the new rotation (from rsqrt of c^2 + sq, sq the
// squared norm that tt is the root of), the rotated residual g and the convergence reason.  Writes H
// column `it` (ld = restart+1).  For restarts that a warp cannot hold; givens_finish_warp otherwise.
__device__ void givens_step(double* __restrict__ col, const double* __restrict__ h, double tt, double sq, int it,
                            double* __restrict__ cs, double* __restrict__ sn, double* __restrict__ g, double prev_res,
                            double ttol, double* res_out, int* reason_out) {
  const bool hapend = happy_breakdown(tt, g[it]);
  double c = h[0];
  for (int j = 0; j < it; ++j) {
    const double nxt = h[j + 1];
    const double cj = cs[j], sj = sn[j];
    col[j] = fma(sj, nxt, cj * c);
    c = fma(-sj, c, cj * nxt);
  }
  col[it + 1] = tt;
  double res;
  int reason = 0;
  if (!hapend) {
    const double r2 = fma(c, c, sq);
    if (r2 == 0.0) {
      reason = -9;  // KSP_DIVERGED_NULL
      res = prev_res;
      col[it] = c;
    } else {
      const double rn = rsqrt(r2);
      const double ci = c * rn, si = tt * rn;
      cs[it] = ci;
      sn[it] = si;
      g[it + 1] = -(si * g[it]);
      g[it] = ci * g[it];
      col[it] = fma(si, tt, ci * c);
      res = fabs(g[it + 1]);
    }
  } else {
    col[it] = c;
    res = 0.0;
  }
  if (reason == 0) {
    if (res <= ttol) reason = 2;
    else if (hapend) reason = -3;
  }
  *res_out = res;
  *reason_out = reason;
}

// The previous rotations applied to the new Hessenberg column h[0..it], on one whole warp (it < 32).
// Rotation j maps the carried value c to -sn_j c + cs_j h_{j+1}; lane j holds that affine map and the
// maps are composed by a parallel prefix (5 levels at most; one dependent FMA per rotation took 64
// cycles each, longer than the rest of the step once the cycle was ten vectors long).  Returns the
// value after all of them; *colv is entry `lane` of the rotated column (lane < it).
__device__ __forceinline__ double givens_chain_warp(const double* h, const double* cs, const double* sn, int it,
                                                    double* colv) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool mine = lane < it;
  const double csj = mine ? cs[lane] : 0.0, snj = mine ? sn[lane] : 0.0;
  const double hj1 = mine ? h[lane + 1] : 0.0, h0 = h[0];
  double A = -snj, B = csj * hj1;
  if (lane == 0) {   // the first map at its argument: a constant
    B = fma(A, h0, B);
    A = 0.0;
  }
  for (int d = 1; d < it; d <<= 1) {
    const double Ap = __shfl_up_sync(full, A, d), Bp = __shfl_up_sync(full, B, d);
    if (lane >= d) {
      B = fma(A, Bp, B);
      A = A * Ap;
    }
  }
  const double before = __shfl_up_sync(full, B, 1);   // the value before rotation `lane`
  *colv = fma(snj, hj1, csj * (lane == 0 ? h0 : before));
  return it > 0 ? __shfl_sync(full, B, it - 1) : h0;
}

// The rest of step `it` from the chain's value c, tt and rn = rsqrt(r2), r2 = c^2 + tt^2: givens_step's.
__device__ __forceinline__ void givens_finish_warp(double* col, double c, double colv, double r2, double rn, double tt,
                                                   int it, double* cs, double* sn, double* g, double prev_res,
                                                   double ttol, double* res_out, int* reason_out) {
  const int lane = threadIdx.x & 31;
  const double gi = g[it];   // read by every lane before lane 0 rewrites it
  if (lane < it) col[lane] = colv;
  const bool hapend = happy_breakdown(tt, gi);
  const double ci = c * rn, si = tt * rn;
  __syncwarp();
  if (lane == 0) {
    col[it + 1] = tt;
    double res;
    int reason = 0;
    if (!hapend) {
      if (r2 == 0.0) {
        reason = -9;  // KSP_DIVERGED_NULL
        res = prev_res;
        col[it] = c;
      } else {
        cs[it] = ci;
        sn[it] = si;
        g[it + 1] = -(si * gi);
        g[it] = ci * gi;
        col[it] = fma(si, tt, ci * c);
        res = fabs(g[it + 1]);
      }
    } else {
      col[it] = c;
      res = 0.0;
    }
    if (reason == 0) {
      if (res <= ttol) reason = 2;
      else if (hapend) reason = -3;
    }
    *res_out = res;
    *reason_out = reason;
  }
  __syncwarp();
}

// KSPGMRESBuildSoln back substitution y[0..k] = R^-1 g (R the rotated Hessenberg, ld = R+1), on
// one whole warp: the pivot reciprocals at once, then a column sweep on the unscaled r_j, from which
// every r_l, l < j, loses (R_lj / R_jj) r_j on its own lane (the quotients stand beside the chain);
// y_j = r_j / R_jj as r_j * (1/R_jj).  rc: k+1 doubles.
__device__ void back_substitute(const double* __restrict__ H, int R, const double* __restrict__ g, int k,
                                double* __restrict__ y, double* __restrict__ rc) {
  const int lane = threadIdx.x & 31;
  auto HH = [&](int r, int c) { return H[(size_t)c * (R + 1) + r]; };
  for (int l = lane; l <= k; l += 32) {
    y[l] = g[l];
    rc[l] = __drcp_rn(HH(l, l));
  }
  __syncwarp();
  for (int j = k; j >= 0; --j) {
    const double rj = y[j], rcj = rc[j];
    __syncwarp();
    for (int l = lane; l < j; l += 32) y[l] = fma(-(HH(l, j) * rcj), rj, y[l]);
    if (lane == 0) y[j] = rj * rcj;
    __syncwarp();
  }
}

__global__ void k_gmres_init(GmresDev G) {
  IB_GRID_DEP_WAIT();
  if (threadIdx.x == 0) {
    G.ist[0] = 0; G.ist[1] = 0; G.ist[2] = 0; G.ist[3] = 0; G.ist[4] = 0;
  }
}

// Cycle start: r = b - A x (A x in G.Av), V0 = r/||r||, tolerance on the first cycle.
__global__ void k_gmres_start(GmresDev G, const double* __restrict__ b, const double* __restrict__ x, double rtol,
                              double atol, int max_it, cudaGraphConditionalHandle h_inner, int use_cond) {
  IB_GRID_DEP_WAIT();
  __shared__ double part[2 * kSlices];
  __shared__ double s_norm[2];
  const int nf = G.nf, tid = threadIdx.x;
  for (int i = tid; i < nf; i += blockDim.x) G.V[i] = b[i] - G.Av[i];
  __syncthreads();
  if (tid < 2 * kSlices) {
    int lo, hi;
    slice_range(nf, tid % kSlices, &lo, &hi);
    const double* v = tid < kSlices ? G.V : b;
    part[tid] = slice_dot_seq(v, v, lo, hi);
  }
  __syncthreads();
  if (tid == 0) {
    s_norm[0] = sqrt(tree8_seq(part));
    s_norm[1] = sqrt(tree8_seq(part + kSlices));
  }
  __syncthreads();
  const double rnorm = s_norm[0], bnorm = s_norm[1];
  const int its = G.ist[0];
  double ttol;
  if (its == 0) {
    double rnorm0 = bnorm != 0.0 ? bnorm : rnorm;
    ttol = fmax(rtol * rnorm0, atol);
  } else {
    ttol = G.scal[0];
  }
  const double inv = rnorm != 0.0 ? 1.0 / rnorm : 0.0;
  for (int i = tid; i < nf; i += blockDim.x) {
    double v = rnorm != 0.0 ? G.V[i] * inv : G.V[i];
    G.V[i] = v;
    G.xin[i] = v;
  }
  if (tid == 0) {
    G.scal[0] = ttol;
    G.scal[1] = rnorm;
    G.scal[2] = bnorm;
    G.scal[3] = rnorm;
    G.scal[4] = 1.0;   // xin is V0 itself
    G.g[0] = rnorm;
    G.ist[2] = 0;
    int reason = 0;
    if (rnorm == 0.0) reason = 2;                 // KSP_CONVERGED_ATOL (zero residual)
    else if (rnorm <= ttol) reason = 3;           // converged at the initial residual
    else if (its >= max_it) reason = -3;
    G.ist[1] = reason;
    G.ist[3] = reason == 0 ? 1 : 0;
    G.ist[4] += 1;  // restart cycles
    if (use_cond) cudaGraphSetConditional(h_inner, reason == 0 ? 1u : 0u);
  }
}

// One Arnoldi step on w = A V[it] (scal[4] G.Av: the operator is applied to the vector before its
// normalisation, and its output scaled): classical Gram-Schmidt (all projections against the
// unmodified w), normalisation, Givens update.
__global__ void k_gmres_arnoldi(GmresDev G, int max_it, cudaGraphConditionalHandle h_inner, int use_cond) {
  IB_GRID_DEP_WAIT();
  __shared__ double part[64 * kSlices];
  __shared__ double h[64];
  __shared__ double s_tt[3];
  if (G.ist[3] == 0) {
    if (use_cond && threadIdx.x == 0) cudaGraphSetConditional(h_inner, 0u);
    return;
  }
  const int nf = G.nf, R = G.restart, tid = threadIdx.x;
  const int it = G.ist[2];
  double* w = G.V + (size_t)(it + 1) * nf;
  double* Av = G.Av;
  const double scale = G.scal[4];
  for (int i = tid; i < nf; i += blockDim.x) Av[i] = Av[i] * scale;
  __syncthreads();
  // projections: a partial per (j, slice), then the slices in order
  for (int q = tid; q < (it + 1) * kSlices; q += blockDim.x) {
    const int j = q / kSlices, c = q % kSlices;
    int lo, hi;
    slice_range(nf, c, &lo, &hi);
    part[q] = slice_dot_seq(Av, G.V + (size_t)j * nf, lo, hi);
  }
  __syncthreads();
  if (tid <= it) h[tid] = tree8_seq(part + tid * kSlices);
  __syncthreads();
  for (int i = tid; i < nf; i += blockDim.x) w[i] = cgs_row_seq(Av[i], h, G.V, nf, i, it);
  __syncthreads();
  if (tid < kSlices) {
    int lo, hi;
    slice_range(nf, tid, &lo, &hi);
    part[tid] = slice_dot_seq(w, w, lo, hi);
  }
  __syncthreads();
  if (tid == 0) {
    s_tt[2] = tree8_seq(part);
    norm_and_scale(s_tt[2], &s_tt[0], &s_tt[1]);
  }
  __syncthreads();
  const double tt = s_tt[0];
  const double inv = s_tt[1];
  const double sfac = tt != 0.0 ? inv : 1.0;
  for (int i = tid; i < nf; i += blockDim.x) {
    const double v = w[i];
    G.xin[i] = v;
    w[i] = v * sfac;
  }
  if (tid >= 32) return;
  const double sq = s_tt[2], prev_res = G.scal[1], ttol = G.scal[0];
  double* col = G.H + (size_t)it * (R + 1);
  double res = 0.0;
  int reason = 0;
  if (R <= 32) {
    double colv;
    const double c = givens_chain_warp(h, G.cs, G.sn, it, &colv);
    const double r2 = fma(c, c, sq);
    givens_finish_warp(col, c, colv, r2, r2 != 0.0 ? rsqrt(r2) : 0.0, tt, it, G.cs, G.sn, G.g, prev_res, ttol, &res,
                       &reason);
  } else if (tid == 0) {
    givens_step(col, h, tt, sq, it, G.cs, G.sn, G.g, prev_res, ttol, &res, &reason);
  }
  if (tid == 0) {
    const int itn = it + 1;
    const int its = G.ist[0] + 1;
    G.ist[2] = itn;
    G.ist[0] = its;
    G.scal[1] = res;
    G.scal[4] = sfac;
    G.ist[1] = reason;
    const int active = (reason == 0 && itn < R && its < max_it) ? 1 : 0;
    G.ist[3] = active;
    if (use_cond) cudaGraphSetConditional(h_inner, (unsigned)active);
  }
}

// KSPGMRESBuildSoln: back substitution and x += V y.
__global__ void k_gmres_update(GmresDev G, double* __restrict__ x, int max_it, cudaGraphConditionalHandle h_outer,
                               int use_cond) {
  IB_GRID_DEP_WAIT();
  __shared__ double y[64], rc[64];
  const int nf = G.nf, R = G.restart;
  const int it = G.ist[2];
  if (threadIdx.x < 32 && it > 0) back_substitute(G.H, R, G.g, it - 1, y, rc);
  __syncthreads();
  if (it > 0) {
    for (int i = threadIdx.x; i < nf; i += blockDim.x) {
      double p[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        p[q] = 0.0;
        for (int j = q; j < it; j += 8) p[q] = fma(y[j], G.V[(size_t)j * nf + i], p[q]);
      }
      x[i] = x[i] + tree8_seq(p);
    }
  }
  if (threadIdx.x == 0) {
    G.ist[3] = 0;
    // the iteration cap reached inside a cycle ends the solve as KSP_DIVERGED_ITS
    if (G.ist[1] == 0 && G.ist[0] >= max_it) G.ist[1] = -3;
    if (use_cond) cudaGraphSetConditional(h_outer, G.ist[1] == 0 ? 1u : 0u);
  }
}

__global__ void k_copy(int n, const double* __restrict__ a, double* __restrict__ b) {
  IB_GRID_DEP_WAIT();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = a[i];
}

int launch_gmres_init(const GmresDev& G, cudaStream_t st) {
  count_launch();
  k_gmres_init<<<1, 32, 0, st>>>(G);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}
int launch_gmres_start(const GmresDev& G, const double* b, const double* x, double rtol, double atol, int max_it,
                       cudaStream_t st, cudaGraphConditionalHandle h, int use_cond) {
  count_launch();
  k_gmres_start<<<1, kGmresThreads, 0, st>>>(G, b, x, rtol, atol, max_it, h, use_cond);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}
int launch_gmres_arnoldi(const GmresDev& G, int max_it, cudaStream_t st, cudaGraphConditionalHandle h,
                         int use_cond) {
  count_launch();
  k_gmres_arnoldi<<<1, kGmresThreads, 0, st>>>(G, max_it, h, use_cond);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}
int launch_gmres_update(const GmresDev& G, double* x, int max_it, cudaStream_t st, cudaGraphConditionalHandle h,
                        int use_cond) {
  count_launch();
  k_gmres_update<<<1, kGmresThreads, 0, st>>>(G, x, max_it, h, use_cond);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}
int launch_copy(int n, const double* a, double* b, cudaStream_t st) {
  if (n <= 0) return IB_OK;
  count_launch();
  k_copy<<<cdiv(n, 256), 256, 0, st>>>(n, a, b);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

// ---------------------------------------------------------------- Cholesky
// Dense Cholesky of the upper triangle of A (row-major n x n: A[i*n+j], the
// reference factors the upper triangle, PETSc MATSOLVERELEMENTAL), producing the
// lower factor L in place of the lower triangle (L[i*n+j], j<=i).  One CTA,
// right-looking, column by column.
__global__ void k_cholesky(int n, double* A, int* err) {
  IB_GRID_DEP_WAIT();
  __shared__ double piv;
  for (int k = 0; k < n; ++k) {
    if (threadIdx.x == 0) {
      double d = A[(size_t)k * n + k];
      if (!(d > 0.0)) { atomicExch(err, IB_ERR_ARG); d = 1.0; }
      piv = sqrt(d);
      A[(size_t)k * n + k] = piv;
    }
    __syncthreads();
    // column k below the diagonal, read from the upper triangle (A[k][i], i>k)
    for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x) A[(size_t)i * n + k] = A[(size_t)k * n + i] / piv;
    __syncthreads();
    // trailing update of the upper triangle: A[r][c] -= L[r][k] L[c][k] for k<r<=c
    long long rem = (long long)(n - k - 1);
    for (long long t = threadIdx.x; t < rem * rem; t += blockDim.x) {
      int r = k + 1 + (int)(t / rem), c = k + 1 + (int)(t % rem);
      if (c < r) continue;
      A[(size_t)r * n + c] -= A[(size_t)r * n + k] * A[(size_t)c * n + k];
    }
    __syncthreads();
  }
}

// M's lower triangle from its upper one, and F = M (the factorisation reads the upper triangle alone).
__global__ void k_symmetrise(int n, double* M, double* __restrict__ F) {
  IB_GRID_DEP_WAIT();
  const int c = blockIdx.x * blockDim.x + threadIdx.x, r = blockIdx.y;
  if (c >= n) return;
  const double v = M[(size_t)min(r, c) * n + max(r, c)];
  if (c < r) M[(size_t)r * n + c] = v;
  F[(size_t)r * n + c] = v;
}

// Z = L^-1 for the Cholesky factor L (row-major, in F's lower triangle), one warp per column by forward
// substitution, into F's upper triangle, Z[r][c] at F[c][r] for r > c, and its diagonal into diag: no
// column reads what another writes.  Run once per factorisation, k_tri_mirror after it.
__global__ void __launch_bounds__(32) k_tri_inverse(int n, double* F, double* __restrict__ diag) {
  IB_GRID_DEP_WAIT();
  extern __shared__ double col[];   // n entries of the column
  const int j = blockIdx.x, lane = threadIdx.x;
  for (int i = j; i < n; ++i) {
    const double* row = F + (size_t)i * n;
    double a0 = 0.0, a1 = 0.0;
    int k = j + lane;
    for (; k + 32 < i; k += 64) {
      a0 = fma(row[k], col[k], a0);
      a1 = fma(row[k + 32], col[k + 32], a1);
    }
    if (k < i) a0 = fma(row[k], col[k], a0);
    double s = a0 + a1;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) col[i] = ((i == j ? 1.0 : 0.0) - s) / row[i];
    __syncwarp();
  }
  if (lane == 0) diag[j] = col[j];
  for (int i = j + 1 + lane; i < n; i += 32) F[(size_t)j * n + i] = col[i];
}

// F's lower triangle from its upper one and its diagonal from diag: both products of the solve read rows.
__global__ void k_tri_mirror(int n, double* F, const double* __restrict__ diag) {
  IB_GRID_DEP_WAIT();
  const int c = blockIdx.x * blockDim.x + threadIdx.x, r = blockIdx.y;
  if (c < r) F[(size_t)r * n + c] = F[(size_t)c * n + r];
  if (c == r) F[(size_t)r * n + r] = diag[r];
}

// y = L^-1 b (upper = 0) or y = L^-T b (upper = 1) from Z, added to y with `add`; a warp per row, four
// chains a lane.  What bounds it: latency, a few dependent FP64 operations of 64 cycles and the row's loads
// from L2.
constexpr int kTriRows = 4;   // rows (warps) per CTA
__global__ void __launch_bounds__(32 * kTriRows) k_tri_product(int n, const double* __restrict__ Z,
                                                               const double* __restrict__ b, double* __restrict__ y,
                                                               int upper, int add) {
  IB_GRID_DEP_WAIT();
  const int r = blockIdx.x * kTriRows + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= n) return;
  const int c0 = upper ? r : 0, c1 = upper ? n : r + 1;
  const double* row = Z + (size_t)r * n;
  double a[4] = {0.0, 0.0, 0.0, 0.0};
  for (int c = c0 + lane; c < c1; c += 128) {
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c + 32 * u < c1) a[u] = fma(row[c + 32 * u], b[c + 32 * u], a[u]);
  }
  double s = (a[0] + a[1]) + (a[2] + a[3]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) y[r] = add ? y[r] + s : s;
}

// A sum in two parts: s and what its roundings left out (Knuth's two-sum).
struct Sum2 {
  double s, c;
  __device__ __forceinline__ void add(double v) {
    const double t = s + v, z = t - s;
    c += (s - (t - z)) + (v - z);
    s = t;
  }
};

// r = b - M x, each row a compensated product (Ogita, Rump and Oishi's Dot2) on one warp: as if formed in
// twice the working precision.  FP64 issue bounds it, ten operations a term.
__global__ void __launch_bounds__(32 * kTriRows) k_residual(int n, const double* __restrict__ M,
                                                            const double* __restrict__ b, const double* __restrict__ x,
                                                            double* __restrict__ r) {
  IB_GRID_DEP_WAIT();
  const int i = blockIdx.x * kTriRows + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= n) return;
  const double* row = M + (size_t)i * n;
  Sum2 a{lane == 0 ? b[i] : 0.0, 0.0};
#pragma unroll 4
  for (int c = lane; c < n; c += 32) {
    const double m = row[c], v = x[c], h = __dmul_rn(-m, v);   // no contraction into the sum
    a.c -= fma(m, v, h);
    a.add(h);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double s = __shfl_xor_sync(0xffffffffu, a.s, o), c = __shfl_xor_sync(0xffffffffu, a.c, o);
    a.add(s);
    a.c += c;
  }
  if (lane == 0) r[i] = a.s + a.c;
}

__global__ void k_copy_col(int n, const double* __restrict__ src, double* M, int col) {
  IB_GRID_DEP_WAIT();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) M[(size_t)i * n + col] = src[i];
}
__global__ void k_unit(int n, int i, double* e) {
  IB_GRID_DEP_WAIT();
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) e[t] = (t == i) ? 1.0 : 0.0;
}

int launch_cholesky(int n, double* A, int* d_err, cudaStream_t st) {
  count_launch();
  k_cholesky<<<1, 1024, 0, st>>>(n, A, d_err);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}
int launch_tri_inverse(int n, double* F, double* diag, cudaStream_t st) {
  const size_t smem = sizeof(double) * (size_t)n;
  IB_CUDA_CHECK(allow_dyn_smem(k_tri_inverse, smem));
  count_launches(2);
  k_tri_inverse<<<n, 32, smem, st>>>(n, F, diag);
  k_tri_mirror<<<dim3(cdiv(n, 256), n), 256, 0, st>>>(n, F, diag);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}
int launch_symmetrise(int n, double* M, double* F, cudaStream_t st) {
  count_launch();
  k_symmetrise<<<dim3(cdiv(n, 256), n), 256, 0, st>>>(n, M, F);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}
// x = M^-1 b: the two products with the inverse factor, then one step of refinement.  The substitutions by
// blocks of 32 that the products replaced ran on one CTA, 2 n / 32 dependent triangles: 304 us for the 314
// unknowns of the 157-point cylinder, against 7 us for the two products and 18 us for the five launches.  Products
// with an inverse alone are not backward stable: at 130 to 314 unknowns their residual was up to 10 times the
// substitutions', their error up to 20 times, by right-hand side.  The refinement, with the residual in two
// parts, leaves an error of the result's last place, below the substitutions'.
int launch_chol_solve(int n, const double* M, const double* Z, const double* b, double* y, double* r, double* x,
                      cudaStream_t st) {
  const int blocks = cdiv(n, kTriRows), threads = 32 * kTriRows;
  count_launches(5);
  k_tri_product<<<blocks, threads, 0, st>>>(n, Z, b, y, 0, 0);
  k_tri_product<<<blocks, threads, 0, st>>>(n, Z, y, x, 1, 0);
  k_residual<<<blocks, threads, 0, st>>>(n, M, b, x, r);
  k_tri_product<<<blocks, threads, 0, st>>>(n, Z, r, y, 0, 0);
  k_tri_product<<<blocks, threads, 0, st>>>(n, Z, y, x, 1, 1);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}
int launch_copy_col(int n, const double* src, double* M, int col, cudaStream_t st) {
  count_launch();
  k_copy_col<<<cdiv(n, 256), 256, 0, st>>>(n, src, M, col);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}
int launch_unit(int n, int i, double* e, cudaStream_t st) {
  count_launch();
  k_unit<<<cdiv(n, 256), 256, 0, st>>>(n, i, e);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

// ---------------------------------------------------------------- cluster dense solve
namespace {
// Shared-memory layout of one CTA of the cluster solver (doubles).
struct ClusterSmem {
  int nf, R, ns;
  size_t base() const {
    return (size_t)(R + 1) * ns + nf + 3 * (size_t)ns + (kSlices + 1) * (size_t)(R + 1) + (size_t)(R + 1) * R +
           4 * (size_t)(R + 1) + 8 + kSlices + 32;
  }
  size_t with_a() const { return base() + (size_t)ns * nf; }
};
}  // namespace

// Warps 0-3 run the dense product, the projections and the vector updates; warp 4 the norm and the
// Givens update meanwhile.  Warps 0-3 sit on an SM sub-partition each, and an FP64 instruction
// holds its sub-partition's FP64 pipe for the same time whatever its active lanes, so every
// sum below is spread over lanes (shuffle trees) rather than run down one thread.
constexpr int kClusterThreads = 160;
constexpr int kProdThreads = 128;

// back_substitute with a row per lane (k < 32): the same operations, r_l and R's entries in registers
__device__ __forceinline__ void back_substitute_lanes(const double* H, int R, const double* g, int k, double* y) {
  const int lane = threadIdx.x & 31;
  double r = 0.0, rc = 0.0;
  if (lane <= k) {
    r = g[lane];
    rc = __drcp_rn(H[(size_t)lane * (R + 1) + lane]);
  }
#pragma unroll 4
  for (int j = k; j > 0; --j) {
    const double hl = lane < j ? H[(size_t)j * (R + 1) + lane] : 0.0;
    const double q = hl * __shfl_sync(0xffffffffu, rc, j);
    const double rj = __shfl_sync(0xffffffffu, r, j);
    if (lane < j) r = fma(-q, rj, r);
  }
  if (lane <= k) y[lane] = r * rc;
  __syncwarp();
}

// One restarted GMRES solve on the assembled operator A (column-major, At[j*nf + r] = A[r][j])
// across a cluster of kSlices CTAs.  CTA c owns the rows and vector elements of slice c: its
// rows of A, its slice of every Krylov vector, of x and of b.  Per Arnoldi step:
//   A: warps 0-3 form the product of their rows with the new vector, not yet normalised (rows in
//      groups of S lanes), scale it and their slice of the vector by 1/norm and send every CTA
//      their partial projections; meanwhile warp 4 sums the norm, leaves the scale and finishes
//      the Givens update of the previous step, whose decision CTA 0 sends;   cluster barrier
//   B: w = A v - sum h_j v_j on the slice (8 lanes per row, each lane sending the element to one
//      CTA) and its partial norm, sent likewise; meanwhile warp 4 applies the earlier rotations to
//      the new Hessenberg column;                                            cluster barrier
// What bounds it is latency: about 45 dependent FP64 instructions a step, 64 cycles each, and two
// cluster barriers of 500.  Scaling after the product keeps the norm's sum and square root beside the
// product instead of before it; sending takes the place of reads of other CTAs' memory after the
// barriers, 500 cycles each.
// No thread waits on a flag: the only waits are the cluster and CTA barriers, which every
// thread of every CTA reaches the same number of times (the scale's: warp 4 arrives once and warps
// 0-3 wait once in each step with k > 0, k the same on all of them).
__global__ void __cluster_dims__(kSlices, 1, 1) __launch_bounds__(kClusterThreads)
    k_gmres_cluster(GmresDev G, const double* __restrict__ At, int a_in_smem, const double* __restrict__ b,
                    double* __restrict__ x, double rtol, double atol, int max_it) {
  IB_GRID_DEP_WAIT();
  const unsigned full = 0xffffffffu;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int nf = G.nf, R = G.restart;
  const int ns = slice_size(nf);
  int r0, r1;
  slice_range(nf, rank, &r0, &r1);
  const int nl = r1 - r0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  extern __shared__ double sm[];
  double* Vs = sm;                                  // (R+1) x ns
  double* vfull = Vs + (size_t)(R + 1) * ns;        // nf
  double* avs = vfull + nf;                         // ns
  double* xsl = avs + ns;                           // ns
  double* bsl = xsl + ns;                           // ns
  double* hp = bsl + ns;                            // kSlices x (R+1): every slice's partial projections
  double* h = hp + kSlices * (size_t)(R + 1);       // R+1
  double* H = h + (R + 1);                          // (R+1) x R
  double* cs = H + (size_t)(R + 1) * R;
  double* sn = cs + (R + 1);
  double* g = sn + (R + 1);
  double* yv = g + (R + 1);
  double* scal = yv + (R + 1);                      // [0],[1] partials (read remotely), [2] tt, [3] res,
                                                    // [4] 1/tt, [5] rnorm, [6] bnorm, [7] ttol
  double* npart = scal + 8;                         // kSlices: every slice's partial norm
  double* nblk = npart + kSlices;                   // 32: block partials of the slice's norm
  double* As = nblk + 32;                           // nl x nf row-major when a_in_smem
  __shared__ int s_reason;                          // CTA 0's decision
  auto remote = [&](double* p, int c) -> double* { return cl.map_shared_rank(p, c); };
  auto bar_prod = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(kProdThreads) : "memory"); };
  // the new vector's scale: warp 4 leaves it, warps 0-3 wait for it (each once a step after the first)
  auto bar_scale_put = [&]() { asm volatile("bar.arrive 2, %0;" ::"r"(kClusterThreads) : "memory"); };
  auto bar_scale_get = [&]() { asm volatile("bar.sync 2, %0;" ::"r"(kClusterThreads) : "memory"); };
  // slice partial of a.b in the fixed order: lane blk of an aligned group of LP lanes forms
  // block blk ((p0+p1)+(p2+p3) over rows 4blk..4blk+3), the group's xor tree the rest (valid
  // on every lane of the group); every lane of the warp calls it
  const int LP = slice_blocks_p2(nl);
  auto slice_dot_lanes = [&](const double* a, const double* bb, int blk, bool on) -> double {
    double p[4] = {0.0, 0.0, 0.0, 0.0};
    if (on)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int i = 4 * blk + t;
        if (i < nl) p[t] = a[i] * bb[i];
      }
    double v = (p[0] + p[1]) + (p[2] + p[3]);
    for (int off = 1; off < LP; off <<= 1) v += __shfl_xor_sync(full, v, off);
    return v;
  };
  // pairwise tree over an aligned group of 8 lanes (valid on all 8)
  auto tree8 = [&](double p) -> double {
    p += __shfl_xor_sync(full, p, 1);
    p += __shfl_xor_sync(full, p, 2);
    p += __shfl_xor_sync(full, p, 4);
    return p;
  };

  for (int i = tid; i < nl; i += blockDim.x) {
    xsl[i] = x[r0 + i];
    bsl[i] = b[r0 + i];
  }

  // avs = rows of A times vfull (warps 0-3): rows in groups of S lanes, one column segment
  // per lane, joined by seg_tree (k_dense_mv's layout and order)
  const int S = mv_segments(nf), gpw = 32 / S, cw = (nf + S - 1) / S;
  const int grp = lane / S, seg = lane - grp * S;
  // When the slice's rows take one pass of the four warps and a segment fits, each lane keeps
  // its segment of its row in registers for the whole solve (the same two chains, same order)
  constexpr int kRegSeg = 20;
  constexpr int kProdWarps = kProdThreads / 32;
  const bool a_in_regs = ns <= kProdWarps * gpw && cw <= kRegSeg;
  const int rl_r = warp * gpw + grp;
  const bool live_r = warp < kProdWarps && grp < gpw && rl_r < nl;
  const int j0_r = min(nf, seg * cw), len_r = live_r ? min(nf, j0_r + cw) - j0_r : 0;
  double areg[kRegSeg];
  if (a_in_regs) {
#pragma unroll
    for (int t = 0; t < kRegSeg; ++t) {
      areg[t] = 0.0;
      if (t < len_r) areg[t] = At[(size_t)(j0_r + t) * nf + r0 + rl_r];
    }
  } else if (a_in_smem) {
#pragma unroll 8
    for (int q = tid; q < nl * nf; q += kClusterThreads) {
      const int j = q / nl, rl = q - j * nl;
      As[rl * nf + j] = At[(size_t)j * nf + r0 + rl];
    }
  }
  __syncthreads();
  auto matvec = [&]() {
    if (a_in_regs) {
      double p = 0.0;
      if (live_r) {
        double e = 0.0, o = 0.0;
        const double* v = vfull + j0_r;
#pragma unroll
        for (int t = 0; t < kRegSeg; t += 2) {
          if (t >= cw) break;   // the same for every lane: no instructions for segments shorter than kRegSeg
          if (t < len_r) e = fma(areg[t], v[t], e);
          if (t + 1 < len_r) o = fma(areg[t + 1], v[t + 1], o);
        }
        p = e + o;
      }
      p = seg_tree(p, seg, S);
      if (live_r && seg == 0) avs[rl_r] = p;
      return;
    }
    for (int rb = 0; rb < nl; rb += kProdWarps * gpw) {
      const int rl = rb + warp * gpw + grp;
      const bool live = grp < gpw && rl < nl;
      double p = 0.0;
      if (live) {
        const int j0 = min(nf, seg * cw), j1 = min(nf, j0 + cw);
        if (a_in_smem) {
          const double* Ar = As + (size_t)rl * nf;
              p = seg_dot(j0, j1, [&](int j, double acc) { return fma(Ar[j], vfull[j], acc); });
        } else {
          p = seg_dot(j0, j1, [&](int j, double acc) { return fma(At[(size_t)j * nf + r0 + rl], vfull[j], acc); });
        }
      }
      p = seg_tree(p, seg, S);
      if (live && seg == 0) avs[rl] = p;
    }
  };
  auto gather = [&](double* src, int stride_slot) {   // vfull[i] = slot of the owner's slice
    for (int i = tid; i < nf; i += blockDim.x) {
      const int c = i / ns;
      vfull[i] = remote(src + (size_t)stride_slot * ns, c)[i - c * ns];
    }
  };

  int its = 0, cycles = 0, reason = 0, k = 0;
  double ttol = 0.0;
  for (;;) {
    // ---- cycle start (k_gmres_start): r = b - A x, V0 = r/||r||
    cl.sync();                                    // every x slice is final
    gather(xsl, 0);
    __syncthreads();
    if (warp < kProdWarps) matvec();
    __syncthreads();
    for (int i = tid; i < nl; i += blockDim.x) Vs[i] = bsl[i] - avs[i];
    __syncthreads();
    if (warp == 0) {   // lanes 0-15: ||r||^2 partial, lanes 16-31: ||b||^2 partial
      const double* v = lane < 16 ? Vs : bsl;
      const double t = slice_dot_lanes(v, v, lane & 15, (lane & 15) < LP);
      if (lane == 0) scal[0] = t;
      if (lane == 16) scal[1] = t;
    }
    cl.sync();
    if (warp == 0) {   // lanes 0-7: the slices' r partials, lanes 8-15: their b partials
      const double p = tree8(lane < 16 ? remote(scal, lane & 7)[lane >> 3] : 0.0);
      const double nrm = sqrt(p);
      const double rnorm = __shfl_sync(full, nrm, 0), bnorm = __shfl_sync(full, nrm, 8);
      if (lane == 0) {
        if (its == 0) {
          double rnorm0 = bnorm != 0.0 ? bnorm : rnorm;
          scal[7] = fmax(rtol * rnorm0, atol);
        }
        scal[5] = rnorm;
        scal[6] = bnorm;
        scal[3] = rnorm;
        g[0] = rnorm;
        int rs = 0;
        if (rnorm == 0.0) rs = 2;
        else if (rnorm <= scal[7]) rs = 3;
        else if (its >= max_it) rs = -3;
        s_reason = rs;
      }
    }
    __syncthreads();
    {
      const double rnorm = scal[5];
      const double inv = rnorm != 0.0 ? 1.0 / rnorm : 0.0;
      for (int i = tid; i < nl; i += blockDim.x) Vs[i] = rnorm != 0.0 ? Vs[i] * inv : Vs[i];
    }
    cycles += 1;
    cl.sync();                                    // V0 slices and CTA 0's decision are visible
    reason = *cl.map_shared_rank(&s_reason, 0);
    ttol = scal[7];
    if (reason != 0) break;
    gather(Vs, 0);
    __syncthreads();
    // ---- Arnoldi steps (k_gmres_arnoldi), the norm and the Givens update of step k-1 during step k
    k = 0;
    double gc = 0.0, gcol = 0.0;   // warp 4: the last column's value after its earlier rotations, its entries
    for (;;) {
      if (warp < kProdWarps) {
        matvec();
        if (k > 0) {
          bar_scale_get();   // scal[4]; and the raw product is complete
          const double sfac = scal[4];
          if (warp < 2)
            for (int i = tid; i < nl; i += 64) avs[i] = avs[i] * sfac;
          else
            for (int i = tid - 64; i < nl; i += 64) Vs[(size_t)k * ns + i] = vfull[r0 + i] * sfac;
        }
        bar_prod();
        for (int q0 = 0; q0 < LP * (k + 1); q0 += kProdThreads) {   // LP lanes per projection
          const int q = q0 + tid, j = q / LP, blk = q - j * LP;
          const bool on = j <= k;
          const double t = slice_dot_lanes(avs, Vs + (size_t)(on ? j : 0) * ns, blk, on);
          if (on)
            for (int c = blk; c < kSlices; c += LP) remote(hp, c)[rank * (R + 1) + j] = t;
        }
      } else if (k > 0) {
        // one reciprocal square root serves the norm (lane 0) and the new rotation (lane 1)
        const double sq = tree8(npart[lane & 7]);
        const double r2 = fma(gc, gc, sq);
        const double r = rsqrt(lane == 0 ? sq : r2);
        double inv = __shfl_sync(full, r, 0);
        const double r1 = __shfl_sync(full, r, 1), rn = r2 != 0.0 ? r1 : 0.0;
        double tt = sq * inv;
        if (!(sq > 0.0)) {
          tt = sqrt(sq);
          inv = 0.0;
        }
        if (lane == 0) scal[4] = tt != 0.0 ? inv : 1.0;
        __syncwarp();
        bar_scale_put();
        double res = 0.0;
        int rs = 0;
        givens_finish_warp(H + (size_t)(k - 1) * (R + 1), gc, gcol, r2, rn, tt, k - 1, cs, sn, g, scal[3], ttol, &res,
                           &rs);
        if (lane == 0) scal[3] = res;
        rs = __shfl_sync(full, rs, 0);
        if (rank == 0 && lane < kSlices) *cl.map_shared_rank(&s_reason, lane) = rs;
      }
      cl.sync();                                  // partial projections; Givens of step k-1
      if (k > 0) {
        reason = s_reason;
        if (reason != 0 || k >= R || its >= max_it) break;
      }
      for (int q0 = 0; q0 < kSlices * (k + 1); q0 += kClusterThreads) {   // 8 lanes (slices) per projection
        const int q = q0 + tid, j = q >> 3;
        const double p = tree8(j <= k ? hp[(q & 7) * (R + 1) + j] : 0.0);
        if (j <= k && (q & 7) == 0) h[j] = p;
      }
      __syncthreads();
      if (warp < kProdWarps) {
        // w = avs - sum_j h_j V_j on the slice (8 lanes, one chain each, per row), lane c's copy to
        // CTA c; the lanes 0, 8, 16, 24 of a warp hold 4 consecutive rows: one block of the norm partial
        const int npass = (8 * nl + kProdThreads - 1) / kProdThreads;
        for (int q0 = 0; q0 < 8 * nl; q0 += kProdThreads) {
          const int q = q0 + tid, i = q >> 3, gq = q & 7;
          double p = 0.0;
          if (i < nl) {
            p = gq == 0 ? avs[i] : 0.0;
            for (int j = gq; j <= k; j += 8) p = fma(-h[j], Vs[(size_t)j * ns + i], p);
          }
          p = tree8(p);
          if (i < nl) remote(vfull, gq)[r0 + i] = p;
          double sq = i < nl ? p * p : 0.0;
          sq += __shfl_xor_sync(full, sq, 8);
          sq += __shfl_xor_sync(full, sq, 16);
          if (lane == 0) nblk[q >> 5] = sq;
        }
        bar_prod();
        if (warp == 0) {
          double v = lane < LP && lane < kProdWarps * npass ? nblk[lane] : 0.0;
          for (int off = 1; off < LP; off <<= 1) v += __shfl_xor_sync(full, v, off);
          v = __shfl_sync(full, v, 0);
          if (lane < kSlices) remote(npart, lane)[rank] = v;
        }
      } else {
        gc = givens_chain_warp(h, cs, sn, k, &gcol);
      }
      cl.sync();                                  // the new vector and its partial norms
      its += 1;
      k += 1;
    }
    // ---- KSPGMRESBuildSoln (k_gmres_update): back substitution and x += V y on the slice
    if (warp == 0 && k > 0) back_substitute_lanes(H, R, g, k - 1, yv);
    __syncthreads();
    if (k > 0 && warp < kProdWarps)
      for (int q0 = 0; q0 < 8 * nl; q0 += kProdThreads) {   // 8 lanes, one chain each, per row
        const int q = q0 + tid, i = q >> 3, gq = q & 7;
        double u = 0.0;
        if (i < nl)
          for (int j = gq; j < k; j += 8) u = fma(yv[j], Vs[(size_t)j * ns + i], u);
        u = tree8(u);
        if (i < nl && gq == 0) xsl[i] = xsl[i] + u;
      }
    __syncthreads();
    if (reason != 0 || its >= max_it) break;
  }
  for (int i = tid; i < nl; i += blockDim.x) x[r0 + i] = xsl[i];
  if (rank == 0 && tid == 0) {
    G.ist[0] = its;
    G.ist[1] = reason == 0 && its >= max_it ? -3 : reason;   // KSP_DIVERGED_ITS
    G.ist[2] = k;
    G.ist[3] = 0;
    G.ist[4] = cycles;
    G.scal[0] = ttol;
    G.scal[1] = scal[3];
  }
  cl.sync();                                      // no CTA exits while others read its memory
}

int launch_gmres_fused(const GmresDev& G, FusedPlan* plan, const double* At, const double* b, double* x, double rtol,
                       double atol, int max_it, cudaStream_t st) {
  if (plan->state < 0) {
    plan->state = 0;
    if (G.nf <= 0 || G.restart > 32) return IB_ERR_ARG;   // the Givens warp holds a rotation per lane
    ClusterSmem cs{G.nf, G.restart, (G.nf + kSlices - 1) / kSlices};
    if (slice_blocks_p2(cs.ns) > 16) return IB_ERR_ARG;   // a slice's norm blocks on 16 lanes
    const int threads = kClusterThreads;
    int dev = 0, optin = 0;
    IB_CUDA_CHECK(cudaGetDevice(&dev));
    IB_CUDA_CHECK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const size_t limit = (size_t)optin - 1024;
    int a_in = 1;
    size_t bytes = 8 * cs.with_a();
    if (bytes > limit) {
      a_in = 0;
      bytes = 8 * cs.base();
      if (bytes > limit) return IB_ERR_ARG;
    }
    IB_CUDA_CHECK(allow_dyn_smem(k_gmres_cluster, bytes));
    // the cluster must fit on the device as launched
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSlices);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, k_gmres_cluster, &cfg) != cudaSuccess || nclusters < 1) {
      cudaGetLastError();
      return IB_ERR_ARG;
    }
    plan->threads = threads;
    plan->a_in = a_in;
    plan->bytes = bytes;
    plan->state = 1;
  }
  if (plan->state != 1) return IB_ERR_ARG;
  count_launch();
  k_gmres_cluster<<<kSlices, plan->threads, plan->bytes, st>>>(G, At, plan->a_in, b, x, rtol, atol, max_it);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

}  // namespace ib
