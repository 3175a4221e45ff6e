// Chunked per-mode tridiagonal solver (see tri.cuh).
#include <algorithm>
#include <cmath>
#include <thread>
#include <vector>

#include "tri.cuh"

namespace ib {

// The chunk lengths with a register-resident kernel (k_tri_reg), and those of them that also take a
// shorter last chunk.
#define IB_TRI_EVEN(X) X(1) X(2) X(4) X(5) X(6) X(8) X(9) X(12) X(14) X(24) X(29)
#define IB_TRI_BOTH(X) X(3) X(7) X(11) X(15) X(19) X(23) X(31) X(39) X(63)
constexpr int kTriMaxM = 31;   // most interfaces (C-1) of the register-resident kernel

static bool tri_reg_length(int s, bool tail) {
  switch (s) {
#define IB_CASE(SS) case SS:
    IB_TRI_BOTH(IB_CASE) return true;
    IB_TRI_EVEN(IB_CASE) return !tail;
#undef IB_CASE
    default: return false;
  }
}

// Every FP64 warp instruction holds its SM sub-partition's FP64 pipe for the same time whatever its
// active lanes, so the cost of one solve is the FP64 instructions of one chunk thread (about 5 per
// chunk row and one per interface) times the warps a sub-partition runs, minimised over the launch
// shapes (Mb modes x C chunks per CTA, Mb a power of two) the tuner can pick.
static long long tri_cost(int s, int C, int nx) {
  constexpr int kSMs = 152;   // GB300: 4 sub-partitions each
  const long long per = 5LL * s + C;
  long long best = -1;
  for (int Mb = 1; Mb <= 32; Mb *= 2) {
    if (Mb * C > 1024) break;
    const long long wpc = (Mb * C + 31) / 32;                 // warps per CTA
    const long long ncta = (nx + Mb - 1) / Mb;
    const long long mult = ((ncta + kSMs - 1) / kSMs * wpc + 3) / 4;   // warps per sub-partition
    if (best < 0 || per * mult < best) best = per * mult;
  }
  return best;
}

TriShape tri_chunking_even(int n, int nx) {
  // the chunk period d = s+1 divides n, at most 32 chunks
  long long best = -1;
  int bestd = n;
  for (int d = 2; d <= n; ++d) {
    if (n % d || n / d > 32) continue;
    const long long cost = tri_cost(d - 1, n / d, nx);
    if (best < 0 || cost < best || (cost == best && d > bestd)) { best = cost; bestd = d; }
  }
  return TriShape{bestd - 1, n / bestd, bestd - 1};
}

// Of the lengths with a register kernel, the cheapest; a shorter last chunk counts a tenth more (its
// rows are predicated), and 63 rows, which spill, are taken only where no shorter chunk will do.  The
// shared-memory kernel took 37 us for 999 modes of 539 rows in its cheapest equal chunks (15 of 35) and
// 160 us for 800 modes of 400 rows, whose period 401 is prime (one chunk); in 14 chunks of 39 the first
// takes 19 us, and the second in 13 of 31 12 us.  It remains for more than 32 x 64 rows.
TriShape tri_chunking(int ny, int nx, size_t max_doubles) {
  TriShape best;
  double bestc = -1.0;
  for (int s = 1; s <= 63; ++s) {
    const int C = (ny + 1 + s) / (s + 1), r = ny - (C - 1) * (s + 1);
    if (C - 1 > kTriMaxM || r < 1 || r > s || !tri_reg_length(s, r < s) || (s == 63 && bestc >= 0)) continue;
    const TriShape t{s, C, r};
    if (max_doubles && tri_table_doubles(nx, t) > max_doubles) continue;
    const double cost = (double)tri_cost(s, C, nx) * (r < s ? 1.1 : 1.0);
    if (bestc < 0 || cost <= bestc) { bestc = cost; best = t; }
  }
  return bestc < 0 ? tri_chunking_even(ny + 1, nx) : best;
}

size_t tri_table_doubles(int nx, const TriShape& t) {
  const size_t m = t.C > 1 ? (size_t)(t.C - 1) : 1;
  return (size_t)nx * ((t.r < t.s ? 4 : 3) * (size_t)t.s + m * m);
}

int tri_build(TriOp* op, int nx, int ny, const TriShape& t, const double* shift, double sigma, double* dev) {
  const int s = t.s, C = t.C, r = t.r;
  if ((C - 1) * (s + 1) + r != ny) return IB_ERR_ARG;
  op->nx = nx; op->ny = ny; op->s = s; op->C = C; op->r = r; op->sigma = sigma;
  const int m = C > 1 ? C - 1 : 1;
  const size_t S = (size_t)s * nx, R = (size_t)m * m * nx;
  std::vector<double> tab((r < s ? 4 : 3) * S + R, 0.0);
  double* gT = tab.data() + 3 * S + R;
  double* inv = tab.data();
  double* sinv = inv + S;
  double* gL = inv + 2 * S;
  double* rinv = inv + 3 * S;
  // the modes are independent: they are split over host threads (long double arithmetic is
  // software-emulated on some hosts and costs milliseconds per operator otherwise)
  auto modes = [&](int k0, int k1) {
  std::vector<long double> beta(s), d(s), g(s), gt(r), bp(m), z(m), x(m);
  for (int k = k0; k < k1; ++k) {
    long double a = 2.0L + (long double)shift[k];
    beta[0] = a;
    for (int j = 1; j < s; ++j) beta[j] = a - 1.0L / beta[j - 1];
    for (int j = 0; j < s; ++j) {
      inv[(size_t)j * nx + k] = (double)(1.0L / beta[j]);
      sinv[(size_t)j * nx + k] = (double)((long double)sigma / beta[j]);
    }
    // response to a unit value just left of the chunk: T_s g = e_0
    d[0] = 1.0L / beta[0];
    for (int j = 1; j < s; ++j) d[j] = d[j - 1] / beta[j];
    g[s - 1] = d[s - 1];
    for (int j = s - 2; j >= 0; --j) g[j] = d[j] + g[j + 1] / beta[j];
    for (int j = 0; j < s; ++j) gL[(size_t)j * nx + k] = (double)g[j];
    gt[r - 1] = d[r - 1];
    for (int j = r - 2; j >= 0; --j) gt[j] = d[j] + gt[j + 1] / beta[j];
    if (r < s)
      for (int j = 0; j < r; ++j) gT[(size_t)j * nx + k] = (double)gt[j];
    if (C < 2) continue;
    // interface system tridiag(-B, A, -B) of size m = C-1 (the last diagonal entry with the last
    // chunk's response), tabulated as its dense inverse (one Thomas solve per unit vector, in
    // extended precision)
    const long double A = a - 2.0L * g[0], B = g[s - 1], AT = a - g[0] - gt[0];
    bp[0] = m == 1 ? AT : A;
    for (int c = 1; c < m; ++c) bp[c] = (c == m - 1 ? AT : A) - B * B / bp[c - 1];
    for (int j = 0; j < m; ++j) {
      for (int c = 0; c < m; ++c) z[c] = ((c == j ? 1.0L : 0.0L) + (c > 0 ? B * z[c - 1] : 0.0L)) / bp[c];
      x[m - 1] = z[m - 1];
      for (int c = m - 2; c >= 0; --c) x[c] = z[c] + (B / bp[c]) * x[c + 1];
      for (int c = 0; c < m; ++c) rinv[((size_t)c * m + j) * nx + k] = (double)x[c];
    }
  }
  };
  const int nth = std::max(1, std::min(16, (int)std::thread::hardware_concurrency()));
  if (nth == 1 || nx < 64) {
    modes(0, nx);
  } else {
    std::vector<std::thread> th;
    for (int t = 0; t < nth; ++t) th.emplace_back(modes, (int)((long long)nx * t / nth), (int)((long long)nx * (t + 1) / nth));
    for (auto& x : th) x.join();
  }
  op->inv = dev;
  op->sinv = dev + S;
  op->gL = dev + 2 * S;
  op->rinv = dev + 3 * S;
  op->gT = r < s ? dev + 3 * S + R : nullptr;
  IB_CUDA_CHECK(cudaMemcpy(dev, tab.data(), 8 * tab.size(), cudaMemcpyHostToDevice));
  return IB_OK;
}

// Row r of mode k's right-hand side with the boundary terms (TriBc).
__device__ __forceinline__ double tri_rhs(const TriBc& b, int ny, int nx, int r, int k, double f) {
  double v = b.post_scale == 1.0 ? f : b.post_scale * f;
  if (b.sd) {
    v = fma(__ldg(b.sk2 + k), b.sd[(k & 1) * ny + r], v);
    if (r == 0) v += b.edge[k];
    if (r == ny - 1) v += b.edge[nx + k];
  }
  return v;
}

// One CTA: Mb consecutive modes x C chunks (thread t: mode t % Mb, chunk t / Mb, so a warp
// holds 32/Mb chunks of Mb modes).  The CTA's ny x Mb tile and its factor tables are staged
// in shared memory, so the sequential recurrences run on shared-memory latency.  The
// interface values come from the tabulated inverse of the interface system: every chunk
// thread forms one of them with C-1 independent products, instead of one thread per mode
// running a 2(C-1)-step recurrence while the rest of its warp idles (an FP64 warp
// instruction costs the same issue time whatever its active lanes).
__global__ void k_tri(TriOp op, const double* __restrict__ F, double* U, int ld, int Mb, TriBc bc) {
  IB_GRID_DEP_WAIT();
  extern __shared__ double sm[];
  const int C = op.C, s = op.s, d = s + 1, nx = op.nx, ny = op.ny;
  const int m = C > 1 ? C - 1 : 1;
  const int trows = 3 * s + (C > 1 ? m * m : 0);   // table rows staged: inv, sinv, gL, rinv
  double* tile = sm;                       // ny x Mb
  double* t_inv = tile + (size_t)ny * Mb;  // s x Mb
  double* t_sinv = t_inv + s * Mb;
  double* t_gL = t_sinv + s * Mb;
  double* t_r = t_gL + s * Mb;             // m*m x Mb
  double* pfirst = t_inv + (size_t)trows * Mb;  // C x Mb
  double* plast = pfirst + C * Mb;
  double* hv = plast + C * Mb;             // (C+1) x Mb: interface right-hand sides
  double* yv = hv + (C + 1) * Mb;          // (C+1) x Mb: interface values
  const int k0 = blockIdx.x * Mb;
  const int nthr = blockDim.x;
  // stage the tile (rows of F) and the tables (rows of op.inv.., contiguous with stride nx),
  // coalesced along modes, 8 loads in flight per thread: thread t owns mode column t % Mb
  // and rows t / Mb + i * (nthr / Mb)
  const int rstep = nthr / Mb;
  const int kl0 = threadIdx.x % Mb, r00 = threadIdx.x / Mb;
  const bool kin = k0 + kl0 < nx && r00 < rstep;
  {
    const double* src = F + k0 + kl0;
    const double* tsrc = op.inv + min(k0 + kl0, nx - 1);
    const int tot = ny + trows;
    for (int r = r00; r < tot; r += 8 * rstep) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        int rr = r + u * rstep;
        v[u] = 0.0;
        if (rr < ny) {
          if (kin) {
            double f = src[(size_t)rr * ld];
            if (bc.add2) f = f + bc.add2[(size_t)rr * ld + k0 + kl0];
            v[u] = tri_rhs(bc, ny, nx, rr, k0 + kl0, f);
          }
        }
        else if (rr < tot) v[u] = __ldg(tsrc + (size_t)(rr - ny) * nx);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        int rr = r + u * rstep;
        if (rr < tot && r00 < rstep) tile[rr * Mb + kl0] = v[u];
      }
    }
  }
  __syncthreads();
  const int t = threadIdx.x;
  const int kl = t % Mb, c = t / Mb;
  const bool active = c < C;
  // phase 1: chunk solves with zero ends; interface rows keep f until phase 2
  if (active) {
    double* col = tile + c * d * Mb + kl;
    const double* ti = t_inv + kl;
    const double* ts = t_sinv + kl;
    double dp = 0.0;
    for (int j = 0; j < s; ++j) {
      dp = fma(ti[j * Mb], dp, ts[j * Mb] * col[j * Mb]);
      col[j * Mb] = dp;
    }
    plast[c * Mb + kl] = dp;
    double u = dp;
    for (int j = s - 2; j >= 0; --j) {
      u = fma(ti[j * Mb], u, col[j * Mb]);
      col[j * Mb] = u;
    }
    pfirst[c * Mb + kl] = u;
  }
  __syncthreads();
  // phase 2a: right-hand side of interface c (between chunks c-1 and c)
  if (active && c >= 1)
    hv[c * Mb + kl] = fma(op.sigma, tile[(c * d - 1) * Mb + kl], plast[(c - 1) * Mb + kl] + pfirst[c * Mb + kl]);
  __syncthreads();
  // phase 2b: interface value c = row c-1 of the interface inverse times the right-hand sides
  if (active) {
    if (c >= 1) {
      const double* rr = t_r + (size_t)(c - 1) * m * Mb + kl;
      const double* hh = hv + Mb + kl;
      double y0 = 0.0, y1 = 0.0;
      int j = 0;
      for (; j + 1 < m; j += 2) {
        y0 = fma(rr[j * Mb], hh[j * Mb], y0);
        y1 = fma(rr[(j + 1) * Mb], hh[(j + 1) * Mb], y1);
      }
      if (j < m) y0 = fma(rr[j * Mb], hh[j * Mb], y0);
      yv[c * Mb + kl] = y0 + y1;
    } else {
      yv[kl] = 0.0;
      yv[C * Mb + kl] = 0.0;
    }
  }
  __syncthreads();
  // phase 3: add the interface responses; interface rows take the interface values
  if (active) {
    double* col = tile + c * d * Mb + kl;
    const double* tg = t_gL + kl;
    double yl = yv[c * Mb + kl], yr = yv[(c + 1) * Mb + kl];
    for (int j = 0; j < s; ++j) {
      double u = col[j * Mb];
      u = fma(yl, tg[j * Mb], u);
      u = fma(yr, tg[(s - 1 - j) * Mb], u);
      col[j * Mb] = u;
    }
    if (c >= 1) col[-Mb] = yl;
  }
  __syncthreads();
  if (kin) {
    double* dst = U + k0 + kl0;
    for (int r = r00; r < ny; r += rstep) dst[(size_t)r * ld] = tile[r * Mb + kl0];
  }
}

// The same solve with each thread's chunk in registers (S = op.s known at compile time): the
// chunk rows and the interface row above are loaded straight from F (all loads in flight at
// once), the tables (pivots and responses, shared by a mode's chunks, and each thread's row of the
// interface inverse) arrive in shared memory by asynchronous copies meanwhile, and the result is
// stored straight to U.  Same arithmetic as k_tri.  In place allowed: a thread writes only the
// rows it read, after the CTA's barriers.
// What bounds it: the FP64 pipe, 5 S + C - 1 instructions of 64 cycles a warp, and the latency of
// the loads.  128 registers a thread let every CTA be resident (1535 modes in 32 chunks: 384 CTAs of
// four warps in one wave; with the inverse's rows in registers, 246 a thread, they took two).
// Measured, before and after: 1535 modes of 1023 rows 37.2 and 31.5 us; 1599 of 799, 29.2 and 21.5; 999 of
// 539 (TAIL), 21.9 and 18.5; 799 of 399, 11.0 and 10.4.
// TAIL: the last chunk has op.r < S rows.
__device__ __forceinline__ void tri_copy8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

template <int S, bool TAIL>
__device__ __forceinline__ void tri_reg_body(const TriOp& op, const double* __restrict__ F, double* U, int ld, int Mb,
                                             const TriBc& bc, double* sm) {
  const int C = op.C, d = S + 1, nx = op.nx;
  const int m = C > 1 ? C - 1 : 1;
  double* t_inv = sm;                      // S x Mb
  double* t_sinv = t_inv + S * Mb;
  double* t_gL = t_sinv + S * Mb;
  double* pfirst = t_gL + S * Mb;          // C x Mb
  double* plast = pfirst + C * Mb;
  double* hv = plast + C * Mb;             // (C+1) x Mb
  double* yv = hv + (C + 1) * Mb;          // (C+1) x Mb
  double* t_r = yv + (C + 1) * Mb;         // m x C Mb: row c-1 of a mode's interface inverse, per thread
  double* t_gT = t_r + m * C * Mb;         // S x Mb (TAIL)
  const int k0 = blockIdx.x * Mb, nthr = blockDim.x;
  const int t = threadIdx.x, kl = t % Mb, c = t / Mb;
  const int k = min(k0 + kl, nx - 1);
  const int len = TAIL && c == C - 1 ? op.r : S;
  const bool chunk = c < C, store = chunk && k0 + kl < nx;
  const int r0 = c * d;
  // the tables are constant (built at creation): fetched before the wait for the previous
  // kernel, so that under a programmatic edge they arrive while it finishes
  for (int q = t; q < 3 * S * Mb; q += nthr) {
    const int row = q / Mb, kk = min(k0 + q - row * Mb, nx - 1);
    tri_copy8(t_inv + q, op.inv + (size_t)row * nx + kk);
    if (TAIL && row < S) tri_copy8(t_gT + q, op.gT + (size_t)row * nx + kk);
  }
  if (chunk && c >= 1) {
    const double* src = op.rinv + (size_t)(c - 1) * m * nx + k;
    for (int j = 0; j < m; ++j) tri_copy8(t_r + j * C * Mb + t, src + (size_t)j * nx);
  }
  asm volatile("cp.async.commit_group;\n");
  if (!bc.early) IB_GRID_DEP_WAIT();
  double f[S];
#pragma unroll
  for (int j = 0; j < S; ++j) f[j] = chunk && (!TAIL || j < len) ? F[(size_t)(r0 + j) * ld + k] : 0.0;
  double fi = (chunk && c >= 1) ? F[(size_t)(r0 - 1) * ld + k] : 0.0;
  if (chunk && bc.add2) {
#pragma unroll
    for (int j = 0; j < S; ++j)
      if (!TAIL || j < len) f[j] = f[j] + bc.add2[(size_t)(r0 + j) * ld + k];
    if (c >= 1) fi = fi + bc.add2[(size_t)(r0 - 1) * ld + k];
  }
  if (bc.early) IB_GRID_DEP_WAIT();
  if (chunk && (bc.sd || bc.post_scale != 1.0)) {
    // boundary terms (tri_rhs) on the chunk rows and the interface row above; row 0 is chunk
    // 0's first row and row ny-1 chunk C-1's last
    const double ps = bc.post_scale;
    if (bc.sd) {
      const double a = __ldg(bc.sk2 + k);
      const double* sdk = bc.sd + (k & 1) * op.ny;
#pragma unroll
      for (int j = 0; j < S; ++j)
        if (!TAIL || j < len) f[j] = fma(a, sdk[r0 + j], ps == 1.0 ? f[j] : ps * f[j]);
      if (c >= 1) fi = fma(a, sdk[r0 - 1], ps == 1.0 ? fi : ps * fi);
      if (c == 0) f[0] += bc.edge[k];
      if (!TAIL && c == C - 1) f[S - 1] += bc.edge[nx + k];
      if (TAIL && c == C - 1) {
        const double e = bc.edge[nx + k];
#pragma unroll
        for (int j = 0; j < S; ++j)
          if (j == len - 1) {
            f[j] += e;
            asm volatile("" : "+d"(f[j]));   // keeps the rows in registers (not one indexed store)
          }
      }
    } else {
#pragma unroll
      for (int j = 0; j < S; ++j) f[j] *= ps;
      fi *= ps;
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  // phase 1: chunk solve with zero ends (the products sigma/pivot * f are off the forward
  // recurrence, which takes one FMA per row)
  if (chunk) {
    double dp = 0.0;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      dp = fma(t_inv[j * Mb + kl], dp, t_sinv[j * Mb + kl] * f[j]);
      f[j] = dp;
    }
    plast[c * Mb + kl] = dp;
    double u = dp;
#pragma unroll
    for (int j = S - 2; j >= 0; --j) {
      u = !TAIL || j < len - 1 ? fma(t_inv[j * Mb + kl], u, f[j]) : f[j];
      f[j] = u;
    }
    pfirst[c * Mb + kl] = u;
  }
  __syncthreads();
  // phase 2a: right-hand side of interface c
  if (chunk && c >= 1) hv[c * Mb + kl] = fma(op.sigma, fi, plast[(c - 1) * Mb + kl] + pfirst[c * Mb + kl]);
  __syncthreads();
  // phase 2b: interface value c
  if (chunk) {
    if (c >= 1) {
      const double* hh = hv + Mb + kl;
      const double* rr = t_r + t;
      double y0 = 0.0, y1 = 0.0;
      int j = 0;
#pragma unroll 4
      for (; j + 1 < m; j += 2) {
        y0 = fma(rr[j * C * Mb], hh[j * Mb], y0);
        y1 = fma(rr[(j + 1) * C * Mb], hh[(j + 1) * Mb], y1);
      }
      if (j < m) y0 = fma(rr[j * C * Mb], hh[j * Mb], y0);
      yv[c * Mb + kl] = y0 + y1;
    } else {
      yv[kl] = 0.0;
      yv[C * Mb + kl] = 0.0;
    }
  }
  __syncthreads();
  // phase 3: interface responses, straight to U
  if (store) {
    const double yl = yv[c * Mb + kl], yr = yv[(c + 1) * Mb + kl];
    double* dst = U + k;
    const double* tg = TAIL && c == C - 1 ? t_gT : t_gL;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      double u = f[j];
      u = fma(yl, tg[j * Mb + kl], u);
      u = fma(yr, t_gL[(S - 1 - j) * Mb + kl], u);   // the last chunk's right end value is 0
      if (!TAIL || j < len) dst[(size_t)(r0 + j) * ld] = u;
    }
    if (c >= 1) dst[(size_t)(r0 - 1) * ld] = yl;
  }
}

template <int S, bool TAIL>
__global__ void __launch_bounds__(256, 2) k_tri_reg(TriOp op, const double* __restrict__ F, double* U, int ld, int Mb,
                                                 TriBc bc) {
  extern __shared__ double sm[];
  tri_reg_body<S, TAIL>(op, F, U, ld, Mb, bc, sm);   // waits for the previous kernel after its tables
}

// The same solve for every item of a batch, blockIdx.y picking the item (its tables, input,
// output and boundary terms); the items share the chunking.
template <int S, bool TAIL>
__global__ void __launch_bounds__(256, 2) k_tri_reg_batch(const __grid_constant__ TriBatch b, int ld, int Mb) {
  extern __shared__ double sm[];
  const int y = blockIdx.y;
  tri_reg_body<S, TAIL>(b.op[y], b.F[y], b.U[y], ld, Mb, b.bc[y], sm);
}

static size_t tri_reg_smem(const TriOp& op, int Mb) {
  return sizeof(double) * (size_t)Mb *
         ((op.r < op.s ? 4 : 3) * (size_t)op.s + 2 * (size_t)op.C + 2 * ((size_t)op.C + 1) +
          (size_t)op.C * std::max(op.C - 1, 1));
}

template <int S, bool TAIL>
static int launch_tri_reg(const TriOp& op, const double* F, double* U, int ld, int Mb, int threads, const TriBc& bc,
                          cudaStream_t st) {
  const size_t smem = tri_reg_smem(op, Mb);
  if (allow_dyn_smem(k_tri_reg<S, TAIL>, smem) != cudaSuccess) return IB_ERR_CUDA;
  count_launch();
  k_tri_reg<S, TAIL><<<cdiv(op.nx, Mb), threads, smem, st>>>(op, F, U, ld, Mb, bc);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

size_t tri_smem(const TriOp& op, int Mb) {
  const size_t m = op.C > 1 ? (size_t)(op.C - 1) : 0;
  return sizeof(double) * (size_t)Mb * ((size_t)op.ny + 3 * (size_t)op.s + m * m + 2 * (size_t)op.C + 2 * ((size_t)op.C + 1));
}

int tri_solve(const TriOp& op, const double* F, double* U, int ld, const TriLaunch& L, cudaStream_t st,
              const TriBc& bc) {
  int Mb = L.Mb;
  int threads = Mb * op.C;
  threads = ((threads + 31) / 32) * 32;
  if (threads > 1024) { Mb = 1024 / op.C; threads = ((Mb * op.C + 31) / 32) * 32; }
  if (op.C - 1 <= kTriMaxM && op.C <= 256) {
    // at most 256 threads (the register-resident chunk needs the registers)
    const int Mr = std::max(1, std::min(Mb, 256 / op.C));
    const int tr = ((Mr * op.C + 31) / 32) * 32;
    const bool tail = op.r < op.s;
    switch (op.s) {
#define IB_TRI_REG(SS) \
      case SS: if (!tail) return launch_tri_reg<SS, false>(op, F, U, ld, Mr, tr, bc, st); break;
      IB_TRI_EVEN(IB_TRI_REG)
#undef IB_TRI_REG
#define IB_TRI_REG(SS) \
      case SS: return tail ? launch_tri_reg<SS, true>(op, F, U, ld, Mr, tr, bc, st) \
                           : launch_tri_reg<SS, false>(op, F, U, ld, Mr, tr, bc, st);
      IB_TRI_BOTH(IB_TRI_REG)
#undef IB_TRI_REG
      default: break;
    }
  }
  if (op.r < op.s) return IB_ERR_ARG;   // tri_chunking gives the shared-memory kernel equal chunks
  size_t smem = tri_smem(op, Mb);
  if (allow_dyn_smem(k_tri, smem) != cudaSuccess) return IB_ERR_CUDA;
  count_launch();
  k_tri<<<cdiv(op.nx, Mb), threads, smem, st>>>(op, F, U, ld, Mb, bc);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

template <int S, bool TAIL>
static int launch_tri_reg_batch(const TriBatch& b, int ld, int Mb, int threads, cudaStream_t st) {
  const size_t smem = tri_reg_smem(b.op[0], Mb);
  if (allow_dyn_smem(k_tri_reg_batch<S, TAIL>, smem) != cudaSuccess) return IB_ERR_CUDA;
  count_launch();
  k_tri_reg_batch<S, TAIL><<<dim3(cdiv(b.op[0].nx, Mb), b.n), threads, smem, st>>>(b, ld, Mb);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

bool tri_batch_supported(const TriOp& op) {
  return op.C - 1 <= kTriMaxM && op.C <= 256 && tri_reg_length(op.s, op.r < op.s);
}

int tri_solve_batch(const TriBatch& b, int ld, const TriLaunch& L, cudaStream_t st) {
  if (b.n < 1 || b.n > kTriBatch) return IB_ERR_ARG;
  const TriOp& o = b.op[0];
  if (!tri_batch_supported(o)) return IB_ERR_ARG;
  for (int i = 1; i < b.n; ++i)
    if (b.op[i].nx != o.nx || b.op[i].ny != o.ny || b.op[i].s != o.s || b.op[i].C != o.C) return IB_ERR_ARG;
  const int Mr = std::max(1, std::min(L.Mb, 256 / o.C));
  const int tr = ((Mr * o.C + 31) / 32) * 32;
  const bool tail = o.r < o.s;
  switch (o.s) {
#define IB_TRI_REG(SS) \
    case SS: return tail ? IB_ERR_ARG : launch_tri_reg_batch<SS, false>(b, ld, Mr, tr, st);
    IB_TRI_EVEN(IB_TRI_REG)
#undef IB_TRI_REG
#define IB_TRI_REG(SS) \
    case SS: return tail ? launch_tri_reg_batch<SS, true>(b, ld, Mr, tr, st) \
                         : launch_tri_reg_batch<SS, false>(b, ld, Mr, tr, st);
    IB_TRI_BOTH(IB_TRI_REG)
#undef IB_TRI_REG
    default: return IB_ERR_ARG;
  }
}

}  // namespace ib
