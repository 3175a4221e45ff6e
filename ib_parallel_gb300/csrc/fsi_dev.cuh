// Device bodies shared by the per-stage kernels of the FSI iteration (structure update,
// delta-function weights, influence patches) and the device FSI loop's fused kernel, so that
// both evaluate the same arithmetic.
#pragma once
#include "kernels.cuh"

namespace ib {

// The smoothed 6-point delta function (grid.F90:955-1003) over dr, from its table (delta_table,
// ibm.cu): on each of its three pieces (r1 = |x1 - x2| / dr up to 1, 2 and 3) kDeltaSub polynomials of
// degree kDeltaDeg.  The pieces do not meet exactly (single-precision literals), so which one a point
// falls on follows from r1 rounded as the reference rounds it.
// What bounds it: a chain of FP64 operations of 64 cycles.  The closed form (an arcsine, a square root,
// two divisions) takes about 218 on one lane, the division for r1 and the polynomial about 30.  The
// weights of 78 unknowns (k_reg_weights) took 17.4 us with it and take 4.5, the end of an FSI iteration
// of 102 (k_fsi_update) 25.5 and 15.0.
constexpr int kDeltaSub = 32, kDeltaDeg = 16;
constexpr int kDeltaTable = 3 * kDeltaSub * (kDeltaDeg + 1);
__device__ __forceinline__ double deltafnc_dev(double x1, double x2, double dr, const double* __restrict__ tab) {
  const double r1 = fabs(x1 - x2) / dr;
  if (!(r1 <= 3.0)) return 0.0;
  const int piece = r1 <= 1.0 ? 0 : (r1 <= 2.0 ? 1 : 2);
  const double s = (double)kDeltaSub * (r1 - (double)piece);
  const int sub = min((int)s, kDeltaSub - 1);
  const double x = fma(2.0, s, -(double)(2 * sub + 1));
  const double* c = tab + (piece * kDeltaSub + sub) * (kDeltaDeg + 1);
  double v = __ldg(c + kDeltaDeg);
#pragma unroll
  for (int i = kDeltaDeg - 1; i >= 0; --i) v = fma(v, x, __ldg(c + i));
  return v;
}

// compute_dx + update_xb (operators_struct.F90:402-505, 600-620) of torsional body t, the
// scalar part, on one whole warp: BR . f from lane-strided partials joined by an xor tree and
// the Newmark update of theta (with the body's step constants); g = gamma0 - theta_new, whose
// sin and cos the caller evaluates.  Every lane returns the same.
struct TorsDx {
  double thn, dth, g;
};
__device__ __forceinline__ TorsDx tors_dx_warp(const TorsBody& b, const TorsState& s, int t,
                                               const double* __restrict__ f) {
  const int lane = threadIdx.x & 31;
  const double th = s.theta[t], th0 = s.theta0[t], thd0 = s.thetad0[t], thdd0 = s.thetadd0[t];
  const double I = b.itheta, C = b.ctheta;
  const double sn0 = s.sinv[t], cs0 = s.cosv[t];
  double part = 0.0;
  for (int j = lane; j < 2 * b.npts; j += 32) part += br_val(b, sn0, cs0, j) * f[b.off + j];
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  double brf = 0.0 + part;
  const double jr = b.keff_inv * (I * (b.a44 * th0 + b.a4 * thd0 + thdd0) + C * (thd0 + b.a2 * th0) - b.keff * th);
  brf = b.bq * brf * b.bs;
  TorsDx u;
  u.dth = jr + brf;
  u.thn = th + u.dth;
  u.g = b.gamma0 - u.thn;
  return u;
}
// The new velocity and acceleration of the Newmark update.
__device__ __forceinline__ void tors_rates(const TorsBody& b, double thn, double th0, double thd0, double thdd0,
                                           double* thd, double* thdd) {
  *thd = -thd0 + b.a2 * (thn - th0);
  *thdd = -thdd0 - b.a4 * thd0 + b.a44 * (thn - th0);
}
// Position of unknown idx (0..2 npts-1) of a torsional body at sin, cos (gamma0 - theta).
// Each product and the sum are rounded separately, as update_xb writes them
// (operators_struct.F90:600-620): the positions decide which side of a stencil edge a grid
// point falls on.
__device__ __forceinline__ double2 tors_point(const TorsBody& b, int idx, double sg, double cg) {
  const int j = idx < b.npts ? idx : idx - b.npts;
  const double r = __dmul_rn((double)j, b.deltas);
  return make_double2(__dadd_rn(b.xbf0, __dmul_rn(r, cg)), __dadd_rn(b.ybf0, __dmul_rn(r, sg)));
}

// Stencil origins and the 49 weights (l outer, p inner) of the 8 unknowns k0..k0+7 on one CTA
// of 4 warps, from their positions pos[u] = (x, y): a thread per unknown, axis and offset q (the
// eighth of each axis idle); the factors meet in shared memory for the products.  Writes the weights
// to w (and wsm[u][.] when given), the origins to ix, iy and org[u][.]; stale |= 1 when an origin
// moved; err = IB_ERR_DOMAIN when a stencil leaves the grid.  Ends with a CTA barrier.
__device__ __forceinline__ void reg_weights_cta(const GridDims& g, int nf, int k0, const double (*pos)[2], double d,
                                                double ox, double oy, const double* __restrict__ tab,
                                                const int* __restrict__ comp, int* ix, int* iy, double* w, int* stale,
                                                int* err, double (*fac)[7], double (*wsm)[49], int (*org)[2]) {
  const int tid = threadIdx.x;
  const int u = tid >> 4, axis = (tid >> 3) & 1, q = tid & 7, k = k0 + u;
  if (k < nf && q < 7) {
    const double z = pos[u][axis], o = axis ? oy : ox;
    // Fortran INT truncates toward zero.  A point far outside, or one that is not a number, keeps its
    // origin within 16 cells of the grid (and is reported below): the boxes and offsets formed from
    // origins then fit an int, and no list index does worse than leave its capacity, which is checked.
    const int c = min(max((int)((z + o) / d), -16), (axis ? g.n : g.m) + 16) + 1;
    // The grid coordinate is rounded after the product and again after the sum, as the
    // reference's expression delta*(indexx-1+p)-offsetx is (grid.F90:459-528): the delta
    // function is discontinuous at 3 cells (its single-precision constants leave about 1e-8
    // there), so a point on a grid line (e.g. x = 0 with offsetx = 1, delta = 0.02) must see
    // the same side of that edge, which a fused multiply-add could change by one rounding.
    double x = __dsub_rn(__dmul_rn(d, (double)(c - 1 + q - 3)), o);
    if ((comp[k] == 1) == (axis == 1)) x = __dadd_rn(x, 0.5 * d);   // faces lie half a cell off across
    const double fv = deltafnc_dev(x, z, d, tab);
    fac[2 * u + axis][q] = axis == 0 ? d * d * fv : fv;
    if (q == 0) org[u][axis] = c;
  }
  __syncthreads();
  if (tid < 8 && k0 + tid < nf) {
    const int kk = k0 + tid, cx = org[tid][0], cy = org[tid][1];
    const bool isx = comp[kk] == 1;
    // the contribution lists depend on the stencil origins only: rebuild them when one moved
    if (ix[kk] != cx || iy[kk] != cy) atomicOr(stale, 1);
    ix[kk] = cx;
    iy[kk] = cy;
    // faces touched: u-face i in [1,m+1], j in [1,n]; v-face i in [1,m], j in [1,n+1]
    const int imax = isx ? g.m + 1 : g.m, jmax = isx ? g.n : g.n + 1;
    if (cx - 3 < 1 || cx + 3 > imax || cy - 3 < 1 || cy + 3 > jmax) atomicExch(err, IB_ERR_DOMAIN);
  }
  for (int t = tid; t < 8 * 49; t += blockDim.x) {
    const int uu = t / 49, sl = t - uu * 49;
    if (k0 + uu >= nf) break;
    const int l = sl / 7, p = sl - l * 7;
    const double wv = fac[2 * uu][p] * fac[2 * uu + 1][l];
    w[(size_t)(k0 + uu) * 49 + sl] = wv;
    if (wsm) wsm[uu][sl] = wv;
  }
  __syncthreads();
}

// Entry q (of 64) of unknown k's influence patch: rot(E^T e_k) on the vertices
// I in [cx-3, cx+4], J in [cy-3, cy+4], with the vertex's index in the band (tiles of
// tile x tile vertices).  flag |= 1 when the vertex lies outside the band, |= 2 when it is
// not an interior vertex (its streamfunction would come from the boundary ring).
__device__ __forceinline__ void patch_entry(const GridDims& g, int k, int q, bool isx, int cx, int cy,
                                            const double* wk, const int* __restrict__ tile_of, int ntx, int tile,
                                            double* __restrict__ pval, int* __restrict__ pidx, int* __restrict__ used,
                                            int* __restrict__ flag) {
  const int di = q & 7, dj = q >> 3;
  auto W = [&](int p, int l) -> double {
    return (p >= -3 && p <= 3 && l >= -3 && l <= 3) ? wk[(l + 3) * 7 + (p + 3)] : 0.0;
  };
  const int p = di - 3, l = dj - 3;
  // rot (operators_fluid.F90:203-233) of the spread unit force: a u-face (i,j) adds -1 to
  // vertex (i,j) and +1 to (i,j+1); a v-face adds +1 to (i,j) and -1 to (i+1,j)
  double v = isx ? W(p, l - 1) - W(p, l) : W(p, l) - W(p - 1, l);
  const int a = cx - 3 + di - 2, b = cy - 3 + dj - 2;   // 0-based interior vertex
  int idx = -1, fl = 0;
  if (a < 0 || a >= g.nsx || b < 0 || b >= g.nsy) {
    fl = 2;
  } else if (!tile_of) {
    fl = 1;
  } else {
    const int t = tile_of[(b / tile) * ntx + a / tile];
    if (t < 0) fl = 1;
    else idx = t * 64 + (b % tile) * tile + (a % tile);
  }
  if (idx < 0) v = 0.0;
  pval[(size_t)k * 64 + q] = v;
  pidx[(size_t)k * 64 + q] = idx;
  if (idx >= 0) used[idx] = 1;
  if (fl) atomicOr(flag, fl);
}

}  // namespace ib
