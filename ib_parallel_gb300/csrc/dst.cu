// Batched DST-I kernels (see dst.cuh for the algorithm).
#include "dst.cuh"

#include <algorithm>
#include <cmath>
#include <vector>


namespace ib {

// ---------------------------------------------------------------- tables
static const long double PI_L = 3.141592653589793238462643383279502884L;

// The factors of a plan, in the order they lie in device memory: of P stage twiddles c + i d and then
// of the P/2 factors exp(-2 pi i k/M), the pairs (c, d - c); of both, the third factors c + d; P of
// 2 sin(j pi/M); and P + 1 doubles sin(j pi/M).
//
// The Stockham stages' twiddles lie stage by stage: the stage of span Ns (the product of the earlier
// radices) and radix R uses w^(r k P/(Ns R)), r = 1..R-1, k = 0..Ns-1, at Ns - 1 + (r-1) Ns + k, so
// that a warp's lanes (consecutive k) read consecutive entries.  The stages' blocks
// [Ns - 1, R Ns - 1) tile [0, P - 1).
static void plan_tables(const DstPlan& p, std::vector<double>& out) {
  const int P = p.P, H = p.P / 2;
  out.assign(dst_plan_doubles(p.M), 0.0);
  FxW* pair = reinterpret_cast<FxW*>(out.data());
  FxW* third = pair + 2 * (P + H);
  auto put = [&](int i, long long num, long long den) {
    const long double a = 2.0L * PI_L * (long double)(num % den) / (long double)den;
    const long double x = cosl(a), y = -sinl(a);
    pair[2 * i] = fx_factor(x);
    pair[2 * i + 1] = fx_factor(y - x);
    third[i] = fx_factor(x + y);
  };
  int Ns = 1;
  for (int s = 0; s < p.nrad; ++s) {
    const int R = p.rad[s], step = P / (Ns * R);
    for (int r = 1; r < R; ++r)
      for (int k = 0; k < Ns; ++k) put(Ns - 1 + (r - 1) * Ns + k, (long long)r * k * step, P);
    Ns *= R;
  }
  for (int k = 0; k < H; ++k) put(P + k, k, p.M);
  FxW* f = third + P + H;
  for (int j = 0; j < P; ++j) f[j] = fx_factor(2.0L * sinl(PI_L * (long double)j / (long double)p.M));
  double* sn = reinterpret_cast<double*>(f + P);
  for (int j = 0; j <= P; ++j) sn[j] = (double)sinl(PI_L * (long double)j / (long double)p.M);
}

static int plan_init(DstPlan* p, int N) {
  const int M = N + 1;
  if (N < 3 || M % 4 != 0) return IB_ERR_ARG;
  p->N = N; p->M = M; p->P = M / 2;
  p->nrad = fx_radices(p->P, p->rad, kMaxRadices);
  return p->nrad > 0 ? IB_OK : IB_ERR_ARG;
}

static void plan_pointers(DstPlan* p, double* dev) {
  const size_t n = (size_t)p->P + p->P / 2;
  p->tw = reinterpret_cast<FxW*>(dev);
  p->tw3 = p->tw + 2 * n;
  p->sx = p->tw3 + n;
  p->sn = reinterpret_cast<double*>(p->sx + p->P);
}

size_t dst_plan_doubles(int M) {
  const size_t P = M / 2;
  return 3 * P + 3 * (P / 2) + P + P + 1;
}

int dst_plan_create(DstPlan* p, int N) {
  int rc = plan_init(p, N);
  if (rc != IB_OK) return rc;
  std::vector<double> h;
  plan_tables(*p, h);
  double* dev = nullptr;
  if (cudaMalloc(&dev, sizeof(double) * h.size()) != cudaSuccess) return IB_ERR_NOMEM;
  plan_pointers(p, dev);
  IB_CUDA_CHECK(cudaMemcpy(dev, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice));
  return IB_OK;
}

size_t dst_plan_table_doubles(int N) {
  DstPlan p;
  return plan_init(&p, N) == IB_OK ? dst_plan_doubles(p.M) : 0;
}

int dst_plan_init_external(DstPlan* p, int N, double* dev, cudaStream_t st) {
  int rc = plan_init(p, N);
  if (rc != IB_OK) return rc;
  std::vector<double> h;
  plan_tables(*p, h);
  plan_pointers(p, dev);
  IB_CUDA_CHECK(cudaMemcpyAsync(dev, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice, st));
  IB_CUDA_CHECK(cudaStreamSynchronize(st));
  return IB_OK;
}

void dst_plan_destroy(DstPlan* p) {
  if (p->tw) cudaFree(p->tw);
  p->tw = p->tw3 = p->sx = nullptr; p->sn = nullptr;
}

struct DstDev {
  int N, M, P, nrad;
  int rad[kMaxRadices];
  FastDiv fd_ns[kMaxRadices];   // span of each stage (product of the earlier radices)
  const int4* tw;   // (c, d - c) of the stages' twiddles, then of the unpacking's factors
  const int2* tw3;  // c + d of both
  const int2* sx;
  const double* sn;
};

static DstDev to_dev(const DstPlan& p) {
  DstDev d;
  d.N = p.N; d.M = p.M; d.P = p.P; d.nrad = p.nrad;
  int Ns = 1;
  for (int i = 0; i < kMaxRadices; ++i) {
    d.rad[i] = p.rad[i];
    if (i < p.nrad) {
      d.fd_ns[i] = FastDiv(Ns);
      Ns *= p.rad[i];
    }
  }
  d.tw = reinterpret_cast<const int4*>(p.tw);
  d.tw3 = reinterpret_cast<const int2*>(p.tw3);
  d.sx = reinterpret_cast<const int2*>(p.sx);
  d.sn = p.sn;
  return d;
}

// ------------------------------------------------------- device helpers
__device__ __forceinline__ FxW ld_factor(const int2* __restrict__ p) {
  const int2 v = __ldg(p);
  return FxW{v.x, v.y};
}

// v times the complex factor at tw, tw3
__device__ __forceinline__ FxC twiddle(FxC v, const int4* __restrict__ tw, const int2* __restrict__ tw3) {
  const int4 a = __ldg(tw);
  return fx_cmul(v, FxW{a.x, a.y}, FxW{a.z, a.w}, ld_factor(tw3));
}

constexpr int kMaxLines = 16;         // lines per CTA
constexpr int kMaxWarps = 16;         // warps per CTA
constexpr int kNotFinite = 1 << 20;   // in place of a line's exponent

// The warps of a CTA over its B lines: wpl warps per line, `groups` lines at once (computed on the
// host: the divisions cost every warp of a short kernel).  A warp works on one line at a time, so a
// line's maxima and sums are warp reductions.
struct LineShape {
  int B, wpl, groups, inv;
  LineShape(int B_, int NT) : B(B_) {
    const int nwarps = NT / 32;
    wpl = nwarps >= B ? nwarps / B : 1;
    groups = nwarps >= B ? B : nwarps;
    inv = (65536 + wpl - 1) / wpl;   // (warp inv) >> 16 = warp / wpl for the few warps there are
  }
};
struct LineGroups {
  int B, wpl, groups, grp, gw, gt, gsz;
  __device__ __forceinline__ explicit LineGroups(const LineShape& s) : B(s.B), wpl(s.wpl), groups(s.groups) {
    const int warp = threadIdx.x >> 5;
    grp = (warp * s.inv) >> 16;
    gw = warp - grp * wpl;
    gt = gw * 32 + (threadIdx.x & 31);
    gsz = wpl * 32;
    if (grp >= groups) grp = 1 << 20;   // spare warps: no lines
  }
};

// What a CTA keeps of its lines beside their samples: a word per line and warp, so that nothing has
// to be cleared or added atomically.
struct FxLines {
  unsigned mag[2][kMaxWarps];   // largest magnitudes, of the phase before and of this one
  unsigned l1[kMaxWarps];       // a bound of sum |x| / 2^40
  int e[kMaxWarps];             // largest biased exponent of the samples (fx_exponent)
  int shift[kMaxLines];         // right shifts so far
  fx wt[kMaxWarps];             // warp totals of the prefix sums
};

// Dynamic shared memory of the transforms: the FxLines, then two buffers of B P complex values.
extern __shared__ longlong2 fx_smem[];
constexpr int kLinesWords = (sizeof(FxLines) + sizeof(longlong2) - 1) / sizeof(longlong2);
__device__ __forceinline__ FxLines& fx_lines() { return *reinterpret_cast<FxLines*>(fx_smem); }
__device__ __forceinline__ double* fx_line(int b, int P) {   // line b's 2P slots in the first buffer
  return reinterpret_cast<double*>(fx_smem + kLinesWords + b * P);
}
// the samples' largest exponent that this warp has met on line b
__device__ __forceinline__ void fx_note(const LineGroups& G, int b, int emax) {
  emax = __reduce_max_sync(0xffffffffu, emax);
  if ((threadIdx.x & 31) == 0) fx_lines().e[b * G.wpl + G.gw] = emax;
}
// line b's words of its warps, one per lane (`none` on the others)
template <typename T>
__device__ __forceinline__ T fx_words(const LineGroups& G, const T* words, int b, T none) {
  const int lane = threadIdx.x & 31;
  return lane < G.wpl ? words[b * G.wpl + lane] : none;
}
__device__ __forceinline__ unsigned fx_or(const LineGroups& G, const unsigned* words, int b) {
  return __reduce_or_sync(0xffffffffu, fx_words(G, words, b, 0u));
}

// A result's bits where a line's exponent leaves the normal range or a sample was not finite.
__device__ __noinline__ long long line_bits(fx v, int E) {
  return E == kNotFinite ? 0x7ff8000000000000LL : fx_to_bits(v, E);
}

// One Stockham stage of one line on the gsz threads of its group; the inputs are taken 2^-sh.
template <int R>
__device__ __forceinline__ unsigned stockham_stage(const longlong2* __restrict__ in, longlong2* __restrict__ out, int P,
                                                   const FastDiv& fns, const int4* __restrict__ tw,
                                                   const int2* __restrict__ tw3, int sh, int gt, int gsz) {
  const int nb = P / R, Ns = fns.d;
  FxPeak peak;
  for (int j = gt; j < nb; j += gsz) {
    FxC v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const longlong2 z = in[j + r * nb];
      v[r] = FxC{z.x, z.y};
    }
    if (sh) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = FxC{fx_shr(v[r].x, sh), fx_shr(v[r].y, sh)};
    }
    int k = 0;
    if (Ns > 1) {
      k = fns.mod(j);
#pragma unroll
      for (int r = 1; r < R; ++r) {
        const unsigned i = (unsigned)(r * Ns - 1 + k);   // this stage's twiddles (plan_tables)
        v[r] = twiddle(v[r], tw + i, tw3 + i);
      }
    }
    FxDft<R>::run(v);
    longlong2* dst = out + ((j - k) * R + k);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      dst[r * Ns] = make_longlong2(v[r].x, v[r].y);
      peak.add(v[r].x, v[r].y);
    }
  }
  return peak.mag();
}

// Transform the CTA's lines: line b holds x_1..x_N as doubles at slots 1..N of fx_line(b), its largest
// exponents noted (fx_note); every thread calls it after a barrier.  Returns where the lines'
// Y_1..Y_N lie (line b at b*M, Y_(j+1) at slot dst_slot(j, P)).
//
// In block fixed point (fixed.cuh).  What bounds it: instruction issue and the latency of the chain of
// phases (the FP64 butterflies before held the FP64 pipe for 600 x 64 cycles a line of 799); at 2000
// lines the ALU and multiply pipes are half busy, 0.6 instructions a cycle and sub-partition.  The
// twiddles loaded ahead of each barrier took 128 registers and 15% more time.
// Measured with FP64 butterflies, and so: 800 lines of 1599, 80 and 28 us; 2000 of 799, 84 and 31; 399
// of 799, 27 and 11.5; 199 of 399, 16 and 9.2; 31 of 63, 7.5 and 6.4.
__device__ __forceinline__ const double* dst_lines(const DstDev& pl, const LineGroups& G) {
  FxLines& S = fx_lines();
  const int lane = threadIdx.x & 31;
  const int P = pl.P, M = pl.M, H = P / 2, B = G.B;
  longlong2* cur = fx_smem + kLinesWords;
  longlong2* nxt = cur + B * P;
  int w = 0;   // the set of magnitudes written
  // --- pre-processing: 2 y (length M, real), each pair (j, M - j) in its own slots
  for (int b = G.grp; b < B; b += G.groups) {
    fx* y = reinterpret_cast<fx*>(cur + b * P);
    const int emax = __reduce_max_sync(0xffffffffu, fx_words(G, S.e, b, 1));
    FxPeak peak;
    unsigned l1 = 0;
    for (int t = G.gt; t < P; t += G.gsz) {
      if (t == 0) {
        const fx xp = fx_from_bits(y[P], emax);
        y[0] = 0;
        y[P] = 4 * xp;
        peak.add(4 * xp, 0);
        l1 += (fx_mag(xp) >> 8) + 1u;
      } else {
        const fx xj = fx_from_bits(y[t], emax), xm = fx_from_bits(y[M - t], emax);
        const fx a = fx_mul(xj + xm, ld_factor(pl.sx + t)), d = xj - xm;
        y[t] = a + d;
        y[M - t] = a - d;
        peak.add(a + d, a - d);
        l1 += (fx_mag(xj) >> 8) + (fx_mag(xm) >> 8) + 2u;
      }
    }
    const unsigned mag = __reduce_or_sync(0xffffffffu, peak.mag());
    l1 = __reduce_add_sync(0xffffffffu, l1);
    if (lane == 0) {
      S.mag[0][b * G.wpl + G.gw] = mag;
      S.l1[b * G.wpl + G.gw] = l1;
      if (G.gw == 0) S.shift[b] = 0;
    }
  }
  __syncthreads();
  // --- complex FFT of length P (Stockham, between the two buffers)
  for (int s = 0; s < pl.nrad; ++s) {
    for (int b = G.grp; b < B; b += G.groups) {
      const int sh = fx_shift_for(fx_or(G, S.mag[w], b));
      const longlong2* in = cur + b * P;
      longlong2* out = nxt + b * P;
      unsigned mag;
      switch (pl.rad[s]) {
#define IB_STAGE(R) \
        case R: mag = stockham_stage<R>(in, out, P, pl.fd_ns[s], pl.tw, pl.tw3, sh, G.gt, G.gsz); break;
        IB_STAGE(2) IB_STAGE(3) IB_STAGE(4)
#undef IB_STAGE
        default: mag = stockham_stage<5>(in, out, P, pl.fd_ns[s], pl.tw, pl.tw3, sh, G.gt, G.gsz); break;
      }
      mag = __reduce_or_sync(0xffffffffu, mag);
      if (lane == 0) {
        S.mag[w ^ 1][b * G.wpl + G.gw] = mag;
        if (G.gw == 0) S.shift[b] += sh;
      }
    }
    __syncthreads();
    longlong2* t = cur; cur = nxt; nxt = t;
    w ^= 1;
  }
  // what the unpacking shifts by (an odd output is a sum of increments, at most 4 ||x||_1 in these
  // units: it must fit as well), and the exponent of its results
  auto last = [&](int b, int* E) {
    const unsigned l1 = __reduce_add_sync(0xffffffffu, fx_words(G, S.l1, b, 0u));
    const int e = __reduce_max_sync(0xffffffffu, fx_words(G, S.e, b, 1));
    const int done = S.shift[b];
    const int sh = max(fx_shift_for(fx_or(G, S.mag[w], b)), (32 - fx_clz32(l1)) + 40 + 2 - done - 62);
    *E = e < 2047 ? e - 1075 - (kFxFrac - 53) - 1 + done + sh : kNotFinite;
    return sh;
  };
  // --- unpack the real FFT: even outputs D_2, D_4, .. to slots P.., the odd ones' increments to 0..P-1
  for (int b = G.grp; b < B; b += G.groups) {
    int E;
    const int sh = last(b, &E);
    const bool plain = fx_plain(E);
    const longlong2* Z = cur + b * P;
    long long* odd = reinterpret_cast<long long*>(nxt + b * P);
    long long* even = odd + P;
    auto at = [&](int i) {
      const longlong2 z = Z[i];
      return sh ? FxC{fx_shr(z.x, sh), fx_shr(z.y, sh)} : FxC{z.x, z.y};
    };
    for (int k = G.gt; k < H; k += G.gsz) {
      if (k == 0) {
        const FxC z0 = at(0), zh = at(H);
        odd[0] = z0.x + z0.y;                       // D_1
        even[H - 1] = line_bits(zh.y + zh.y, E);    // D_P
        odd[H] = zh.x + zh.x;                       // Re(2Y_{P/2})
      } else {
        const FxC zk = at(k), zp = at(P - k);
        const FxC Ev = FxC{zk.x + zp.x, zk.y - zp.y};
        const FxC O = FxC{zk.y + zp.y, zp.x - zk.x};
        const FxC T = twiddle(O, pl.tw + (unsigned)(P + k), pl.tw3 + (unsigned)(P + k));
        odd[k] = Ev.x + T.x;
        odd[P - k] = Ev.x - T.x;
        const fx e0 = -Ev.y - T.y, e1 = Ev.y - T.y;
        even[k - 1] = plain ? fx_to_bits_plain(e0, E) : line_bits(e0, E);
        even[P - k - 1] = plain ? fx_to_bits_plain(e1, E) : line_bits(e1, E);
      }
    }
  }
  __syncthreads();
  // --- inclusive prefix sum of the increments: the odd outputs.  Integer sums: exact, and the same
  // bits whatever the split into threads.
  const int c = (P + G.gsz - 1) / G.gsz;
  for (int b0 = 0; b0 < B; b0 += G.groups) {
    const int b = b0 + G.grp;
    const bool act = G.grp < G.groups && b < B;
    long long* odd = reinterpret_cast<long long*>(nxt + (act ? b : 0) * P);
    const int s0 = min(G.gt * c, P), s1 = min(s0 + c, P);
    fx acc = 0;
    if (act)
      for (int i = s0; i < s1; ++i) acc += odd[i];
    fx incl = acc;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const fx v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    if (G.wpl > 1) {
      if (lane == 31 && act) S.wt[G.grp * G.wpl + G.gw] = incl;
      __syncthreads();
    }
    if (act) {
      int E;
      last(b, &E);
      const bool plain = fx_plain(E);
      fx run = incl - acc;
      for (int j = 0; j < G.gw; ++j) run += S.wt[G.grp * G.wpl + j];
      for (int i = s0; i < s1; ++i) {
        run += odd[i];
        odd[i] = plain ? fx_to_bits_plain(run, E) : line_bits(run, E);
      }
    }
    __syncthreads();
  }
  return reinterpret_cast<const double*>(nxt);
}

// Where dst_lines leaves Y_(j+1) in a line's slots.
__device__ __forceinline__ int dst_slot(int j, int P) { return (j >> 1) + ((j & 1) ? P : 0); }

// ------------------------------------------------------------- x pass
// The pre-op operands of one CTA's level (the top-level fields, or level blockIdx.y of a batch).
struct XPre {
  const double *in2, *in3, *in4, *ring;
  double* save;
  double ca, cb, alpha, beta, fac;
  int bi0, bj0, bi1, bj1;   // PRE_ROT: the face box [bi0, bi1) x [bj0, bj1), read once per CTA
};
__device__ __forceinline__ XPre x_pre(const DstXArgs& a, int l, bool batch) {
  XPre p;
  if (batch) {
    p.in2 = a.lin2[l]; p.in3 = nullptr; p.in4 = a.lin4[l]; p.ring = a.lring[l]; p.save = a.lsave[l];
    p.ca = a.lca[l]; p.cb = a.lcb[l]; p.alpha = a.lalpha[l]; p.beta = a.lbeta[l]; p.fac = a.lfac[l];
    p.bi0 = p.bj0 = p.bi1 = p.bj1 = 0;
  } else {
    p.in2 = a.in2; p.in3 = a.in3; p.in4 = a.in4; p.ring = a.ring; p.save = a.save;
    p.ca = a.ca; p.cb = a.cb; p.alpha = a.alpha; p.beta = a.beta; p.fac = a.fac;
    p.bi0 = p.bj0 = p.bi1 = p.bj1 = 0;
    if (a.box) {
      p.bi0 = a.box[0];
      p.bj0 = a.box[1];
      p.bi1 = p.bi0 + a.box[2];
      p.bj1 = p.bj0 + a.box[3];
    }
  }
  return p;
}

template <int PRE>
__device__ __forceinline__ double x_load(const XPre& a, const double* __restrict__ in, const GridDims& g, int row,
                                         int j, int nrows, int N, int ld) {
  size_t idx = (size_t)row * ld + j;
  double v = 0.0;
  if (PRE == PRE_COPY) {
    v = in[idx];
  } else if (PRE == PRE_COMBINE) {
    v = fma(a.cb, a.in2[idx], a.ca * in[idx]) + a.in3[idx];
  } else if (PRE == PRE_ROT) {
    const int I = j + 2, J = row + 2;
    auto inbox = [&](int i, int jj) { return i >= a.bi0 && i < a.bi1 && jj >= a.bj0 && jj < a.bj1; };
    const double* hx = in;
    const double* hy = a.in2;
    const double va = inbox(I, J) ? hy[(size_t)(J - 1) * g.nvx + (I - 1)] : 0.0;
    const double vb = inbox(I - 1, J) ? hy[(size_t)(J - 1) * g.nvx + (I - 2)] : 0.0;
    const double vc = inbox(I, J) ? hx[(size_t)(J - 1) * g.nux + (I - 1)] : 0.0;
    const double vd = inbox(I, J - 1) ? hx[(size_t)(J - 2) * g.nux + (I - 1)] : 0.0;
    v = va - vb - vc + vd;
  } else if (PRE == PRE_PRED) {
    // con1 rhs + con2 rhs_old + rhsbc + (w - c L w)/normalize, L the 5-point
    // Laplacian with zero boundary: alpha = (1-4c)/normalize, beta = c/normalize
    const double ro = a.in2[idx], r = in[idx];
    double base = fma(a.cb, ro, a.ca * r);
    if (a.save) a.save[idx] = r;
    if (a.in3) {
      base = base + a.in3[idx];
    } else {
      const int I = j + 2, J = row + 2;
      if (I == 2 || I == g.m || J == 2 || J == g.n) {
        // rhsbc = 0; apply_bc(rhsbc, lastbc, f)
        double x = 0.0;
        const double* ra = a.ring;
        if (I == 2) x = x + a.fac * ra[g.left + J - 1];
        if (I == g.m) x = x + a.fac * ra[g.right + J - 1];
        if (J == 2) x = x + a.fac * ra[g.bottom + I - 1];
        if (J == g.n) x = x + a.fac * ra[g.top + I - 1];
        base = base + x;
      }
    }
    const double* w = a.in4;
    const double wl = j > 0 ? w[idx - 1] : 0.0, wr = j < N - 1 ? w[idx + 1] : 0.0;
    const double wd = row > 0 ? w[idx - ld] : 0.0, wu = row < nrows - 1 ? w[idx + ld] : 0.0;
    v = fma(a.beta, (wl + wr) + (wd + wu), fma(a.alpha, w[idx], base));
  } else {
    // apply_bc (operators_fluid.F90:539-549): left, right, bottom, top; a null input is zero
    v = in ? in[idx] : 0.0;
    int I = j + 2, J = row + 2;
    if (I == 2) v = v + a.fac * a.ring[g.left + J - 1];
    if (I == g.m) v = v + a.fac * a.ring[g.right + J - 1];
    if (J == 2) v = v + a.fac * a.ring[g.bottom + I - 1];
    if (J == g.n) v = v + a.fac * a.ring[g.top + I - 1];
  }
  return v;
}

// 64 registers a thread for every pre-operation: the predictor's FP64 stencil then overlaps other CTAs'
// integer phases (at 86 registers 236 us for 5119 lines of 1535, at 64 199 us; plain passes need 60 to 64).
template <int PRE>
__global__ void __launch_bounds__(512, 2) k_dst_x(DstDev pl, int nrows, int ld, const __grid_constant__ DstXArgs a,
                                               GridDims g, LineShape shape) {
  IB_GRID_DEP_WAIT();
  const double* ain = a.nlev ? a.lin[blockIdx.y] : a.in;
  double* aout = a.nlev ? a.lout[blockIdx.y] : a.out;
  const XPre pre = x_pre(a, blockIdx.y, PRE == PRE_PRED && a.nlev > 0);
  const LineGroups G(shape);
  const int B = G.B, N = pl.N, M = pl.M;
  // the row and treatment of the CTA's line b
  auto line_of = [&](int b, int* row) -> int {
    const int line = blockIdx.x * B + b;
    const int r = a.nlines ? a.row0 + line * a.row_step : line;
    *row = r;
    if (line >= (a.nlines ? a.nlines : nrows) || r >= nrows) return ROW_SKIP;
    if (a.rowrange) {
      const int lo = max(0, a.rowrange[0] - a.row_margin), hi = min(nrows, a.rowrange[1] + a.row_margin);
      if (a.rows_used && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        a.rows_used[0] = lo;
        a.rows_used[1] = hi;
      }
      if ((r >= lo && r < hi) || (a.fft_edge_rows && (r == 0 || r == nrows - 1))) return ROW_FFT;
      return a.rowrange[2];
    }
    if (a.rowmode && (int)blockIdx.y >= a.rowmode_level0) return a.rowmode[r];
    return ROW_FFT;
  };
  int any_fft = 0;
  for (int b = G.grp; b < B; b += G.groups) {
    int row;
    any_fft |= line_of(b, &row) == ROW_FFT;
  }
  if (B > 1) any_fft = __syncthreads_or(any_fft);   // of one line every warp knows
  const double* xb = nullptr;   // the transformed lines, M apart
  if (any_fft) {
    // 4 independent loads in flight per thread before the shared-memory stores
    for (int b = G.grp; b < B; b += G.groups) {
      int row;
      const bool live = line_of(b, &row) == ROW_FFT;
      double* x = fx_line(b, pl.P) + 1;
      int emax = 1;
      for (int j0 = G.gt; j0 < N; j0 += 4 * G.gsz) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + u * G.gsz;
          v[u] = live && j < N ? x_load<PRE>(pre, ain, g, row, j, nrows, N, ld) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + u * G.gsz;
          if (j < N) x[j] = v[u];
          emax = max(emax, (__double2hiint(v[u]) >> 20) & 0x7ff);
        }
      }
      fx_note(G, b, emax);
    }
    __syncthreads();
    xb = dst_lines(pl, G);
  }
  for (int b = G.grp; b < B; b += G.groups) {
    int row;
    const int mode = line_of(b, &row);
    if (mode == ROW_SKIP) continue;
    const size_t off = (size_t)row * ld;
    double* o = aout + off;
    const double* padd = a.post_add ? a.post_add + off : nullptr;
    if (mode == ROW_FFT) {
      const double* y = xb + b * M;
      if (padd) {
        // out may alias post_add: every load of a thread's outputs comes before their stores
        for (int j0 = G.gt; j0 < N; j0 += 4 * G.gsz) {
          double v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int j = j0 + u * G.gsz;
            if (j < N) v[u] = padd[j];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int j = j0 + u * G.gsz;
            if (j < N) o[j] = fma(a.post_scale, v[u], y[dst_slot(j, pl.P)]);
          }
        }
      } else {
#pragma unroll 4
        for (int j = G.gt; j < N; j += G.gsz) o[j] = y[dst_slot(j, pl.P)];
      }
      continue;
    }
    double x1 = 0.0, xn = 0.0;
    if (mode == ROW_EDGES) {
      x1 = x_load<PRE>(pre, ain, g, row, 0, nrows, N, ld);
      xn = x_load<PRE>(pre, ain, g, row, N - 1, nrows, N, ld);
    }
    const double* in2 = mode == ROW_SCALE ? (a.nlev ? a.lin2[blockIdx.y] : a.in2) + off : nullptr;
    for (int j = G.gt; j < N; j += G.gsz) {
      double v = 0.0;
      if (mode == ROW_EDGES) {
        const int k = j + 1;
        const double sk = __ldg(&pl.sn[k <= pl.P ? k : pl.M - k]);
        v = 2.0 * sk * ((k & 1) ? x1 + xn : x1 - xn);
      } else if (mode == ROW_SCALE) {
        v = a.row_scale * in2[j];
      }
      if (padd) v = fma(a.post_scale, padd[j], v);
      o[j] = v;
    }
  }
}


// fac * get_bc (operators_fluid.F90:475-535) of the inverse x transform of a coarser level's
// modes, without the transform (dot products with W at the points get_bc reads), and with it
// what the finer level's solve adds to its right-hand side modes
// (the boundary terms of apply_bc, operators_fluid.F90:539-549, transformed along x):
//  - sd[r] = x_1 + x_N and sd[nsy + r] = x_1 - x_N of its row r, the ring's left and right
//    entries r+1 (closed form 2 sin(pi k/M)(x_1 + (-1)^(k+1) x_N) of every row's two end values);
//  - edge[k] and edge[N + k]: the x transform of the ring's bottom and top entries 1..m-1,
//    which is fac E s_J, E the edge matrix and s_J the coarse modes of the row get_bc reads.
// The points get_bc reads come in mirror pairs about the centre column (the left and right
// sides; a bottom or top vertex and its mirror), and each pair is one warp's dot product
// (warp_sum_mirror); E keeps only its entries of equal parity.  CTAs of kReWarps warps:
// [0, nlr) take kReSeg entries of both the left and the right side (kReWarps vertex pairs);
// [nlr, nlr + 2 nbt) kReSeg entries of the left half of the bottom or top side and their
// mirrors; then one warp per mode k for the two edge dot products.  dst_ring_from_modes launches
// the first two groups alone (sd and edge null); a caller that reads sd and edge only launches the
// second group empty (nbt 0, ring null).  What bounds it is FP64: the bottom and top vertices are a
// quarter of its dot products at 800 x 400.
// The solve launched next may read the modes behind its right-hand side before it waits for this kernel
// (TriBc::early): so every thread here waits first, and none triggers dependents early.
// 4 against 8 warps: 401 CTAs against 187 at 800 x 400, so no SM has twice its share; 7.6 against 7.9 us
// (8.2 before the two edge sums of a mode shared one reduction, warp_sum2)
constexpr int kReWarps = 4;
constexpr int kReSeg = 2 * (kReWarps - 1);   // entries a CTA writes on a side (kReWarps vertices)
__global__ void __launch_bounds__(32 * kReWarps) k_ring_edge(int N, GridDims g, const double* __restrict__ spec,
                                                             int ld, const double* __restrict__ W,
                                                             const double* __restrict__ Ec, double fac,
                                                             double* __restrict__ ring, double* __restrict__ sd,
                                                             double* __restrict__ edge, int nlr, int nbt) {
  IB_GRID_DEP_WAIT();
  __shared__ double sp[kReWarps], spm[kReWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int b = blockIdx.x;
  if (b < nlr) {
    // vertex q of the left side (row J = n/4+1+q, column m/4+1) and of the right (its mirror)
    const int len = g.n + 1, qmax = (len - 1) / 2;
    const int q0 = b * (kReSeg / 2), q = q0 + warp;
    double2 v = make_double2(0.0, 0.0);
    if (q <= qmax)
      v = warp_sum_mirror(warp_dot_part(spec + (size_t)(g.n / 4 - 1 + q) * ld, W + (size_t)(g.m / 4 - 1) * N, N, lane));
    if (lane == 0) {
      sp[warp] = v.x;
      spm[warp] = v.y;
    }
    __syncthreads();
    if ((int)threadIdx.x < kReSeg) {
      const int p = b * kReSeg + (int)threadIdx.x;
      if (p < len) {
        const int qq = p / 2 - q0;
        const double vl = (p & 1) ? 0.5 * (sp[qq] + sp[qq + 1]) : sp[qq];
        const double vr = (p & 1) ? 0.5 * (spm[qq] + spm[qq + 1]) : spm[qq];
        const double xl = vl * fac, xr = vr * fac;
        if (ring) {
          ring[g.left + p] = xl;
          ring[g.right + p] = xr;
        }
        const int r = p - 1;
        if (sd && r >= 0 && r < g.nsy) {
          sd[r] = xl + xr;
          sd[g.nsy + r] = xl - xr;
        }
      }
    }
    return;
  }
  b -= nlr;
  if (b < 2 * nbt) {
    // vertex q <= m/4 of the bottom or top side (column m/4+1+q) and its mirror m/2-q
    const int side = b / nbt, cc = b - side * nbt;
    const int J = side == 0 ? g.n / 4 + 1 : 3 * g.n / 4 + 1;
    const int qc = g.m / 4;   // the centre vertex, its own mirror
    const int q0 = cc * (kReSeg / 2), q = q0 + warp;
    double2 v = make_double2(0.0, 0.0);
    if (q <= qc)
      v = warp_sum_mirror(warp_dot_part(spec + (size_t)(J - 2) * ld, W + (size_t)(g.m / 4 - 1 + q) * N, N, lane));
    if (lane == 0) {
      sp[warp] = v.x;
      spm[warp] = q == qc ? v.x : v.y;
    }
    __syncthreads();
    if ((int)threadIdx.x < kReSeg) {
      const int p = cc * kReSeg + (int)threadIdx.x;   // an entry of the left half
      if (p <= g.m / 2) {
        const int qq = p / 2 - q0;
        double* rs = ring + (side == 0 ? g.bottom : g.top);
        rs[p] = ((p & 1) ? 0.5 * (sp[qq] + sp[qq + 1]) : sp[qq]) * fac;
        if (p < g.m / 2) rs[g.m - p] = ((p & 1) ? 0.5 * (spm[qq] + spm[qq + 1]) : spm[qq]) * fac;
      }
    }
    return;
  }
  b -= 2 * nbt;
  const int k = b * kReWarps + warp;
  if (k >= N) return;
  const double2 e = warp_edge_dot(Ec, N, k, spec + (size_t)(g.n / 4 - 1) * ld, spec + (size_t)(3 * g.n / 4 - 1) * ld,
                                  lane);   // rows J = n/4 + 1 and 3n/4 + 1
  if (lane == 0) {
    edge[k] = fac * e.x;
    edge[N + k] = fac * e.y;
  }
}

// The ring alone (sd and edge null): the side and bottom/top CTAs only.
int dst_ring_from_modes(const DstPlan& px, const GridDims& g, const double* spec, int ld, const double* W, double fac,
                        double* ring, cudaStream_t st) {
  const int nlr = cdiv(g.n + 1, kReSeg), nbt = cdiv(g.m / 2 + 1, kReSeg);
  count_launch();
  k_ring_edge<<<nlr + 2 * nbt, 32 * kReWarps, 0, st>>>(px.N, g, spec, ld, W, nullptr, fac, ring, nullptr, nullptr,
                                                       nlr, nbt);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

int dst_ring_edge_from_modes(const DstPlan& px, const GridDims& g, const double* spec, int ld, const double* W,
                             const double* E, double fac, double* ring, double* sd, double* edge, cudaStream_t st) {
  const int nlr = cdiv(g.n + 1, kReSeg), nbt = ring ? cdiv(g.m / 2 + 1, kReSeg) : 0;
  count_launch();
  k_ring_edge<<<nlr + 2 * nbt + cdiv(px.N, kReWarps), 32 * kReWarps, 0, st>>>(px.N, g, spec, ld, W, E, fac, ring, sd,
                                                                              edge, nlr, nbt);
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

// E[k][k'] = sum_j W[k][j] P(j, k'), P(j, .) the row of W at the coarse vertex get_bc puts on
// entry p = j+1 of a side (I = m/4 + 1 + p/2 for even p, the mean of two for odd p), for k' of
// k's parity (stored at t = k'/2 of row k, pitch (N+1)/2).  One thread per entry; compensated
// dot product (Ogita, Rump and Oishi's Dot2: error-free product by fma and Knuth's two-sum),
// so E is close to the exact product of the tabulated W.
__global__ void k_edge_matrix(int N, int mq, const double* __restrict__ W, double* __restrict__ E) {
  const int Nh = (N + 1) / 2;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)N * Nh) return;
  const int k = (int)(idx / Nh), kp = 2 * (int)(idx - (long long)k * Nh) + (k & 1);
  if (kp >= N) {
    E[idx] = 0.0;
    return;
  }
  const double* wk = W + (size_t)k * N;
  double sum = 0.0, comp = 0.0;
  for (int j = 0; j < N; ++j) {
    const int p = j + 1, r0 = mq - 1 + p / 2;
    const double pw = (p & 1) ? 0.5 * (W[(size_t)r0 * N + kp] + W[(size_t)(r0 + 1) * N + kp]) : W[(size_t)r0 * N + kp];
    const double a = wk[j];
    const double h = a * pw, l = fma(a, pw, -h);
    const double t = sum + h, z = t - sum;
    comp += ((sum - (t - z)) + (h - z)) + l;
    sum = t;
  }
  E[idx] = sum + comp;
}

int dst_edge_matrix(const DstPlan& px, const GridDims& g, const double* W, double* E) {
  const long long n = (long long)px.N * ((px.N + 1) / 2);
  k_edge_matrix<<<(unsigned)cdiv(n, 256), 256, 0, cudaStreamLegacy>>>(px.N, g.m / 4, W, E);
  IB_CUDA_CHECK(cudaGetLastError());
  return wait_uploads();
}


// out = post_scale*post_add + S_x(apply_bc(ring)) on every row (operators_fluid.F90:539-549 with
// factor 1 on a zero field).  The first nEdge CTAs take the two edge rows 0 and n-2, whose
// boundary field is a full row: both rows are built once per CTA in shared memory and one warp
// per mode k reads row k of the (symmetric) DST matrix once for both dot products.  The other
// CTAs take kRowsPerCta interior rows each, whose boundary field is zero except
// x_1 = ring(left) and x_N = ring(right): Y_k = 2 sin(pi k/M)(x_1 + (-1)^(k+1) x_N), one FMA per
// output from the row's two sums and the tabulated 2 sin(pi k/M).  With fft_edges the two edge
// rows are instead transformed by the FFT line transform, one CTA each (about 2 x 700 FP64
// instructions instead of 2 N^2 multiply-adds: for the band build's and the sub-domain
// precompute's concurrent columns, which share the FP64 pipes).  In place allowed.
constexpr int kRowsPerCta = 8;
__global__ void __launch_bounds__(256) k_dst_bc_modes(DstDev pl, GridDims g, const double* __restrict__ ring,
                                                      const double* __restrict__ W, const double* __restrict__ sk2,
                                                      const double* __restrict__ post_add, double post_scale,
                                                      double* __restrict__ out, int nEdge, int fft_edges,
                                                      LineShape shape) {
  IB_GRID_DEP_WAIT();
  const int N = pl.N;
  if (fft_edges && (int)blockIdx.x < nEdge) {
    const LineGroups G(shape);   // one line, the row
    double* x = fx_line(0, pl.P) + 1;
    const int e = blockIdx.x;
    const int J = e == 0 ? 2 : g.n;
    int emax = 1;
    for (int j = threadIdx.x; j < N; j += blockDim.x) {
      const int I = j + 2;
      double v = 0.0;
      if (I == 2) v = v + ring[g.left + J - 1];
      if (I == g.m) v = v + ring[g.right + J - 1];
      if (J == 2) v = v + ring[g.bottom + I - 1];
      if (J == g.n) v = v + ring[g.top + I - 1];
      x[j] = v;
      emax = max(emax, (__double2hiint(v) >> 20) & 0x7ff);
    }
    fx_note(G, 0, emax);
    __syncthreads();
    const double* line = dst_lines(pl, G);
    const size_t row = e == 0 ? 0 : (size_t)(g.nsy - 1) * g.nsx;
    for (int k = threadIdx.x; k < N; k += blockDim.x) {
      const size_t o = row + k;
      const double y = line[dst_slot(k, pl.P)];
      out[o] = post_add ? fma(post_scale, post_add[o], y) : y;
    }
    return;
  }
  if ((int)blockIdx.x >= nEdge) {
    __shared__ double s_sum[kRowsPerCta][2];   // x_1 + x_N, x_1 - x_N per row
    const int r0 = 1 + ((int)blockIdx.x - nEdge) * kRowsPerCta;
    const int nr = min(kRowsPerCta, g.nsy - 1 - r0);
    if ((int)threadIdx.x < nr) {
      const int J = r0 + (int)threadIdx.x + 2;
      const double x1 = 0.0 + ring[g.left + J - 1];
      const double xn = 0.0 + ring[g.right + J - 1];
      s_sum[threadIdx.x][0] = x1 + xn;
      s_sum[threadIdx.x][1] = x1 - xn;
    }
    __syncthreads();
    // out may alias post_add: every load of a thread's outputs is issued before its stores
    for (int k = threadIdx.x; k < N; k += blockDim.x) {
      const double a = __ldg(&sk2[k]);
      const int par = (k & 1);   // mode kk = k+1 odd <=> k even
      double pa[kRowsPerCta];
#pragma unroll
      for (int i = 0; i < kRowsPerCta; ++i)
        pa[i] = (post_add && i < nr) ? post_add[(size_t)(r0 + i) * g.nsx + k] : 0.0;
#pragma unroll
      for (int i = 0; i < kRowsPerCta; ++i) {
        if (i >= nr) break;
        const double sv = s_sum[i][par];
        out[(size_t)(r0 + i) * g.nsx + k] = post_add ? fma(a, sv, post_scale * pa[i]) : a * sv;
      }
    }
    return;
  }
  extern __shared__ double bc[];   // 2 x N: rows 0 and n-2 of the boundary field
  for (int q = threadIdx.x; q < 2 * N; q += blockDim.x) {
    const int e = q / N, j = q - e * N;
    const int I = j + 2, J = e == 0 ? 2 : g.n;
    double v = 0.0;
    if (I == 2) v = v + ring[g.left + J - 1];
    if (I == g.m) v = v + ring[g.right + J - 1];
    if (J == 2) v = v + ring[g.bottom + I - 1];
    if (J == g.n) v = v + ring[g.top + I - 1];
    bc[q] = v;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (k >= N) return;
  const double* wk = W + (size_t)k * N;
  double a0 = 0.0, a1 = 0.0;
#pragma unroll 5
  for (int j = lane; j < N; j += 32) {
    const double w = wk[j];
    a0 = fma(bc[j], w, a0);
    a1 = fma(bc[N + j], w, a1);
  }
  for (int o = 16; o > 0; o >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
  }
  if (lane == 0) {
    const size_t o0 = (size_t)k, o1 = (size_t)(g.nsy - 1) * g.nsx + k;
    out[o0] = post_add ? fma(post_scale, post_add[o0], a0) : a0;
    out[o1] = post_add ? fma(post_scale, post_add[o1], a1) : a1;
  }
}

int dst_x_bc_modes(const DstPlan& px, const GridDims& g, const double* ring, const double* W, const double* sk2,
                   const double* post_add, double post_scale, double* out, cudaStream_t st, bool fft_edges) {
  const int N = px.N;
  const size_t smem = fft_edges ? dst_smem_x(px, 1) : 2 * sizeof(double) * (size_t)N;
  if (allow_dyn_smem(k_dst_bc_modes, dst_smem_x(px, 1)) != cudaSuccess) return IB_ERR_CUDA;
  const int nEdge = fft_edges ? 2 : cdiv(N, 8);
  const int nblk = nEdge + cdiv(std::max(0, g.nsy - 2), kRowsPerCta);
  DstDev d = to_dev(px);
  count_launch();
  k_dst_bc_modes<<<nblk, 256, smem, st>>>(d, g, ring, W, sk2, post_add, post_scale, out, nEdge, fft_edges ? 1 : 0,
                                          LineShape(1, 256));
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

int dst_sin2_table(const DstPlan& px, double* dev_out) {
  std::vector<double> v(px.N);
  for (int k = 1; k <= px.N; ++k) {
    const int kk = k <= px.P ? k : px.M - k;   // the plan's sin table entry the transform uses
    const double sk = (double)sinl(PI_L * (long double)kk / (long double)px.M);
    v[k - 1] = 2.0 * sk;
  }
  IB_CUDA_CHECK(cudaMemcpy(dev_out, v.data(), 8 * v.size(), cudaMemcpyHostToDevice));
  return IB_OK;
}

int dst_matrix_table(const DstPlan& px, double* dev_out) {
  const int N = px.N, M = px.M;
  // entry (j, k) is 2 sin(pi r / M) with r = jk mod 2M: one table of the 2M values (long double is
  // software-emulated on some hosts, so it is not evaluated N^2 times)
  std::vector<double> tab(2 * (size_t)M);
  for (long long r = 0; r < 2LL * M; ++r) tab[r] = (double)(2.0L * sinl(PI_L * (long double)r / (long double)M));
  std::vector<double> w((size_t)N * N);
  for (int j = 1; j <= N; ++j)
    for (int k = 1; k <= N; ++k) w[(size_t)(j - 1) * N + (k - 1)] = tab[(long long)j * k % (2LL * M)];
  IB_CUDA_CHECK(cudaMemcpy(dev_out, w.data(), 8 * w.size(), cudaMemcpyHostToDevice));
  return IB_OK;
}



// ------------------------------------------------------------- y pass
__global__ void __launch_bounds__(512) k_dst_y(DstDev pl, int ncols, int ld, DstYArgs a, LineShape shape) {
  IB_GRID_DEP_WAIT();
  const LineGroups G(shape);
  const int B = G.B, N = pl.N, M = pl.M;
  const int col0 = blockIdx.x * B;
  for (int it = threadIdx.x; it < B * N; it += blockDim.x) {   // a row's B columns side by side
    const int j = it / B, b = it - j * B;
    const int col = col0 + b;
    fx_line(b, pl.P)[j + 1] = col < ncols ? a.a[(size_t)j * ld + col] : 0.0;
  }
  __syncthreads();
  for (int b = G.grp; b < B; b += G.groups) {
    const double* x = fx_line(b, pl.P) + 1;
    int emax = 1;
    for (int j = G.gt; j < N; j += G.gsz) emax = max(emax, (__double2hiint(x[j]) >> 20) & 0x7ff);
    fx_note(G, b, emax);
  }
  __syncthreads();
  const double* xa = dst_lines(pl, G);
  for (int it = threadIdx.x; it < B * N; it += blockDim.x) {
    const int j = it / B, b = it - j * B;
    const int col = col0 + b;
    if (col < ncols) a.a[(size_t)j * ld + col] = xa[b * M + dst_slot(j, pl.P)];
  }
}

size_t dst_smem_x(const DstPlan& p, int B) { return sizeof(longlong2) * ((size_t)kLinesWords + (size_t)B * p.M); }
size_t dst_smem_y(const DstPlan& p, int B, DstYMode) { return dst_smem_x(p, B); }

template <typename K>
static int launch_cfg(K kern, size_t smem) {
  static_assert(sizeof(K) > 0, "");
  // the largest shared-memory carveout: the transforms' occupancy is bound by shared memory
  if (cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
      cudaSuccess)
    return IB_ERR_CUDA;
  if (allow_dyn_smem(kern, smem) != cudaSuccess) return IB_ERR_CUDA;
  return IB_OK;
}

int dst_pass_x(const DstPlan& px, int nrows, int ld, DstPre pre, const DstXArgs& a, const GridDims& g,
               const DstLaunch& L, cudaStream_t st) {
  if (L.B > kMaxLines || L.NT > 32 * kMaxWarps || a.nlev < 0 || a.nlev > kMaxBatch ||
      (a.nlev && pre != PRE_COPY && pre != PRE_PRED))
    return IB_ERR_ARG;
  DstDev d = to_dev(px);
  size_t smem = dst_smem_x(px, L.B);
  dim3 grid(cdiv(a.nlines ? a.nlines : nrows, L.B), a.nlev ? a.nlev : 1);
  int rc = IB_OK;
  switch (pre) {
    case PRE_COPY:
      rc = launch_cfg(k_dst_x<PRE_COPY>, smem);
      if (rc) return rc;
      count_launch();
      k_dst_x<PRE_COPY><<<grid, L.NT, smem, st>>>(d, nrows, ld, a, g, LineShape(L.B, L.NT));
      break;
    case PRE_COMBINE:
      rc = launch_cfg(k_dst_x<PRE_COMBINE>, smem);
      if (rc) return rc;
      count_launch();
      k_dst_x<PRE_COMBINE><<<grid, L.NT, smem, st>>>(d, nrows, ld, a, g, LineShape(L.B, L.NT));
      break;
    case PRE_PRED:
      rc = launch_cfg(k_dst_x<PRE_PRED>, smem);
      if (rc) return rc;
      count_launch();
      k_dst_x<PRE_PRED><<<grid, L.NT, smem, st>>>(d, nrows, ld, a, g, LineShape(L.B, L.NT));
      break;
    case PRE_ROT:
      if (!a.box || !a.in2) return IB_ERR_ARG;
      rc = launch_cfg(k_dst_x<PRE_ROT>, smem);
      if (rc) return rc;
      count_launch();
      k_dst_x<PRE_ROT><<<grid, L.NT, smem, st>>>(d, nrows, ld, a, g, LineShape(L.B, L.NT));
      break;
    default:
      rc = launch_cfg(k_dst_x<PRE_APPLYBC>, smem);
      if (rc) return rc;
      count_launch();
      k_dst_x<PRE_APPLYBC><<<grid, L.NT, smem, st>>>(d, nrows, ld, a, g, LineShape(L.B, L.NT));
      break;
  }
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

int dst_pass_y(const DstPlan& py, int ncols, int ld, DstYMode, const DstYArgs& a, const DstLaunch& L,
               cudaStream_t st) {
  DstDev d = to_dev(py);
  size_t smem = dst_smem_y(py, L.B, YMODE_NONE);
  dim3 grid(cdiv(ncols, L.B));
  int rc = launch_cfg(k_dst_y, smem);
  if (rc) return rc;
  count_launch();
  k_dst_y<<<grid, L.NT, smem, st>>>(d, ncols, ld, a, LineShape(L.B, L.NT));
  IB_CUDA_CHECK(cudaGetLastError());
  return IB_OK;
}

}  // namespace ib
