// 64-bit block fixed point for the sine transforms.
//
// An FP64 warp instruction holds its SM sub-partition's FP64 pipe for 64 cycles on GB300, a 64-bit
// integer add (two instructions) for 2.5 and the product below for about 17.  The transforms are sums
// of values multiplied by factors of modulus below 2, so a line is transformed in integers that share
// one exponent: x = v 2^E.  Between the stages a line is rescaled by the largest magnitude it holds,
// to at most kFxBits bits, so 58 bits carry what FP64's 53 did (the shared exponent costs the line's
// peak-to-rms ratio, 2 to 3 bits; the error against 64-bit sine matrices is smaller than the FP64
// transform's, tests/test_gpu_dst_fixed.py).
#pragma once
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define IB_FX __host__ __device__ __forceinline__
#else
#define IB_FX inline
#endif

namespace ib {

typedef long long fx;

// Magnitudes entering a stage are below 2^kFxBits: then the operands of every product in it (at most
// 4 sqrt(2) times larger, in the radix-5 butterfly) are below 2^61, which fx_mul needs, and its
// results (at most 5 sqrt(2) times larger) fit 64 bits.
constexpr int kFxBits = 58;
// A line's largest sample starts below 2^kFxFrac, two bits lower: the first stage needs no shift, and
// a line that grows little none at all.
constexpr int kFxFrac = 56;

// A factor |w| < 2 as (hi 2^32 + lo) 2^-62 with lo in [-2^31, 2^31).
struct FxW {
  int hi, lo;
};

inline FxW fx_factor(long double w) {
  const long double s = w * 4611686018427387904.0L;   // 2^62
  const long long v = (long long)(s < 0 ? s - 0.5L : s + 0.5L);
  FxW r;
  r.hi = (int)((v + (1LL << 31)) >> 32);
  r.lo = (int)(unsigned)(unsigned long long)v;
  return r;
}

// x w, |x| below 2^61 (4 x and the carry of its halves fit), to within 0.75 of a unit: the product of
// the low halves is left out (at most a quarter of a unit, of zero mean: both halves are balanced, so
// nothing adds up along the prefix sums).  Three 32 x 32 + 64-bit multiply-adds.
IB_FX fx fx_mul(fx x, int whi, int wlo) {
  const fx x4 = (fx)((unsigned long long)x << 2);
  const int lo = (int)(unsigned)(unsigned long long)x4;
  const int hi = (int)(x4 >> 32) + (int)((unsigned)lo >> 31);
  fx c = (fx)hi * wlo + (1LL << 31);
  c += (fx)lo * whi;
  return (fx)hi * whi + (c >> 32);
}
IB_FX fx fx_mul(fx x, FxW w) { return fx_mul(x, w.hi, w.lo); }

// x 2^-s to nearest, ties to even, 0 <= s < 32.  (Rounding the ties up, three instructions less, is a
// bias that adds up along the prefix sums: five to ten times the error at 800 cells.)
IB_FX fx fx_shr(fx x, int s) {
  if (s == 0) return x;
  return (x + ((1LL << (s - 1)) - 1) + (fx)(((unsigned)x >> s) & 1u)) >> s;
}

// |x|'s high word (one's complement for x < 0): |x| <= (fx_mag(x) + 1) 2^32
IB_FX unsigned fx_mag(fx x) {
  const int h = (int)(x >> 32);
  return (unsigned)(h ^ (h >> 31));
}

// The largest magnitude of a set of values, from their high words' extremes.
struct FxPeak {
  int hi = 0, lo = -1;
  IB_FX void add(fx a, fx b) {
    const int x = (int)(a >> 32), y = (int)(b >> 32);
#if defined(__CUDA_ARCH__)
    hi = __vimax3_s32(hi, x, y);
    lo = __vimin3_s32(lo, x, y);
#else
    hi = x > hi ? x : hi; hi = y > hi ? y : hi;
    lo = x < lo ? x : lo; lo = y < lo ? y : lo;
#endif
  }
  IB_FX unsigned mag() const { return (unsigned)(hi | ~lo); }   // has the top bit of the largest fx_mag
};

IB_FX int fx_clz32(unsigned v) {
#if defined(__CUDA_ARCH__)
  return __clz((int)v);
#else
  return v ? __builtin_clz(v) : 32;
#endif
}
IB_FX int fx_clz64(unsigned long long v) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)v);
#else
  return v ? __builtin_clzll(v) : 64;
#endif
}

// The right shift that brings a line whose values' fx_mag or to `mag` below 2^kFxBits.
IB_FX int fx_shift_for(unsigned mag) {
  const int bits = 64 - fx_clz32(mag);   // magnitudes < 2^bits (bits >= 32)
  return bits > kFxBits ? bits - kFxBits : 0;
}

// A double's biased exponent (1 for zeros and subnormals, 2047 for infinities and NaN).
IB_FX int fx_exponent(unsigned hiword) {
  const int e = (int)((hiword >> 20) & 0x7ffu);
  return e ? e : 1;
}

// The double with bits `b` as a multiple of 2^(emax - 1075 - (FRAC - 53)), below 2^FRAC and cut off
// towards zero; emax is at least its exponent, and both are finite.
template <int FRAC = kFxFrac>
IB_FX fx fx_from_bits(long long b, int emax) {
  const unsigned h = (unsigned)((unsigned long long)b >> 32);
  const int e = (int)((h >> 20) & 0x7ffu);
  const unsigned mh = (h & 0xfffffu) | (e ? 0x100000u : 0u);
  const unsigned long long m = (((unsigned long long)mh << 32) | (unsigned)b) << (FRAC - 53);
  const unsigned s = (unsigned)(emax - (e ? e : 1));
#if defined(__CUDA_ARCH__)
  unsigned long long r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(s));   // 0 from 64 on
#else
  const unsigned long long r = s < 64 ? m >> s : 0ULL;
#endif
  const fx sg = b >> 63;
  return ((fx)r ^ sg) - sg;
}

// v 2^E as a double's bits, rounded to nearest (ties away from zero), for exponents that keep every
// nonzero v normal (fx_plain).
IB_FX bool fx_plain(int E) { return E >= -1022 && E <= 959; }
IB_FX long long fx_to_bits_plain(fx v, int E) {
  const fx sg = v >> 63;
  unsigned long long u = (unsigned long long)((v ^ sg) - sg);
  const int lz = fx_clz64(u | 1ULL);
  u <<= lz;
  // the leading bit of u >> 11 adds 1 to the exponent field, and a rounding carry one more
  const unsigned long long r =
      (u >> 11) + ((u >> 10) & 1ULL) + ((unsigned long long)(unsigned)(1023 + 62 - lz + E) << 52);
  const unsigned long long sign = (unsigned long long)v & 0x8000000000000000ULL;
  return v ? (long long)(sign | r) : 0;
}

// The same for any exponent, with infinities above and subnormals below the normal range.
IB_FX long long fx_to_bits(fx v, int E) {
  if (v == 0) return 0;
  if (fx_plain(E)) return fx_to_bits_plain(v, E);
  const fx sg = v >> 63;
  unsigned long long u = (unsigned long long)((v ^ sg) - sg);
  const int lz = fx_clz64(u);
  u <<= lz;
  const int e = 1023 + 63 - lz + E;   // biased exponent before rounding
  const unsigned long long sign = (unsigned long long)v & 0x8000000000000000ULL;
  if (e >= 2047) return (long long)(sign | 0x7ff0000000000000ULL);
  if (e >= 1) return (long long)(sign | ((u >> 11) + ((u >> 10) & 1ULL) + ((unsigned long long)(e - 1) << 52)));
  const int s = 12 - e;   // subnormal: u >> s, to nearest
  if (s > 64) return (long long)sign;
  const unsigned long long q = s == 64 ? 0ULL : u >> s;
  return (long long)(sign | (q + ((u >> (s - 1)) & 1ULL)));
}

// A complex factor c + i d for the three-product form: c, d - c, c + d (moduli below 2).
struct FxCW {
  FxW c, dmc, cpd;
};
struct FxC {
  fx x, y;
};
IB_FX FxC fx_cmul(FxC a, FxW c, FxW dmc, FxW cpd) {
  const fx k1 = fx_mul(a.x + a.y, c);
  const fx k2 = fx_mul(a.x, dmc);
  const fx k3 = fx_mul(a.y, cpd);
  return FxC{k1 - k3, k1 + k2};
}
IB_FX FxC fx_add(FxC a, FxC b) { return FxC{a.x + b.x, a.y + b.y}; }
IB_FX FxC fx_sub(FxC a, FxC b) { return FxC{a.x - b.x, a.y - b.y}; }

// The butterflies (forward sign).  Constants are factors (hi, lo) as fx_factor rounds them.
template <int R>
struct FxDft;
template <>
struct FxDft<2> {
  IB_FX static void run(FxC* v) {
    const FxC a = v[0], b = v[1];
    v[0] = fx_add(a, b);
    v[1] = fx_sub(a, b);
  }
};
template <>
struct FxDft<4> {
  IB_FX static void run(FxC* v) {
    const FxC s02 = fx_add(v[0], v[2]), d02 = fx_sub(v[0], v[2]);
    const FxC s13 = fx_add(v[1], v[3]), d13 = fx_sub(v[1], v[3]);
    v[0] = fx_add(s02, s13);
    v[2] = fx_sub(s02, s13);
    v[1] = FxC{d02.x + d13.y, d02.y - d13.x};
    v[3] = FxC{d02.x - d13.y, d02.y + d13.x};
  }
};
constexpr int kFxS3h = 929887697, kFxS3l = -1332128537;     // sin(2 pi/3)
template <>
struct FxDft<3> {
  IB_FX static void run(FxC* v) {
    const FxC t = fx_add(v[1], v[2]), d = fx_sub(v[1], v[2]);
    const FxC a = FxC{v[0].x - fx_shr(t.x, 1), v[0].y - fx_shr(t.y, 1)};
    const fx hx = fx_mul(d.x, kFxS3h, kFxS3l), hy = fx_mul(d.y, kFxS3h, kFxS3l);
    v[0] = fx_add(v[0], t);
    v[1] = FxC{a.x + hy, a.y - hx};
    v[2] = FxC{a.x - hy, a.y + hx};
  }
};
// radix 5: cos(2 pi/5) and cos(4 pi/5) are -1/4 +- sqrt(5)/4; the sine part is a rotation of
// (d1, d2) by (s1, s2) in three products, s1 = sin(2 pi/5), s2 = sin(4 pi/5)
constexpr int kFxR5h = 600239927, kFxR5l = 803819395;     // sqrt(5)/4
constexpr int kFxS2h = 631129609, kFxS2l = -357254181;     // s2
constexpr int kFxSmh = 390059550, kFxSml = -1644870943;     // s1 - s2
constexpr int kFxSph = 1652318767, kFxSpl = 1935587992;     // s1 + s2
template <>
struct FxDft<5> {
  IB_FX static void part(fx x0, fx t1, fx t2, fx d1, fx d2, fx* sum, fx* a1, fx* a2, fx* b1, fx* b2) {
    const fx s = t1 + t2;
    const fx u = fx_mul(t1 - t2, kFxR5h, kFxR5l);
    const fx base = x0 - fx_shr(s, 2);
    *sum = x0 + s;
    *a1 = base + u;
    *a2 = base - u;
    const fx k = fx_mul(d1 + d2, kFxS2h, kFxS2l);
    *b1 = k + fx_mul(d1, kFxSmh, kFxSml);
    *b2 = k - fx_mul(d2, kFxSph, kFxSpl);
  }
  IB_FX static void run(FxC* v) {
    const FxC t1 = fx_add(v[1], v[4]), t2 = fx_add(v[2], v[3]);
    const FxC d1 = fx_sub(v[1], v[4]), d2 = fx_sub(v[2], v[3]);
    FxC a1, a2, b1, b2, s;
    part(v[0].x, t1.x, t2.x, d1.x, d2.x, &s.x, &a1.x, &a2.x, &b1.x, &b2.x);
    part(v[0].y, t1.y, t2.y, d1.y, d2.y, &s.y, &a1.y, &a2.y, &b1.y, &b2.y);
    v[0] = s;
    v[1] = FxC{a1.x + b1.y, a1.y - b1.x};
    v[4] = FxC{a1.x - b1.y, a1.y + b1.x};
    v[2] = FxC{a2.x + b2.y, a2.y - b2.x};
    v[3] = FxC{a2.x - b2.y, a2.y + b2.x};
  }
};
// The radices of a transform of P points (2^a 3^b 5^c): 5 and 3 first, whose 16 R-byte stride writes of
// the first stage meet in no shared-memory bank, then 4, then 2 (0 if P has other factors or needs more
// than `most` stages).  Radices up to 12 (8 of 2 x 4, 6, 10 and 12 without inner twiddles) took a line
// in three stages instead of four and within 8% either way at 64 to 1600 cells, for twice the registers.
inline int fx_radices(int P, int* rad, int most) {
  int n = 0;
  for (int r : {5, 3, 4, 2})
    while (P % r == 0 && n < most) {
      rad[n++] = r;
      P /= r;
    }
  return P == 1 ? n : 0;
}

}  // namespace ib
