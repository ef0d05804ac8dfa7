// FP64 values worked on the integer pipes.
//
// The GPU's FP64 pipe issues one warp instruction in 16 cycles for a whole SM,
// its four integer pipes 128 lanes a cycle. A product of two 64-bit mantissas
// to 64 bits is three 32-bit multiplies and two additions, some ten issue
// slots of the 64 that one FP64 instruction holds its pipe for, and keeps 11
// bits more than FP64 does. So the sums that FP64 accuracy needs are taken in
// FP64, and what is formed from a distance -- its square, 1/r, 1/r^3 -- in
// fixed point, rounded to FP64 once at the end.
#pragma once

#include "common.cuh"

namespace gtc {

// High 64 bits of a b, at most three units low (the low halves' product is
// left out).
__device__ __forceinline__ u64 mulhi(u64 a, u64 b) {
  const u32 ah = static_cast<u32>(a >> 32), al = static_cast<u32>(a);
  const u32 bh = static_cast<u32>(b >> 32), bl = static_cast<u32>(b);
  return static_cast<u64>(ah) * bh + (static_cast<u64>(ah) * bl >> 32) +
         (static_cast<u64>(al) * bh >> 32);
}

// A positive FP64 number's mantissa, leading bit at 63 (zero and subnormal
// numbers: 0), and biased exponent.
__device__ __forceinline__ u64 mantissa(double v, int &exponent) {
  const u64 b = static_cast<u64>(__double_as_longlong(v));
  exponent = static_cast<int>(b >> 52) & 0x7ff;
  return exponent ? (b << 11) | 0x8000000000000000ull : 0ull;
}

// 2^62 / sqrt(a 2^-62) for a in [2^62, 2^64), within 2^-59 of itself and below
// 2^62: the SFU's estimate and one third-order step (as rsqrt64 in FP64), in
// fixed point.
__device__ __forceinline__ u64 inverse_sqrt(u64 a) {
  const float f = static_cast<float>(static_cast<u32>(a >> 32)) * (1.f / (1 << 30));
  const u32 y0 = __float2uint_rz(rsqrt_normal(f) * 4294967296.f);
  const long long e = (1ll << 62) - static_cast<long long>(mulhi(a, static_cast<u64>(y0) * y0));
  const long long t = static_cast<long long>(static_cast<u64>(y0) * static_cast<u32>(e) >> 32) +
                      static_cast<long long>(static_cast<int>(e >> 32)) * y0;
  const long long t2 = static_cast<long long>(static_cast<int>(t >> 12)) * static_cast<int>(e >> 12);
  const u64 y = (static_cast<u64>(y0) << 30) + static_cast<u64>((t >> 1) + ((t2 >> 40) * 3 >> 1));
  return y < (1ull << 62) ? y : (1ull << 62) - 1ull;
}

// A softening length squared, taken apart once per thread.
struct Softening {
  u64 m;
  int e;  // biased exponent
  __device__ __forceinline__ explicit Softening(double eps2) { m = mantissa(eps2, e); }
};

// w = (dx^2 + dy^2 + dz^2 + eps2)^-1/2 and w3 = w^3, each within half a unit in the
// last place and 2^-57 of itself. False outside squares of 2^-300 to 2^300 (and
// for infinities, NaNs and zero distances): work them in FP64.
__device__ __forceinline__ bool inverse_powers(double dx, double dy, double dz,
                                               const Softening &soft, double &w, double &w3) {
  int ex, ey, ez;
  const u64 mx = mantissa(dx, ex), my = mantissa(dy, ey), mz = mantissa(dz, ez);
  // the square of a mantissa has its point below bit 62; all terms are shifted
  // to the largest exponent and two places on, so that their sum fits
  const int ee = soft.e + 1023;  // eps2's exponent on the squares' scale
  const int top = max(max(2 * ex, 2 * ey), max(2 * ez, ee));
  if (static_cast<u32>(top - (2 * 1023 - 300)) > 600u) return false;
  auto term = [&](u64 sq, int e) { return sq >> min(top - e + 2, 63); };
  const u64 sum = term(mulhi(mx, mx), 2 * ex) + term(mulhi(my, my), 2 * ey) +
                  term(mulhi(mz, mz), 2 * ez) + term(soft.m >> 1, ee);
  // r^2 = sum 2^-60 2^(top - 2046) = a 2^-62 4^h with a in [2^62, 2^64)
  const int lead = __clzll(static_cast<long long>(sum));  // 0..3
  const int s = lead - ((top - lead) & 1);                // h is whole
  const u64 a = s >= 0 ? sum << s : sum >> 1;
  const int h = (top - 2044 - s) / 2;
  const u64 y = inverse_sqrt(a);
  w = __longlong_as_double((static_cast<long long>(1021 - h) << 52) +
                           static_cast<long long>((y + (1ull << 8)) >> 9));
  const u64 y1 = y << 2, cube = mulhi(mulhi(y1, y1), y1);
  const int lz = __clzll(static_cast<long long>(cube));
  const u64 c = cube << lz;
  w3 = __longlong_as_double((static_cast<long long>(1021 - lz - 3 * h) << 52) +
                            static_cast<long long>((c >> 11) + ((c >> 10) & 1ull)));
  return true;
}

// 1/sqrt(x) in FP64, for the distances inverse_powers does not take: the SFU's
// estimate y (rsqrt.approx.ftz.f64) and one step of the third-order (Halley)
// iteration: with e = 1 - x y^2 exactly, 1/sqrt(x) = y (1 - e)^(-1/2) = y (1 + e/2
// + 3/8 e^2 + 5/16 e^3 + ...). |e| is at most 1.9e-6 < 2^-18 (on every high word;
// tests/test_rsqrt64.py), so what is left out is below 2^-55; the rounding of x y
// leaves 2^-54 in e / 2, the last one 2^-53: within 2^-52 of the value in all
// (1.24e-16 measured; sqrt and a division round twice). Zero, subnormal,
// negative, infinite and NaN inputs take the plain division.
__device__ __forceinline__ double rsqrt64_estimate(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rsqrt64(double x) {
  const u32 hi = static_cast<u32>(__double2hiint(x));
  if (hi - 0x00100000u >= 0x7fe00000u) return 1.0 / sqrt(x);
  const double y = rsqrt64_estimate(x);
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// ------------------------------------------------- differences in fixed point
//
// Coordinates as 96-bit integers in units of 2^(scale - 1115), `scale` the
// largest biased exponent among those taken together: all 53 bits of a
// coordinate down to 2^-40 of the largest fit, and differences are exact.

struct Fixed {
  u32 w[3];  // two's complement, w[2] highest; below 2^93 in magnitude
};

// False if v has bits below the unit (or is not finite or not normal).
__device__ __forceinline__ bool to_fixed(double v, int scale, Fixed &f) {
  const u32 hi = static_cast<u32>(__double2hiint(v)), lo = static_cast<u32>(__double2loint(v));
  const int e = static_cast<int>(hi >> 20 & 0x7ffu), up = e - scale + 40;
  const bool zero = (hi << 1 | lo) == 0u;
  const u32 mh = zero ? 0u : (hi & 0xfffffu) | 0x100000u;
  const u32 s = static_cast<u32>(up) & 31u;
  const u32 a = lo << s, b = __funnelshift_l(lo, mh, s), c = mh >> 1 >> (31u - s);
  const bool far = up >= 32;
  const u32 x0 = far ? 0u : a, x1 = far ? a : b, x2 = far ? b : c;
  const u32 n = static_cast<u32>(static_cast<int>(hi) >> 31);
  const u64 y = (static_cast<u64>(x1 ^ n) << 32 | (x0 ^ n)) - static_cast<u64>(static_cast<long long>(static_cast<int>(n)));
  f.w[0] = static_cast<u32>(y);
  f.w[1] = static_cast<u32>(y >> 32);
  f.w[2] = (x2 ^ n) + (n != 0u && y == 0ull ? 1u : 0u);
  return zero || (e > 0 && up >= 0 && up <= 40);
}

// |a - b|; negative: 1 if a < b, else 0.
__device__ __forceinline__ Fixed difference(const Fixed &a, const Fixed &b, u32 &negative) {
  Fixed d;
  asm("sub.cc.u32 %0, %3, %6;\n\t"
      "subc.cc.u32 %1, %4, %7;\n\t"
      "subc.u32 %2, %5, %8;"
      : "=r"(d.w[0]), "=r"(d.w[1]), "=r"(d.w[2])
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]));
  negative = d.w[2] >> 31;
  const u32 n = 0u - negative;
  Fixed m;
  asm("add.cc.u32 %0, %3, %6;\n\t"
      "addc.cc.u32 %1, %4, 0;\n\t"
      "addc.u32 %2, %5, 0;"
      : "=r"(m.w[0]), "=r"(m.w[1]), "=r"(m.w[2])
      : "r"(d.w[0] ^ n), "r"(d.w[1] ^ n), "r"(d.w[2] ^ n), "r"(negative));
  return m;
}

// A magnitude as FP64, rounded to nearest (ties away from zero). False if it is
// below 2^-29 of the scale and not zero.
__device__ __forceinline__ bool from_fixed(const Fixed &d, u32 negative, int scale, double &v) {
  const u32 a = d.w[2];
  const int lz = __clz(static_cast<int>(a));
  const u32 hi = __funnelshift_l(d.w[1], a, lz), lo = __funnelshift_l(d.w[0], d.w[1], lz);
  const u32 e = static_cast<u32>(scale + 2 - lz) << 20 | negative << 31;  // (leading bit added)
  u32 r0, r1;
  asm("{\n\t.reg .u32 t;\n\t"
      "add.cc.u32 t, %2, 0x80000000;\n\t"
      "addc.cc.u32 %0, %3, 0;\n\t"
      "addc.u32 %1, %4, %5;\n\t}"
      : "=r"(r0), "=r"(r1)
      : "r"(lo << 21), "r"(__funnelshift_r(lo, hi, 11)), "r"(hi >> 11), "r"(e));
  v = __hiloint2double(static_cast<int>(a != 0u ? r1 : 0u), static_cast<int>(r0));
  return a != 0u || (d.w[1] | d.w[0]) == 0u;
}

// A mass's mantissa and exponent; e = 0 marks one that is not taken (see below).
struct Mass {
  u64 m;
  u32 e, sign;
};
constexpr int kScaleSpan = 200, kMassSpan = 300;  // exponents about zero that are taken
__device__ __forceinline__ Mass to_mass(double v) {
  const u32 hi = static_cast<u32>(__double2hiint(v));
  const u32 e = hi >> 20 & 0x7ffu;
  int unused;
  const u64 m = mantissa(fabs(v), unused);
  return Mass{m, e - (1023u - kMassSpan) < 2u * kMassSpan ? e : 0u, hi & 0x80000000u};
}

// Softening in the units of squared differences, once per scale: the largest
// shift of the differences that leaves it room (negative: none does).
struct FixedSoftening {
  u64 m;
  int q, most;
  __device__ __forceinline__ FixedSoftening(const Softening &s, int scale)
      : m(s.m), q(2 * scale - 1016 - s.e), most(s.m ? (2 * scale - 1020 - s.e) >> 1 : 64) {}
};

// From the differences d of two bodies: w = (d^2 + eps2)^-1/2 and gm3 = mass w^3,
// each within half a unit in the last place and 2^-55 of itself. False if the
// bodies are too close for their unit.
__device__ __forceinline__ bool pair_powers(const Fixed &x, const Fixed &y, const Fixed &z,
                                            const FixedSoftening &soft, const Mass &mass,
                                            int scale, double &w, double &gm3) {
  // The differences to 62 bits, the largest (or the softening) leading: 64 bits
  // of their squares' sum without l l, whose three are below a unit each. It is
  // 2^58 to 2^62.
  const int up = min(__clz(static_cast<int>(x.w[2] | y.w[2] | z.w[2])) - 2, soft.most);
  if (up > 29) return false;
  u64 hh = 0, hl = 0;
  auto add = [&](const Fixed &d) {
    const u32 h = __funnelshift_l(d.w[1], d.w[2], up), l = __funnelshift_l(d.w[0], d.w[1], up);
    hh += static_cast<u64>(h) * h;
    hl += static_cast<u64>(h) * l;
  };
  add(x);
  add(y);
  add(z);
  const u64 sum = hh + (hl >> 31) + (soft.m >> min(soft.q - 2 * up, 63));
  // r^2 = a 2^-62 4^h with a in [2^62, 2^64)
  const int s = __clz(static_cast<int>(sum >> 32)) & ~1;
  const int h = scale - 1020 - up - (s >> 1);
  const u64 r = inverse_sqrt(sum << s);
  w = __longlong_as_double((static_cast<long long>(1021 - h) << 52) +
                           static_cast<long long>((r + (1ull << 8)) >> 9));
  const u64 r1 = r << 2, g = mulhi(mulhi(mulhi(r1, r1), r1), mass.m);  // >= 2^59
  const int lz = __clz(static_cast<int>(g >> 32));
  const u64 c = g << lz;
  const u64 v = (c >> 11) + ((c >> 10) & 1ull);
  const int e = static_cast<int>(mass.e) - 1 - lz - 3 * h;
  gm3 = __hiloint2double(
      static_cast<int>((static_cast<u32>(v >> 32) + (static_cast<u32>(e) << 20)) | mass.sign),
      static_cast<int>(static_cast<u32>(v)));
  return true;
}

// ------------------------------------------- the same roundings as FP64's
//
// Products and 1/sqrt rounded as FP64 rounds them (to nearest, ties to even),
// bit for bit, on the integer pipes: about 22 instructions for a product and
// 80 for the root and the quotient, against the time of 64 and of some 1600 on
// the FP64 pipe. For normal numbers and zeros (whose products are +0); the
// caller sees to it that no product leaves the normal range. Factors are kept
// as 53-bit mantissas: their product's point then moves by 11 or 12 places,
// one funnel shift a word, and signs and exponents add up in one word.

struct Factor {
  u32 hi, lo;  // 53-bit mantissa; 0 for zero
  u32 se;      // sign and exponent where a double has them, less the leading bit
};

template <bool kNonZero = false>
__device__ __forceinline__ Factor factor(double v) {
  const u32 hi = static_cast<u32>(__double2hiint(v)), lo = static_cast<u32>(__double2loint(v));
  const u32 m = (hi & 0xfffffu) | 0x100000u;
  // (a comparison of all 64 bits with zero would be made on the FP64 pipe)
  return Factor{kNonZero || (hi << 1) != 0u ? m : 0u, lo, hi - m};
}

template <bool kNonZero = false>
__device__ __forceinline__ double product(const Factor &a, const Factor &b) {
  const u64 t0 = static_cast<u64>(a.lo) * b.lo;
  const u64 t1 = static_cast<u64>(a.hi) * b.lo + (t0 >> 32);
  const u64 t2 = static_cast<u64>(a.lo) * b.hi + t1;
  const u64 t3 = static_cast<u64>(a.hi) * b.hi + (t2 >> 32);
  const u32 p0 = static_cast<u32>(t0), p1 = static_cast<u32>(t2), p2 = static_cast<u32>(t3),
            p3 = static_cast<u32>(t3 >> 32);  // leading bit at 8 or 9, unless zero
  const u32 up = p3 >> 9, s = 12u - up;
  const u32 high = __funnelshift_l(p2, p3, s), low = __funnelshift_l(p1, p2, s);
  const u32 rest = __funnelshift_l(p0, p1, s);
  // ties to even: behind an odd number the half counts as more
  const u32 more = p0 << s | (low & 1u);
  u32 hi, lo;
  asm("{\n\t.reg .u32 t;\n\t"
      "add.cc.u32 t, %2, 0xffffffff;\n\t"    // carry: more != 0
      "addc.cc.u32 t, %3, 0x7fffffff;\n\t"   // carry: above the half
      "addc.cc.u32 %0, %4, 0;\n\t"
      "addc.u32 %1, %5, %6;\n\t}"
      : "=r"(lo), "=r"(hi)
      : "r"(more), "r"(rest), "r"(low), "r"(high), "r"(a.se + b.se + ((up - 1022u) << 20)));
  if (!kNonZero && p3 == 0u) hi = 0u;
  return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
}

// The high word of 2^kExp, its sign shifted out. above<kExp> gathers how far |v|'s
// lies above it, the largest of several: 0 <= v < 2^(kExp + n) or v = 0 for all
// of them if that is below kWord<kExp + n> - kWord<kExp>.
template <int kExp>
constexpr u32 kWord = static_cast<u32>(kExp + 1023) << 21;
template <int kExp>
__device__ __forceinline__ u32 above(double v, u32 most) {
  const u32 k = static_cast<u32>(__double2hiint(v)) << 1, l =
      static_cast<u32>(__double2loint(v));
  return (k | l) == 0u ? most : max(most, k - kWord<kExp>);
}

// 1 / sqrt(x), the root and the quotient each rounded, for a normal x > 0. Each rounding takes the
// candidate below an estimate good to 2^-58 and compares it with the midpoint
// above it exactly, in the low 64 bits of a difference that is known to be small.
__device__ __forceinline__ double recip_sqrt(double x) {
  int ex;
  const u64 m = mantissa(x, ex);
  const int odd = (ex - 1023) & 1;
  const u64 a = odd ? m : m >> 1;  // x = a 2^-62 4^h
  const int h = (ex - 1023 - odd) / 2;
  const u64 y = inverse_sqrt(a);
  // s = sqrt(a 2^-62) in units of 2^-52
  const u64 f = mulhi(a, y << 2) >> 10, mid = 2ull * f + 1ull;
  const u64 s = f + (static_cast<long long>((a << 44) - mid * mid) > 0 ? 1ull : 0ull);
  // 1 / s in units of 2^-53: y and the Newton step that turns 1/sqrt into 1/s
  const long long d = -static_cast<long long>(s * y);
  const u64 r = y + static_cast<u64>(static_cast<long long>(y >> 32) *
                                     static_cast<int>(d >> 32) >> 50);
  const u64 g = r >> 9, mid2 = 2ull * g + 1ull;
  const u64 i = g + (-static_cast<long long>(s * mid2) > 0 ? 1ull : 0ull);
  return __longlong_as_double((static_cast<long long>(1021 - h) << 52) +
                              static_cast<long long>(i));
}

}  // namespace gtc
