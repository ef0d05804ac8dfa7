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
  // y = 2^62 / sqrt(a 2^-62): the SFU's estimate and one third-order step, as
  // rsqrt64 in FP64, in fixed point
  const float f = static_cast<float>(static_cast<u32>(a >> 32)) * (1.f / (1 << 30));
  const u32 y0 = __float2uint_rz(rsqrt_normal(f) * 4294967296.f);
  const long long e = (1ll << 62) - static_cast<long long>(mulhi(a, static_cast<u64>(y0) * y0));
  const long long t = static_cast<long long>(static_cast<u64>(y0) * static_cast<u32>(e) >> 32) +
                      static_cast<long long>(static_cast<int>(e >> 32)) * y0;
  const long long t2 = static_cast<long long>(static_cast<int>(t >> 12)) * static_cast<int>(e >> 12);
  const u64 y = min((static_cast<u64>(y0) << 30) + (t >> 1) + ((t2 >> 40) * 3 >> 1),
                    (1ull << 62) - 1ull);
  w = __longlong_as_double((static_cast<long long>(1021 - h) << 52) +
                           static_cast<long long>((y + (1ull << 8)) >> 9));
  const u64 y1 = y << 2, cube = mulhi(mulhi(y1, y1), y1);
  const int lz = __clzll(static_cast<long long>(cube));
  const u64 c = cube << lz;
  w3 = __longlong_as_double((static_cast<long long>(1021 - lz - 3 * h) << 52) +
                            static_cast<long long>((c >> 11) + ((c >> 10) & 1ull)));
  return true;
}

}  // namespace gtc
