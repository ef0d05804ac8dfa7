// The walks' opening test (group_lists.cpp:145-154): FP64 exactly as the
// reference computes it, and an FP32 form with a rigorous error band that
// decides almost every test and leaves the rest to FP64. Users are compiled
// with -fmad=false.
#pragma once

#include "pipeline.cuh"

namespace gtc {

// The opening test of group_lists.cpp:145-154 for one node, in FP64 exactly
// as the reference computes it.
__device__ __forceinline__ bool accept64(const WalkRec64 &r, const double *gc, const double *gh) {
  bool overlap = true;
  double d2 = 0.0;
  if (fabs(r.cx - gc[0]) > r.slack + gh[0]) overlap = false;
  double d = fabs(r.mx - gc[0]) - gh[0];
  if (d > 0) d2 += d * d;
  if (fabs(r.cy - gc[1]) > r.slack + gh[1]) overlap = false;
  d = fabs(r.my - gc[1]) - gh[1];
  if (d > 0) d2 += d * d;
  if (fabs(r.cz - gc[2]) > r.slack + gh[2]) overlap = false;
  d = fabs(r.mz - gc[2]) - gh[2];
  if (d > 0) d2 += d * d;
  return !overlap && d2 > r.crit2;
}

// The same test in FP32 with a rigorous error band. Every FP32 input is the
// FP64 quantity (relative to the root centre) rounded once; the node record
// carries B_n >= all its |values| + slack and the group B_g >= max|centre| +
// max half-extent, so with B = B_n + B_g every FP32 difference formed below is
// within 8 * 2^-24 B of the value from the exact inputs (three rounded inputs,
// two or three operations on values up to 2 B), half of E = 2^-20 B:
// * overlap: on every axis |c - g| - gh <= slack (group_lists.cpp:147), so the
//   largest of the three decides, outside a band of E;
// * the distance from the box to the centre of mass (:150-151): d^2 is the sum
//   of squares of v_a = max(|m - g| - gh, 0), each within E / 2 of its exact
//   value, so d^2 is within E (v_x + v_y + v_z) + E^2 of the exact one, plus a few
//   2^-24 of itself, which the factors (1 +- 2^-18) cover with the rounding of
//   crit^2. (A lower and an upper bound per axis took half as many
//   instructions again.)
// All of which needs squares that FP32 holds: an infinite d^2 is no proof of a
// large one, as its tolerance is finite (lengths near sqrt(FLT_MAX) = 1.84e19 in
// a tree of 1e23 and more), and below some 1e-37 a rounding may be a subnormal's.
// So d^2 + tol past kFarSquare or below kNearSquare is left to FP64. (Between them
// the tree's bounds are above 1e-15, its E and tolerance normal; an overflown
// crit^2 is the larger, a lost one the smaller; and centres, boxes or bounds that
// overflow have an infinite tolerance. With bounds for E and crit^2 beside this one
// a walk of 1M bodies has 2% more instructions, 325 M for 319 M.)
// A comparison outside its band then has the FP64 outcome; otherwise the caller
// runs the FP64 test. Returns 1 accept, 0 open, 2 undecided (NaNs end up
// undecided).
constexpr float kBand = 1.0f / (1 << 20);
constexpr float kNearSquare = 1e-35f, kFarSquare = 1e38f;

__device__ __forceinline__ int accept32(const WalkRec32 &r, const float *gf, const float *hf,
                                        float gbound) {
  const float e = kBand * (r.bound + gbound);
  const float over = fmaxf(fmaxf(fabsf(r.cx - gf[0]) - hf[0], fabsf(r.cy - gf[1]) - hf[1]),
                           fabsf(r.cz - gf[2]) - hf[2]) - r.slack;
  const float vx = fmaxf(fabsf(r.mx - gf[0]) - hf[0], 0.f),
              vy = fmaxf(fabsf(r.my - gf[1]) - hf[1], 0.f),
              vz = fmaxf(fabsf(r.mz - gf[2]) - hf[2], 0.f);
  const float d2 = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
  const float tol = e * (vx + vy + vz + e);
  const float c2 = r.crit2;
  const bool apart = d2 - tol > c2 * (1.f + 4.f * kBand);   // farther than crit for sure
  const bool close = d2 + tol < c2 * (1.f - 4.f * kBand);   // nearer for sure
  const bool held = d2 + tol >= kNearSquare && d2 + tol <= kFarSquare;
  return !held ? 2 : over < -e || close ? 0 : over > e && apart ? 1 : 2;
}

__device__ __forceinline__ WalkRec32 load32(const WalkRec32 *w, u32 i) {
  const float4 *p = reinterpret_cast<const float4 *>(w + i);
  const float4 a = __ldg(p), b = __ldg(p + 1);
  const uint4 c = __ldg(reinterpret_cast<const uint4 *>(p + 2));
  WalkRec32 r;
  r.cx = a.x;
  r.cy = a.y;
  r.cz = a.z;
  r.slack = a.w;
  r.mx = b.x;
  r.my = b.y;
  r.mz = b.z;
  r.crit2 = b.w;
  r.skip = c.x;
  r.nbody_leaf = c.y;
  r.begin = c.z;
  r.bound = __uint_as_float(c.w);
  return r;
}

__device__ __forceinline__ WalkRec64 load64(const WalkRec64 *w, u32 i) {
  const double2 *p = reinterpret_cast<const double2 *>(w + i);
  const double2 a0 = __ldg(p), a1 = __ldg(p + 1), b0 = __ldg(p + 2), b1 = __ldg(p + 3);
  return WalkRec64{a0.x, a0.y, a1.x, a1.y, b0.x, b0.y, b1.x, b1.y};
}

}  // namespace gtc
