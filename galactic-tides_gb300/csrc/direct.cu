// Direct summation: the tiled FP32 kernel that replaces the reference's
// gt_direct (src/metal/gravity_kernels.metal:18-43; arithmetic of gt_body,
// gravity_kernels.h:71-83), and an FP64 kernel for a sample of targets, the
// accuracy judge of the reference bench (apps/galactic_tides_bench.cpp:74-95)
// and compute_gravity_direct (src/gravity.cpp:28-45).

#include <algorithm>

#include "pipeline.cuh"
#include "wide.cuh"

namespace gtc {
namespace {

// ------------------------------------------------------------------ FP32

constexpr int kDT = 128;          // threads per block = sources per shared tile
constexpr float kFar = 1e15f;     // padding source: far away, zero mass, adds exactly 0

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// Two sources (one in each half of a float2) against one target: FFMA2 /
// FMUL2 / FADD2 do both at once, the two rsqrts go to the SFU. The source
// pair is (x0, x1, y0, y1), (z0, z1, Gm0, Gm1); the target's coordinates are
// negated and doubled (-x, -x). With kMask, `skip` zeroes the half whose
// source is the target itself (the reference skips j == i), before its
// singular 1/r can reach the sums.
template <bool kMask>
__device__ __forceinline__ void add_pair(const float4 s0, const float4 s1, const float2 nx,
                                         const float2 ny, const float2 nz, const float2 e2,
                                         float2 &ax, float2 &ay, float2 &az, float2 &pt,
                                         bool skip0 = false, bool skip1 = false) {
  const float2 dx = __fadd2_rn(f2(s0.x, s0.y), nx);  // source - target
  const float2 dy = __fadd2_rn(f2(s0.z, s0.w), ny);
  const float2 dz = __fadd2_rn(f2(s1.x, s1.y), nz);
  const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
  // (r^2 >= eps^2; without softening only pairs closer than ~1e-19 could
  // give a subnormal r^2, whose 1/r is meaningless either way)
  float2 inv = f2(rsqrt_normal(r2.x), rsqrt_normal(r2.y));
  if (kMask) {
    inv.x = skip0 ? 0.f : inv.x;
    inv.y = skip1 ? 0.f : inv.y;
  }
  const float2 gm = __fmul2_rn(f2(s1.z, s1.w), inv);
  const float2 gm3 = __fmul2_rn(gm, __fmul2_rn(inv, inv));
  ax = __ffma2_rn(gm3, dx, ax);
  ay = __ffma2_rn(gm3, dy, ay);
  az = __ffma2_rn(gm3, dz, az);
  pt = __fadd2_rn(pt, gm);
}

// Block (bx, by) owns targets [bx kR kDT, (bx + 1) kR kDT) -- thread t the
// targets bx kR kDT + r kDT + t, r < kR (the tile shape: more targets per
// thread reuse each staged source more, fewer leave registers for more
// warps) -- and sums the sources of slice by,
// [by len, (by + 1) len), streamed through shared memory in index order,
// kDT at a time. Even and odd sources go to the two halves of each sum.
// Only the tiles holding the block's own targets test j == i. With one
// slice the sums go straight to `out`, otherwise to part[by][target],
// added up in slice order by k_direct_sum (deterministic).
template <int kDR>
__global__ void __launch_bounds__(kDT)
    k_direct(const float4 *__restrict__ bodies, u32 n, u32 len, float G, float eps2,
             float4 *__restrict__ out) {
  grid_wait();
  constexpr u32 kDTB = kDT * kDR;  // targets per block
  __shared__ float4 tile[kDT];  // kDT / 2 source pairs, two float4 each
  const u32 t0 = blockIdx.x * kDTB;
  const u32 j0 = blockIdx.y * len, j1 = min(n, j0 + len);
  const float2 e2 = f2(eps2, eps2);
  u32 ti[kDR];
  float2 nx[kDR], ny[kDR], nz[kDR], ax[kDR], ay[kDR], az[kDR], pt[kDR];
#pragma unroll
  for (int r = 0; r < kDR; ++r) {
    ti[r] = t0 + r * kDT + threadIdx.x;
    const float4 p = ti[r] < n ? bodies[ti[r]] : make_float4(0.f, 0.f, 0.f, 0.f);
    nx[r] = f2(-p.x, -p.x);
    ny[r] = f2(-p.y, -p.y);
    nz[r] = f2(-p.z, -p.z);
    ax[r] = ay[r] = az[r] = pt[r] = f2(0.f, 0.f);
  }
  float *tf = reinterpret_cast<float *>(tile);
  const u32 pair = threadIdx.x >> 1, half = threadIdx.x & 1;
  for (u32 base = j0; base < j1; base += kDT) {
    const u32 j = base + threadIdx.x;
    const float4 b = j < j1 ? bodies[j] : make_float4(kFar, kFar, kFar, 0.f);
    tf[8 * pair + half] = b.x;
    tf[8 * pair + 2 + half] = b.y;
    tf[8 * pair + 4 + half] = b.z;
    tf[8 * pair + 6 + half] = G * b.w;
    __syncthreads();
    const bool own = base < t0 + kDTB && base + kDT > t0;
    if (!own) {
#pragma unroll 4
      for (int q = 0; q < kDT / 2; ++q) {
        const float4 s0 = tile[2 * q], s1 = tile[2 * q + 1];
#pragma unroll
        for (int r = 0; r < kDR; ++r)
          add_pair<false>(s0, s1, nx[r], ny[r], nz[r], e2, ax[r], ay[r], az[r], pt[r]);
      }
    } else {
      for (int q = 0; q < kDT / 2; ++q) {
        const float4 s0 = tile[2 * q], s1 = tile[2 * q + 1];
        const u32 js = base + 2 * q;
#pragma unroll
        for (int r = 0; r < kDR; ++r)
          add_pair<true>(s0, s1, nx[r], ny[r], nz[r], e2, ax[r], ay[r], az[r], pt[r],
                         ti[r] == js, ti[r] == js + 1);
      }
    }
    __syncthreads();
  }
  float4 *dst = out + static_cast<u64>(blockIdx.y) * n;
#pragma unroll
  for (int r = 0; r < kDR; ++r)
    if (ti[r] < n)
      dst[ti[r]] = make_float4(ax[r].x + ax[r].y, ay[r].x + ay[r].y, az[r].x + az[r].y,
                               -(pt[r].x + pt[r].y));
}

// out[i] = the sum of the slices' partial sums of target i, in slice order.
__global__ void k_direct_sum(const float4 *__restrict__ part, u32 n, u32 slices,
                             float4 *__restrict__ out) {
  grid_wait();
  const u32 i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  float4 a = part[i];
  for (u32 k = 1; k < slices; ++k) {
    const float4 v = part[static_cast<u64>(k) * n + i];
    a.x += v.x;
    a.y += v.y;
    a.z += v.z;
    a.w += v.w;
  }
  out[i] = a;
}

// ------------------------------------------------------------------ FP64

constexpr int kST = 128;   // sample targets per block

__device__ __forceinline__ u64 min_u64(u64 a, u64 b) { return a < b ? a : b; }

struct alignas(16) Body64 {
  Fixed p[3];
  Mass mass;  // G times the mass, taken apart; e = 0: not worked in fixed point
  double m;
};

// What a source adds to its target, in FP64 coordinates: for tiles and bodies
// that their tile's fixed point does not hold.
struct Pair64 {
  double dx, dy, dz, w, gm3;
};
__device__ __noinline__ void pair64(const double *__restrict__ source, double px, double py,
                                    double pz, double m, const Softening &soft, double eps2,
                                    Pair64 &o) {
  o.dx = px - source[0];
  o.dy = py - source[1];
  o.dz = pz - source[2];
  double w3;  // 1/r^3
  if (!inverse_powers(o.dx, o.dy, o.dz, soft, o.w, w3)) {
    o.w = rsqrt64(fma(o.dx, o.dx, fma(o.dy, o.dy, fma(o.dz, o.dz, eps2))));
    w3 = o.w * o.w * o.w;
  }
  o.gm3 = m * w3;
}

// Partial sums of targets idx[blockIdx.x*kST + t] over the source slice
// blockIdx.y; slices are reduced in order afterwards (deterministic).
//
// A tile's coordinates and the targets' are kept as 96-bit integers of the
// tile's largest exponent; an interaction is worked in integers from the
// differences to G m / r^3 and issues four FP64 instructions, its additions
// (wide.cuh). Bound: the FP64 pipe (16 cycles of an SM per warp instruction)
// and the integer pipes. 4096 targets x 500k bodies: 102.4 ms with sqrt and
// division (26 FP64 instructions), 66.1 ms with rsqrt64 (18), 30.1 ms with
// 1/r and 1/r^3 in integers (8), 21.1 ms so: both pipes about 65% busy. Fewer
// registers (48) 22.2 ms; the loop unrolled measures the same.
__global__ void __launch_bounds__(kST)
    k_direct64(const double *__restrict__ pos, const double *__restrict__ mass, u64 n,
               const u64 *__restrict__ idx, u64 m, u64 slice, double G, double eps2,
               double2 *part) {
  grid_wait();
  __shared__ Body64 tile[kST];
  __shared__ u32 largest[kST / 32];
  const u64 s = static_cast<u64>(blockIdx.x) * kST + threadIdx.x;
  const bool active = s < m;
  const u64 i = active ? idx[s] : ~0ull;
  double px = 0, py = 0, pz = 0;
  if (active) {
    px = pos[3 * i];
    py = pos[3 * i + 1];
    pz = pos[3 * i + 2];
  }
  auto exponent = [](double v) { return static_cast<u32>(__double2hiint(v)) >> 20 & 0x7ffu; };
  const u32 own = max(exponent(px), max(exponent(py), exponent(pz)));
  double ax = 0, ay = 0, az = 0, phi = 0;
  const Softening soft(eps2);
  const u64 j0 = static_cast<u64>(blockIdx.y) * slice;
  const u64 j1 = min_u64(n, j0 + slice);
  for (u64 base = j0; base < j1; base += kST) {
    const u64 j = base + threadIdx.x;
    double bx = 0, by = 0, bz = 0, bm = 0;
    if (j < j1) {
      bx = pos[3 * j];
      by = pos[3 * j + 1];
      bz = pos[3 * j + 2];
      bm = G * mass[j];
    }
    const u32 e = max(own, max(exponent(bx), max(exponent(by), exponent(bz))));
    const u32 wide = __reduce_max_sync(kFullMask, e);
    if ((threadIdx.x & 31) == 0) largest[threadIdx.x >> 5] = wide;
    __syncthreads();  // (the tile is free: the last one's end is behind a barrier)
    u32 most = largest[0];
#pragma unroll
    for (int k = 1; k < kST / 32; ++k) most = max(most, largest[k]);
    const int scale = static_cast<int>(most);
    Body64 own_body;
    own_body.mass = to_mass(bm);
    own_body.m = bm;
    const bool held = to_fixed(bx, scale, own_body.p[0]) & to_fixed(by, scale, own_body.p[1]) &
                      to_fixed(bz, scale, own_body.p[2]);
    if (!held) own_body.mass.e = 0u;
    tile[threadIdx.x] = own_body;
    Fixed tx, ty, tz;
    const FixedSoftening fs(soft, scale);
    const bool fixed = (to_fixed(px, scale, tx) & to_fixed(py, scale, ty) &
                        to_fixed(pz, scale, tz)) &&
                       most - (1023u - kScaleSpan) < 2u * kScaleSpan && fs.most >= 0;
    __syncthreads();
    const u32 cnt = static_cast<u32>(min_u64(kST, j1 - base));
    // the target's place in this tile (past it: none)
    const u32 self = i - base < kST ? static_cast<u32>(i - base) : kST;
    for (u32 k = 0; k < cnt; ++k) {
      if (k == self) continue;
      const Body64 &b = tile[k];
      const Mass bm = b.mass;
      Pair64 o;
      bool done = false;
      if (fixed && bm.e != 0u) {
        u32 nx, ny, nz;
        const Fixed x = difference(tx, b.p[0], nx), y = difference(ty, b.p[1], ny),
                    z = difference(tz, b.p[2], nz);
        done = pair_powers(x, y, z, fs, bm, scale, o.w, o.gm3);
        done &= from_fixed(x, nx, scale, o.dx) & from_fixed(y, ny, scale, o.dy) &
                from_fixed(z, nz, scale, o.dz);
      }
      if (!done) {
        Pair64 slow;
        pair64(pos + 3 * (base + k), px, py, pz, b.m, soft, eps2, slow);
        o = slow;
      }
      ax = fma(-o.gm3, o.dx, ax);
      ay = fma(-o.gm3, o.dy, ay);
      az = fma(-o.gm3, o.dz, az);
      phi = fma(-b.m, o.w, phi);
    }
    __syncthreads();
  }
  if (active) {
    double2 *o = part + 2 * (static_cast<u64>(blockIdx.y) * m + s);
    o[0] = make_double2(ax, ay);
    o[1] = make_double2(az, phi);
  }
}

__global__ void k_direct64_sum(const double2 *part, u64 m, u32 slices, double *acc, double *pot) {
  grid_wait();
  const u64 s = static_cast<u64>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (s >= m) return;
  double ax = 0, ay = 0, az = 0, phi = 0;
  for (u32 k = 0; k < slices; ++k) {
    const double2 *v = part + 2 * (static_cast<u64>(k) * m + s);
    ax += v[0].x;
    ay += v[0].y;
    az += v[1].x;
    phi += v[1].y;
  }
  acc[3 * s] = ax;
  acc[3 * s + 1] = ay;
  acc[3 * s + 2] = az;
  pot[s] = phi;
}

}  // namespace

void direct_fp32(const float4 *bodies, u32 n, float G, float eps2, float4 *out,
                 DeviceBuffer &scratch, cudaStream_t s, int targets) {
  if (n == 0) return;
  if (targets != 2 && targets != 4) throw InvalidArgument("direct_targets must be 2 or 4");
  int dev = 0, sms = 0;
  GTC_CUDA(cudaGetDevice(&dev));
  GTC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // Slices: enough (target block, source slice) units for 16 per SM, so that all
  // are busy, and as far as the partial sums stay small beside the work (n / 2000
  // slices) up to 96, so that the last ones end close together; two tiles each
  // at least. 3001 bodies 57 -> 29 us (8 tiles each at least before), 20k 192 us
  // from 18 to 78 slices, 50k 1.037 ms with 13, 1.022 with 25, 200k 16.30 with 4,
  // 15.94 with 6, 15.72 with 20 and more.
  const u32 tiles = ceil_div(n, kDT * static_cast<u32>(targets));
  auto per_sm = [&](u32 units) { return ceil_div(units * static_cast<u32>(sms), tiles); };
  u32 slices = std::max(per_sm(16), std::min(per_sm(96), n / 2000));
  slices = std::min(slices, ceil_div(n, 2 * kDT));
  const u32 len = ceil_div(ceil_div(n, slices), kDT) * kDT;
  slices = ceil_div(n, len);
  float4 *dst = out;
  if (slices > 1) {
    scratch.ensure(static_cast<u64>(slices) * n * sizeof(float4));
    dst = scratch.as<float4>();
  }
  if (targets == 4)
    launch(k_direct<4>, dim3(tiles, slices), kDT, 0, s, bodies, n, len, G, eps2, dst);
  else
    launch(k_direct<2>, dim3(tiles, slices), kDT, 0, s, bodies, n, len, G, eps2, dst);
  GTC_LAUNCH_CHECK();
  if (slices > 1) {
    launch(k_direct_sum, ceil_div(n, 256), 256, 0, s, dst, n, slices, out);
    GTC_LAUNCH_CHECK();
  }
}

Fp64SamplePlan plan_fp64_sample(u64 n, u64 m, int sms, u64 max_pairs) {
  const u64 tb = (m + kST - 1) / kST;
  u64 slices = std::max<u64>(1, (8ull * static_cast<u64>(sms) + tb - 1) / tb);
  slices = std::min<u64>(slices, std::max<u64>(1, n / kST));
  slices = std::min<u64>(slices, std::max<u64>(1, max_pairs / std::max<u64>(1, m)));
  const u64 slice = std::max<u64>(1, (n + slices - 1) / slices);
  return {std::max<u64>(1, (n + slice - 1) / slice), slice};
}

void launch_fp64_sample(const double *pos, const double *mass, u64 n, const u64 *idx, u64 m,
                        double G, double eps, const Fp64SamplePlan &plan, double2 *part,
                        double *acc, double *pot, cudaStream_t s) {
  dim3 grid(ceil_div(m, kST), static_cast<u32>(plan.slices));
  launch(k_direct64, grid, kST, 0, s, pos, mass, n, idx, m, plan.slice, G, eps * eps, part);
  GTC_LAUNCH_CHECK();
  launch(k_direct64_sum, ceil_div(m, 256), 256, 0, s, part, m, static_cast<u32>(plan.slices),
         acc, pot);
  GTC_LAUNCH_CHECK();
}

void direct_fp64_sample(const double *pos, const double *mass, u64 n, const u64 *idx, u64 m,
                        double G, double eps, double *acc, double *pot, DeviceBuffer &scratch,
                        cudaStream_t s) {
  if (m == 0) return;
  int dev = 0, sms = 0;
  GTC_CUDA(cudaGetDevice(&dev));
  GTC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const Fp64SamplePlan plan = plan_fp64_sample(n, m, sms, ~0ull);
  scratch.ensure(plan.slices * m * 2 * sizeof(double2));
  launch_fp64_sample(pos, mass, n, idx, m, G, eps, plan, scratch.as<double2>(), acc, pot, s);
}

}  // namespace gtc

namespace gtc {
namespace {

// Eight independent FMA chains per thread, long enough to hide latency.
__global__ void __launch_bounds__(256) k_fma_peak(float *sink, int iters, float a, float b) {
  grid_wait();
  float x[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) x[k] = threadIdx.x * 1e-3f + k;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = fmaf(x[k], a, b);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += x[k];
  if (s == 12345.678f) sink[threadIdx.x] = s;  // keeps the chains live
}

}  // namespace

double fp32_peak_tflops(cudaStream_t s) {
  int dev = 0, sms = 0;
  GTC_CUDA(cudaGetDevice(&dev));
  GTC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  DeviceBuffer sink;
  sink.ensure(256 * sizeof(float));
  const int iters = 1 << 14;
  const u32 blocks = static_cast<u32>(sms) * 8;
  cudaEvent_t a, b;
  GTC_CUDA(cudaEventCreate(&a));
  GTC_CUDA(cudaEventCreate(&b));
  float best = 1e30f;
  for (int rep = 0; rep < 4; ++rep) {
    GTC_CUDA(cudaEventRecord(a, s));
    launch(k_fma_peak, blocks, 256, 0, s, sink.as<float>(), iters, 0.999f, 1e-3f);
    GTC_LAUNCH_CHECK();
    GTC_CUDA(cudaEventRecord(b, s));
    GTC_CUDA(cudaEventSynchronize(b));
    float ms = 0.f;
    GTC_CUDA(cudaEventElapsedTime(&ms, a, b));
    if (rep > 0) best = std::min(best, ms);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  sink.release();
  const double flops = 2.0 * 8.0 * iters * 256.0 * blocks;
  return flops / (best * 1e-3) / 1e12;
}

}  // namespace gtc
