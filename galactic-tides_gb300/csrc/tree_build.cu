// Octree build on the device, bit-identical to the reference's CPU build
// (src/octree.cpp:169-273). Compiled with -fmad=false: every FP64 product
// and sum below rounds separately, as in the reference's x86-64 build.
//
// The reference splits a node at its centre c (body goes up on an axis when
// p >= c) and makes each child's centre c +- h/2, recursively, with a stable
// counting sort. Here every body replays that chain of comparisons and
// additions on its own, writing the octant of every level as a 3-bit digit
// of a key (21 levels per 64-bit word), and one stable radix sort of the
// keys reproduces the reference's tree order. The tree's shape follows from
// the sorted keys alone:
//   * lcp(a, b): the number of leading levels two bodies share;
//   * a node of depth d holds more than L = leaf_size bodies iff some run of
//     L+1 consecutive sorted bodies shares d levels, so a body's leaf depth is
//     1 + max lcp over the L+1 windows that contain it, capped by depth 60 and
//     by the reference's "tiny node" rule (octree.cpp:40-44);
//   * the nodes that end at sorted position b are the depths
//     lcp(b, b+1) < d <= leafdepth(b).
// Numbering nodes by (end descending, depth ascending) gives exactly the
// order in which the reference's group walk pops them (group_lists.cpp:
// 141-164), so each node's subtree is a contiguous index range and a
// "skip" link replaces the walk's stack. Bodies deeper than 21 levels (dense
// clumps, coincident points) get further key words in up to two more rounds,
// sorted within their depth-21 (or 42) node.
//
// Inside a leaf the reference keeps bodies in input order (its sort is
// stable and leaves are not split further), so each leaf's range is put back
// in input order before the moments are taken. Moments are FP64, leaves
// summed in tree order and parents from their children in octant order
// (octree.cpp:46-102), bottom-up with one arrival counter per node.

#include <algorithm>
#include <cstddef>
#include <cstring>

#include "pipeline.cuh"

namespace gtc {
namespace {

constexpr int kT = 256;

// Graph replays pass the abort word of their Scalars and the node count on
// the device; eager calls pass null and their host-known sizes.
__device__ __forceinline__ bool aborted(const u32 *abort) { return abort && *abort; }
__device__ __forceinline__ u32 bounded(u32 cap, const u32 *dev) {
  return dev ? min(cap, *dev) : cap;
}
constexpr u8 kNoTiny = 255;

struct Dbl4 {
  double x, y, z, w;
};
__device__ __forceinline__ Dbl4 make_dbl4(double x, double y, double z, double w) {
  return Dbl4{x, y, z, w};
}

struct KeyView {
  const u64 *w0, *w1, *w2;
  int words;
  const u16 *sys = nullptr;  // a forest: the system of each sorted position
};

__device__ __forceinline__ int word_lcp(u64 a, u64 b, int levels) {
  const u64 x = a ^ b;
  if (x == 0) return levels;
  const int q = (__clzll(static_cast<long long>(x)) - 1) / 3;
  return q < levels ? q : levels;
}

// Levels shared by the bodies at sorted positions a and b.
__device__ __forceinline__ int lcp(const KeyView &kv, u32 a, u32 b) {
  if (kv.sys && kv.sys[a] != kv.sys[b]) return -1;  // two systems share no node
  int l = word_lcp(kv.w0[a], kv.w0[b], kLevelsPerWord);
  if (l < kLevelsPerWord || kv.words == 1) return l;
  l = word_lcp(kv.w1[a], kv.w1[b], kLevelsPerWord);
  if (l < kLevelsPerWord || kv.words == 2) return kLevelsPerWord + l;
  return 2 * kLevelsPerWord + word_lcp(kv.w2[a], kv.w2[b], kMaxDepth - 2 * kLevelsPerWord);
}

// Octant digit of level `lvl` (1-based) of the body at sorted position b.
__device__ __forceinline__ int digit(const KeyView &kv, u32 b, int lvl) {
  const int w = (lvl - 1) / kLevelsPerWord, q = (lvl - 1) % kLevelsPerWord;
  const u64 word = w == 0 ? kv.w0[b] : (w == 1 ? kv.w1[b] : kv.w2[b]);
  return static_cast<int>((word >> (60 - 3 * q)) & 7u);
}

// The reference's "tiny" leaf rule (octree.cpp:43).
__device__ __forceinline__ bool tiny_node(double h, double cx, double cy, double cz) {
  return h < 1e-12 * (fabs(cx) + fabs(cy) + fabs(cz) + 1e-300);
}

__device__ __forceinline__ void step_centre(double &cx, double &cy, double &cz, int o, double h) {
  cx = cx + ((o & 1) ? h : -h);  // octree.cpp:131-132
  cy = cy + ((o & 2) ? h : -h);
  cz = cz + ((o & 4) ? h : -h);
}

// ------------------------------------------------------------ bounding box

// Order-preserving image of a double for integer comparison: a >= b exactly
// when key(a) >= key(b), for finite a, b (-0.0 is taken as +0.0).
__device__ __forceinline__ u64 order_key(double v) {
  u64 b = static_cast<u64>(__double_as_longlong(v));
  if (b == 0x8000000000000000ull) b = 0;
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double from_order_key(u64 k) {
  return __longlong_as_double(static_cast<long long>((k >> 63) ? (k & 0x7fffffffffffffffull) : ~k));
}

// The split table: along an axis the centres of the tree's levels form a binary
// tree (heap order, node 1 the root centre, the children of node k at level d
// the centre stepped down and up by half_at[d + 1], with the reference's FP64
// addition). Node centres (k_nodes) come from the first kSplitLevels levels and
// are stepped below them (a forest of very many systems: fewer levels each).
// Built by one block, level by level.
__device__ void build_split(const double *centre, const double *half_at, int levels,
                            double *split) {
  for (int a = static_cast<int>(threadIdx.x); a < 3; a += kT) split[(a << levels) + 1] = centre[a];
  for (int d = 1; d < levels; ++d) {
    __syncthreads();
    const double h = half_at[d];
    for (u32 j = threadIdx.x; j < 3u << d; j += kT) {
      double *t = split + (static_cast<u64>(j >> d) << levels);
      const u32 k = (1u << d) + (j & ((1u << d) - 1u));
      t[k] = t[k >> 1] + ((k & 1u) ? h : -h);  // step_centre's operation
    }
  }
}

// A block's partial box, from its warps', as order keys: lows, then highs. Not
// a number counts as nothing, as in fmin and fmax.
__device__ __forceinline__ u64 box_key(const u64 (*warps)[6], int a) {
  u64 v = warps[0][a];
  for (int w = 1; w < kT / 32; ++w) {
    const u64 x = warps[w][a];
    v = a < 3 ? (x < v ? x : v) : (x > v ? x : v);
  }
  const u64 least = order_key(-INFINITY), most = order_key(INFINITY);
  if (v < least || v > most) v = a < 3 ? most : least;
  return v;
}
__device__ __forceinline__ void box_of_warp(u64 (&lo)[3], u64 (&hi)[3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a)
    for (int o = 16; o > 0; o >>= 1) {
      const u64 l = __shfl_xor_sync(kFullMask, lo[a], o), h = __shfl_xor_sync(kFullMask, hi[a], o);
      lo[a] = l < lo[a] ? l : lo[a];
      hi[a] = h > hi[a] ? h : hi[a];
    }
}

// Root cube from the partial boxes (octree.cpp:184-198; min and max are exact in
// any order), by one block, and its split table (null: none wanted). A chain of
// FP64 latencies (64 cycles an operation, some 600 a division): lanes 0 to 2 take
// an axis each, lanes 0 and 1 a division.
__device__ void root_from_parts(const u64 *part, int nparts, TreeRoot *root, int levels,
                                double *split) {
  __shared__ u64 s[kT / 32][6];
  __shared__ double half_at[kMaxDepth + 1], centre[3], half_s;
  __shared__ long long tiny_bound;
  __shared__ int not_tiny[2];
  u64 klo[3], khi[3];
  for (int a = 0; a < 3; ++a) {
    klo[a] = order_key(INFINITY);
    khi[a] = order_key(-INFINITY);
  }
  for (int p = threadIdx.x; p < nparts; p += kT)
    for (int a = 0; a < 3; ++a) {
      const u64 l = __ldcg(part + 6 * p + a), h = __ldcg(part + 6 * p + 3 + a);
      klo[a] = l < klo[a] ? l : klo[a];
      khi[a] = h > khi[a] ? h : khi[a];
    }
  box_of_warp(klo, khi);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int a = 0; a < 3; ++a) {
      s[warp][a] = klo[a];
      s[warp][3 + a] = khi[a];
    }
  __syncthreads();
  if (warp == 0) {
    const int axis = lane < 3 ? lane : 0;
    const double lo = from_order_key(box_key(s, axis)), hi = from_order_key(box_key(s, 3 + axis));
    const double c = (lo + hi) * 0.5, e = 0.5 * (hi - lo), far = fmax(fabs(lo), fabs(hi));
    if (lane < 3) {
      root->lo[lane] = lo;
      root->hi[lane] = hi;
      root->center[lane] = c;
      centre[lane] = c;
    }
    double half = 0.0, reach = 0.0, m1 = 0.0;
    for (int a = 0; a < 3; ++a) {
      const double ea = __shfl_sync(kFullMask, e, a);
      half = half < ea ? ea : half;
      reach = fmax(reach, fabs(__shfl_sync(kFullMask, c, a)));
      m1 = m1 + __shfl_sync(kFullMask, far, a);
    }
    half = half * (1.0 + 1e-9) + 1e-300;
    // the grid of the keys (grid_rank): its band covers the roundings of the
    // reference's centres, at most 20 of 2^-53 (|centre| + half) each, and of
    // the rank itself, in units of 2^-31 cells: 5 (|centre| + half) / half + 1
    const double q =
        (lane == 0 ? static_cast<double>(1 << (kLevelsPerWord - 1)) : reach + half) / half;
    const double band = 8.0 * __shfl_sync(kFullMask, q, 1) + 8.0;
    if (lane == 0) {
      half_s = half;
      root->grid = q;
      root->grid_band = band < 1e9 && half > 1e-280 ? static_cast<u32>(band) : ~0u;
      // every body's |x| + |y| + |z| is at most m1 (rounding is monotone), so
      // no body's tiny bound in k_keys exceeds this one
      tiny_bound = __double_as_longlong(2e-12 * (m1 + 1e-300));
    }
  }
  __syncthreads();
  if (threadIdx.x < 64) {  // (half falls with depth: the levels above the bound come first)
    const int d = static_cast<int>(threadIdx.x);
    double h = half_s;
    if (h > 1e-280) {  // exact: the exponent less d
      h = __longlong_as_double(__double_as_longlong(h) - (static_cast<long long>(d) << 52));
    } else {
      for (int k = 0; k < d; ++k) h = 0.5 * h;
    }
    if (d <= kMaxDepth) {
      half_at[d] = h;
      root->half_at[d] = h;
    }
    const unsigned above =
        __ballot_sync(kFullMask, d <= kMaxDepth && __double_as_longlong(h) >= tiny_bound);
    if (lane == 0) not_tiny[warp] = __popc(above);
  }
  __syncthreads();
  if (threadIdx.x == 0) root->tiny_from = not_tiny[0] + not_tiny[1];
  if (split) build_split(centre, half_at, levels, split);
}

// The bounding box, and from it (the last block to finish) the root cube and
// its split table. Min and max are taken on the order-preserving integer
// images (exact, and off the FP64 pipe); with 16-byte aligned positions a
// thread loads two bodies as three 16-byte words. `ticket` counts finished
// blocks and wraps to zero by itself.
__global__ void __launch_bounds__(kT)
    k_bbox(const double *pos, u64 n, u64 *part, u32 *ticket, TreeRoot *root, double *split) {
  grid_wait();
  const u64 inf_lo = order_key(INFINITY), inf_hi = order_key(-INFINITY);
  u64 lo[3] = {inf_lo, inf_lo, inf_lo}, hi[3] = {inf_hi, inf_hi, inf_hi};
  auto take = [&](int a, double v) {
    const u64 k = order_key(v);
    lo[a] = k < lo[a] ? k : lo[a];
    hi[a] = k > hi[a] ? k : hi[a];
  };
  const u64 first = blockIdx.x * static_cast<u64>(kT) + threadIdx.x,
            stride = static_cast<u64>(gridDim.x) * kT;
  if ((reinterpret_cast<uintptr_t>(pos) & 15) == 0) {
    const double2 *p2 = reinterpret_cast<const double2 *>(pos);
    for (u64 q = first; q < n / 2; q += stride) {
      const double2 u = __ldg(p2 + 3 * q), v = __ldg(p2 + 3 * q + 1), w = __ldg(p2 + 3 * q + 2);
      take(0, u.x);
      take(1, u.y);
      take(2, v.x);
      take(0, v.y);
      take(1, w.x);
      take(2, w.y);
    }
    if ((n & 1) && first == 0)
      for (int a = 0; a < 3; ++a) take(a, pos[3 * (n - 1) + a]);
  } else {
    for (u64 i = first; i < n; i += stride)
      for (int a = 0; a < 3; ++a) take(a, pos[3 * i + a]);
  }
  box_of_warp(lo, hi);
  __shared__ u64 s[kT / 32][6];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int a = 0; a < 3; ++a) {
      s[warp][a] = lo[a];
      s[warp][3 + a] = hi[a];
    }
  __syncthreads();
  if (threadIdx.x < 6) {
    part[6 * blockIdx.x + threadIdx.x] = box_key(s, static_cast<int>(threadIdx.x));
    __threadfence();
  }
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  root_from_parts(part, static_cast<int>(gridDim.x), root, kSplitLevels, split);
}

// A forest's boxes: block b covers part of system blk[b].x (rank blk[b].y of
// its blk[b].z blocks), one partial box each; then one block per system
// reduces that system's partials (sys_blk: first block, blocks) into its
// root.
__global__ void __launch_bounds__(kT)
    k_bbox_forest(const double *pos, const uint4 *blk, const u32 *start, u64 *part) {
  grid_wait();
  const uint4 q = blk[blockIdx.x];
  const u64 b0 = start[q.x], b1 = start[q.x + 1];
  const u64 inf_lo = order_key(INFINITY), inf_hi = order_key(-INFINITY);
  u64 lo[3] = {inf_lo, inf_lo, inf_lo}, hi[3] = {inf_hi, inf_hi, inf_hi};
  for (u64 i = b0 + static_cast<u64>(q.y) * kT + threadIdx.x; i < b1;
       i += static_cast<u64>(q.z) * kT)
    for (int a = 0; a < 3; ++a) {
      const u64 k = order_key(pos[3 * i + a]);
      lo[a] = k < lo[a] ? k : lo[a];
      hi[a] = k > hi[a] ? k : hi[a];
    }
  box_of_warp(lo, hi);
  __shared__ u64 s[kT / 32][6];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int a = 0; a < 3; ++a) {
      s[warp][a] = lo[a];
      s[warp][3 + a] = hi[a];
    }
  __syncthreads();
  if (threadIdx.x < 6) {
    part[6 * blockIdx.x + threadIdx.x] = box_key(s, static_cast<int>(threadIdx.x));
  }
}

__global__ void __launch_bounds__(kT)
    k_root_forest(const u64 *part, const uint2 *sys_blk, TreeRoot *roots, int levels,
                  double *split) {
  grid_wait();
  const uint2 q = sys_blk[blockIdx.x];
  root_from_parts(part + 6ull * q.x, static_cast<int>(q.y), roots + blockIdx.x, levels,
                  split + (static_cast<u64>(3u * blockIdx.x) << levels));
}

// ------------------------------------------------------------------- keys


// Bits b of v at bit 3b (v < 2^21).
__device__ __forceinline__ u64 spread3(u64 v) {
  v &= 0x1fffffull;
  v = (v | v << 32) & 0x1f00000000ffffull;
  v = (v | v << 16) & 0x1f0000ff0000ffull;
  v = (v | v << 8) & 0x100f00f00f00f00full;
  v = (v | v << 4) & 0x10c30c30c30c30c3ull;
  v = (v | v << 2) & 0x1249249249249249ull;
  return v;
}

// The first kLevelsPerWord path bits of coordinate x on an axis: up at level d
// iff x >= the centre of level d on the path. But for the roundings of the
// centres, all 2^21 - 1 of them lie on a grid of spacing half / 2^20 about the
// root centre, so the bits are those of x's place on it, the whole part of
// (x - centre) / spacing + 2^20; adding 2^21 puts that into the top 21 mantissa
// bits, with 31 bits of fraction below. Where the fraction is nearer to a
// whole number than the roundings reach (grid_band), the answer is left open.
__device__ __forceinline__ bool grid_rank(double x, double centre, double grid, u32 band,
                                          u64 &bits) {
  constexpr int kFraction = 52 - kLevelsPerWord;
  const double t = __fma_rn(x - centre, grid, static_cast<double>(3u << (kLevelsPerWord - 1)));
  const u64 b = static_cast<u64>(__double_as_longlong(t));
  const u32 f = static_cast<u32>(b) & ((1u << kFraction) - 1u);
  bits = (b >> kFraction) & ((1ull << kLevelsPerWord) - 1ull);
  return (b >> 52) == 1023u + kLevelsPerWord && f >= band && f <= (1u << kFraction) - band;
}

// First key word: levels 1..21 from the root; records the first depth whose
// node is "tiny" (a leaf whatever its count). Digits below a tiny node are 0,
// so bodies of such a leaf stay in input order through the sort.
//
// Two FP64 operations per axis (grid_rank) where no level can be tiny and no
// coordinate lies within the roundings of a centre; else, about one body in
// 10^7 for a box near the origin, the reference's comparisons level by level.
// (A table of all 2^21 centres per axis took four launches and 60 us a call
// to build and check, and 67 us to look up at 2M bodies: box, table and keys
// 90 -> 22 us at 5k, 161 -> 71 us at 2M.)
//
// A node holding body p has |centre|_1 <= |p|_1 + 3 half (plus rounding), so
// it can only be tiny once half < 1e-12 (|p|_1 + 3 half + 1e-300), i.e. once
// half < ~1.0000001e-12 (|p|_1 + 1e-300). Levels whose half is at least
// twice that bound skip the exact FP64 test; the comparison of two positive
// doubles is done on their bit patterns.
__global__ void __launch_bounds__(kT)
    k_keys(const double *pos, u32 n, const u16 *sys, const TreeRoot *roots, u64 *key, u32 *idx,
           u8 *tiny, u32 *error) {
  grid_wait();
  const u32 i = blockIdx.x * kT + threadIdx.x;
  if (i >= n) return;
  const TreeRoot *root = roots + (sys ? sys[i] : 0);  // (a forest: the body's system's)
  const double x = pos[3ull * i], y = pos[3ull * i + 1], z = pos[3ull * i + 2];
  if (!isfinite(x) || !isfinite(y) || !isfinite(z)) atomicOr(error, 4u);
  const double ox = root->center[0], oy = root->center[1], oz = root->center[2];
  const double grid = root->grid;
  const u32 band = root->grid_band;
  u64 k = 0, rx, ry, rz;
  int t = kNoTiny;
  if (root->tiny_from > kLevelsPerWord && band != ~0u && grid_rank(x, ox, grid, band, rx) &&
      grid_rank(y, oy, grid, band, ry) && grid_rank(z, oz, grid, band, rz)) {
    k = spread3(rx) | (spread3(ry) << 1) | (spread3(rz) << 2);
  } else {
    // the first level whose node could be tiny for this body (half_at falls
    // with depth): the levels above it need no tiny test at all
    const long long maybe_tiny =
        __double_as_longlong(2e-12 * (fabs(x) + fabs(y) + fabs(z) + 1e-300));
    int dt = root->tiny_from;
    if (dt <= kLevelsPerWord) {
      dt = 0;
      while (dt <= kLevelsPerWord && __double_as_longlong(root->half_at[dt]) >= maybe_tiny) ++dt;
    }
    const u64 kx = order_key(x), ky = order_key(y), kz = order_key(z);
    double cx = ox, cy = oy, cz = oz;
    for (int d = 0; d < kLevelsPerWord; ++d) {
      if (d >= dt && t == kNoTiny && tiny_node(root->half_at[d], cx, cy, cz)) t = d;
      int o = (kx >= order_key(cx) ? 1 : 0) | (ky >= order_key(cy) ? 2 : 0) |
              (kz >= order_key(cz) ? 4 : 0);
      if (t != kNoTiny) o = 0;
      k = (k << 3) | static_cast<u64>(o);
      step_centre(cx, cy, cz, o, root->half_at[d + 1]);
    }
    if (dt <= kLevelsPerWord && t == kNoTiny &&
        tiny_node(root->half_at[kLevelsPerWord], cx, cy, cz))
      t = kLevelsPerWord;
  }
  key[i] = k;
  idx[i] = i;
  tiny[i] = static_cast<u8>(t);
}

// A forest's last sort pass, by system: the system of each sorted body as
// the key, the position as the value; the key words and bodies are copied
// aside for the gather that follows the pass. (Here and below: what a sort that
// failed leaves behind is not used as places; the solve ends with its error.)
__global__ void __launch_bounds__(kT)
    k_forest_sys_keys(const u64 *key, const u32 *idx, const u16 *sys, u32 n, u64 *skey, u32 *spos,
                      u64 *key_copy, u32 *idx_copy, const u32 *error) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= n || *error) return;
  const u32 i = idx[k];
  skey[k] = sys[i];
  spos[k] = k;
  key_copy[k] = key[k];
  idx_copy[k] = i;
}

__global__ void __launch_bounds__(kT)
    k_forest_gather(const u32 *spos, const u64 *key_copy, const u32 *idx_copy, u32 n, u64 *key,
                    u32 *idx, const u32 *error) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= n || *error) return;
  const u32 j = spos[k];
  key[k] = key_copy[j];
  idx[k] = idx_copy[j];
}

// Per sorted position: levels shared with the next body, the leaf depth, and
// the number of nodes that end there.
__global__ void __launch_bounds__(kT)
    k_levels(KeyView kv, const u32 *idx, const u8 *tiny, u32 n, int L, signed char *lcp_next,
             u8 *leafdepth, u32 *count, Scalars *sc) {
  grid_wait();
  // win[i] = lcp(i, i + L) for the block's positions and the L before them,
  // each computed once; a body's w is the largest over its windows
  constexpr int kMaxWin = 64;
  __shared__ signed char win[kT + kMaxWin];
  if (sc->error) return;
  const u32 base = blockIdx.x * kT, b = base + threadIdx.x;
  const bool shared_win = L <= kMaxWin;
  if (shared_win) {
    for (int k = threadIdx.x; k < kT + L; k += kT) {
      const long long i = static_cast<long long>(base) + k - L;
      win[k] = static_cast<signed char>(
          i >= 0 && i + L < static_cast<long long>(n) ? lcp(kv, static_cast<u32>(i), static_cast<u32>(i + L)) : -1);
    }
    __syncthreads();
  }
  int ld = 0;
  if (b < n) {
    const int next = b + 1 < n ? lcp(kv, b, b + 1) : -1;
    lcp_next[b] = static_cast<signed char>(next);
    int w = -1;
    if (n > static_cast<u32>(L)) {
      const u32 lo = b >= static_cast<u32>(L) ? b - L : 0;
      const u32 hi = min(b, n - 1 - L);
      for (u32 i = lo; i <= hi; ++i)
        w = max(w, shared_win ? static_cast<int>(win[i - base + L]) : lcp(kv, i, i + L));
    }
    ld = min(w + 1, kMaxDepth);
    ld = min(ld, static_cast<int>(tiny[idx[b]]));
    leafdepth[b] = static_cast<u8>(ld);
    count[b] = static_cast<u32>(max(0, ld - next));  // the nodes that end at b
  }
  // one atomic per warp for each counter
  const u32 deep = __popc(__ballot_sync(kFullMask, b < n && ld > kLevelsPerWord * kv.words));
  const u32 dmax = __reduce_max_sync(kFullMask, static_cast<u32>(ld));
  if ((threadIdx.x & 31) == 0) {
    if (deep) atomicAdd(&sc->deep, deep);
    atomicMax(&sc->depth, dmax);
  }
}

// ------------------------------------------------------- deeper key words

__global__ void __launch_bounds__(kT)
    k_deep_flags(const u8 *leafdepth, u32 n, int limit, u32 *flag) {
  grid_wait();
  const u32 b = blockIdx.x * kT + threadIdx.x;
  if (b < n) flag[b] = leafdepth[b] > limit ? 1u : 0u;
}

__global__ void __launch_bounds__(kT)
    k_compact(const u32 *flag, const u32 *scan, u32 n, u32 *out) {
  grid_wait();
  const u32 b = blockIdx.x * kT + threadIdx.x;
  if (b < n && flag[b]) out[scan[b]] = b;
}

// Next key word for the deep bodies: replay the path to depth 21*words from
// the root with the existing digits, then record up to 21 more levels.
__global__ void __launch_bounds__(kT)
    k_deep_keys(KeyView kv, const u32 *dpos, u32 nd, const u32 *idx, const double *pos,
                const TreeRoot *root, u8 *tiny, u64 *word, u32 *rec, u32 *didx) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= nd) return;
  const u32 b = dpos[k];
  const u32 i = idx[b];
  if (kv.sys) root += kv.sys[b];  // a forest: the body's system's root
  const int base = kLevelsPerWord * kv.words;
  double cx = root->center[0], cy = root->center[1], cz = root->center[2];
  for (int lvl = 1; lvl <= base; ++lvl) step_centre(cx, cy, cz, digit(kv, b, lvl), root->half_at[lvl]);
  const double x = pos[3ull * i], y = pos[3ull * i + 1], z = pos[3ull * i + 2];
  const int levels = min(kLevelsPerWord, kMaxDepth - base);
  int t = tiny[i];
  u64 w = 0;
  for (int q = 0; q < levels; ++q) {
    const int d = base + q;  // depth of the node being split
    if (q > 0 && t == kNoTiny && tiny_node(root->half_at[d], cx, cy, cz)) t = d;
    int o = (x >= cx ? 1 : 0) | (y >= cy ? 2 : 0) | (z >= cz ? 4 : 0);
    if (t != kNoTiny) o = 0;
    w = (w << 3) | static_cast<u64>(o);
    step_centre(cx, cy, cz, o, root->half_at[d + 1]);
  }
  if (t == kNoTiny && tiny_node(root->half_at[base + levels], cx, cy, cz)) t = base + levels;
  w <<= 3 * (kLevelsPerWord - levels);
  tiny[i] = static_cast<u8>(t);
  word[k] = w;
  rec[k] = k;
  didx[k] = i;
}

// Segment of each deep record: a new segment starts where the existing key
// words change (a different depth-21*words node).
__global__ void __launch_bounds__(kT)
    k_deep_segments(KeyView kv, const u32 *dpos, u32 nd, u32 *flag) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= nd) return;
  bool start = k == 0;
  if (!start) {
    const u32 a = dpos[k - 1], b = dpos[k];
    start = kv.w0[a] != kv.w0[b] || (kv.words > 1 && kv.w1[a] != kv.w1[b]) ||
            (kv.sys && kv.sys[a] != kv.sys[b]);
  }
  flag[k] = start ? 1u : 0u;
}

__global__ void __launch_bounds__(kT)
    k_seg_keys(const u32 *rec, const u32 *seg_scan, const u32 *seg_flag, u32 nd, u64 *key,
               const u32 *error) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= nd || *error) return;
  const u32 r = rec[k];
  key[k] = seg_scan[r] + seg_flag[r];  // 1-based segment number
}

// Puts the deep records back into their positions, now ordered by (segment,
// new word, input order).
__global__ void __launch_bounds__(kT)
    k_deep_scatter(const u32 *dpos, const u32 *rec, const u32 *didx, const u64 *word, u32 nd,
                   u32 *idx, u64 *word_out, const u32 *error) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= nd || *error) return;
  const u32 r = rec[k];
  idx[dpos[k]] = didx[r];
  word_out[dpos[k]] = word[r];
}

// ------------------------------------------------------------------ nodes

// Writes the nodes ending at sorted position b, shallowest first.
//
// Bound: the threads whose bodies end large nodes (the last body ends all of
// the tree's right spine) and each node's search for its first body, a chain
// of dependent key loads. So a thread gallops back kNear bodies at a step at most
// and leaves longer searches to the block's warps, 32 probes a step: 5k bodies 18
// -> 12 us, 200k 41 -> 19, 2M 125 -> 117.
constexpr u32 kNear = 16;
constexpr u32 kFarTasks = 256;  // of a block; a thread searches on beyond
__global__ void __launch_bounds__(kT)
    k_nodes(KeyView kv, const signed char *lcp_next, const u8 *leafdepth, const u32 *count,
            const u32 *count_scan, u32 n, const Scalars *sc, const TreeRoot *root,
            const double *split, double2 *geom, u32 *nbegin, u32 *nend, u32 *skip, u8 *depth,
            u8 *isleaf, int table_levels, const u32 *abort = nullptr) {
  grid_wait();
  __shared__ u32 far_b[kFarTasks], far_hi[kFarTasks], far_p[kFarTasks], far_n;
  __shared__ u8 far_d[kFarTasks];
  const u32 table_size = 1u << table_levels;
  if (aborted(abort)) return;
  if (threadIdx.x == 0) far_n = 0u;
  __syncthreads();
  const u32 total = sc->n_nodes;
  const bool forest = kv.sys != nullptr;
  const u32 b = blockIdx.x * kT + threadIdx.x;
  const u32 c = b < n ? count[b] : 0u;
  if (c != 0) {
    const u32 first = total - count_scan[b] - c;  // nodes ending after b come first
    const int d0 = lcp_next[b] + 1, ld = leafdepth[b];
    // centres from the split table down to its last level, stepped below it
    // (a forest: `root` and `split` hold every system's root and table)
    const u32 sys = forest ? kv.sys[b] : 0u;
    root += sys;
    const double *tx = split + 3ull * sys * table_size, *ty = tx + table_size,
                 *tz = ty + table_size;
    u32 ix = 1, iy = 1, iz = 1;
    double cx = 0.0, cy = 0.0, cz = 0.0;
    for (int d = 0; d <= ld; ++d) {
      if (d > 0) {
        const int o = digit(kv, b, d);
        if (d < table_levels) {
          ix = 2 * ix + (o & 1);
          iy = 2 * iy + ((o >> 1) & 1);
          iz = 2 * iz + (o >> 2);
        } else {
          if (d == table_levels) {  // the table's deepest centre on this path
            cx = __ldg(tx + ix);
            cy = __ldg(ty + iy);
            cz = __ldg(tz + iz);
          }
          step_centre(cx, cy, cz, o, root->half_at[d]);
        }
      }
      if (d < d0) continue;
      if (d < table_levels) {
        cx = __ldg(tx + ix);
        cy = __ldg(ty + iy);
        cz = __ldg(tz + iz);
      }
      const u32 p = first + static_cast<u32>(d - d0);
      geom[2 * p] = make_double2(cx, cy);
      geom[2 * p + 1] = make_double2(cz, root->half_at[d]);
      nend[p] = b + 1;
      depth[p] = static_cast<u8>(d);
      isleaf[p] = d == ld ? 1 : 0;
    }
    // First body of each node: the smallest position sharing d levels with b.
    // Deepest node first; each shallower node starts at or before the deeper
    // one, so the search gallops back from there (a few probes for the small
    // nodes that most are) and then halves the last interval.
    u32 start = b;  // shares at least d levels with b for every d here
    bool far = false;
    for (int d = ld; d >= d0; --d) {
      const u32 p = first + static_cast<u32>(d - d0);
      u32 lo = 0, hi = start;
      if (d > 0 || forest) {  // (a forest's root starts at its system's first body)
        bool bounded_below = false;
        auto gallop = [&](u64 step, u64 most) {  // 64-bit: never wraps to 0
          for (; step <= most && !bounded_below; step *= 2) {
            bounded_below = step > hi;  // (lo stays 0)
            if (bounded_below) break;
            const u32 cand = hi - static_cast<u32>(step);
            bounded_below = lcp(kv, cand, b) < d;
            if (bounded_below) lo = cand + 1;
            else hi = cand;
          }
        };
        if (!far) gallop(1, kNear);
        if (!bounded_below) {
          far = true;
          const u32 at = atomicAdd(&far_n, 1u);
          start = hi;
          if (at < kFarTasks) {
            far_b[at] = b;
            far_hi[at] = hi;
            far_p[at] = p;
            far_d[at] = static_cast<u8>(d);
            continue;
          }
          gallop(2 * kNear, ~0ull >> 1);
        }
        while (lo < hi) {  // lcp(lo - 1, b) < d (or lo = 0), lcp(hi, b) >= d
          const u32 mid = lo + (hi - lo) / 2;
          if (lcp(kv, mid, b) >= d) hi = mid;
          else lo = mid + 1;
        }
      }
      nbegin[p] = lo;
      skip[p] = total - count_scan[lo];
      start = lo;
    }
  }
  __syncthreads();
  const u32 lane = threadIdx.x & 31u, tasks = min(far_n, kFarTasks);
  for (u32 t = threadIdx.x >> 5; t < tasks; t += kT / 32) {
    const u32 fb = far_b[t];
    const int d = far_d[t];
    u32 lo = 0, hi = far_hi[t];  // lcp(hi, fb) >= d
    while (lo < hi) {
      const u32 q = lo + static_cast<u32>(static_cast<u64>(hi - lo) * lane / 32u);  // below hi
      const u32 in = __ballot_sync(kFullMask, lcp(kv, q, fb) >= d);  // from some lane on
      const u32 k = in ? static_cast<u32>(__ffs(static_cast<int>(in))) - 1u : 32u;
      const u32 below = __shfl_sync(kFullMask, q, (k - 1u) & 31u),
                here = __shfl_sync(kFullMask, q, k & 31u);
      if (k < 32u) hi = here;
      lo = k ? below + 1u : hi;
    }
    if (lane == 0) {
      nbegin[far_p[t]] = lo;
      skip[far_p[t]] = total - count_scan[lo];
    }
  }
}

// Children of a node are p+1, skip[p+1], ... (last octant first) up to skip[p].
__device__ __forceinline__ int children_of(u32 p, const u32 *skip, u32 ch[8]) {
  int k = 0;
  for (u32 c = p + 1; c < skip[p] && k < 8; c = skip[c]) ch[k++] = c;
  return k;
}

// Parents, child counts and every inner node's children (8 slots, last
// octant first), so that the moment kernels load a node's children at once
// instead of following the skip chain.
__global__ void __launch_bounds__(kT)
    k_children(const u32 *skip, const u8 *isleaf, u32 m, u32 *parent, u8 *nchild, uint4 *kids,
               const u32 *m_dev = nullptr, const u32 *abort = nullptr) {
  grid_wait();
  const u32 p = blockIdx.x * kT + threadIdx.x;
  if (aborted(abort) || p >= bounded(m, m_dev)) return;
  if (p == 0) parent[0] = 0xffffffffu;
  if (isleaf[p]) {
    nchild[p] = 0;
    return;
  }
  u32 ch[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  const int k = children_of(p, skip, ch);
  nchild[p] = static_cast<u8>(k);
  for (int j = 0; j < k; ++j) parent[ch[j]] = p;
  kids[2ull * p] = make_uint4(ch[0], ch[1], ch[2], ch[3]);
  kids[2ull * p + 1] = make_uint4(ch[4], ch[5], ch[6], ch[7]);
}

// A forest's roots: system k's root is the first (shallowest) of the nodes
// ending at its last body, and has no parent.
__global__ void __launch_bounds__(kT)
    k_forest_roots(const u32 *start, u32 systems, const u32 *count, const u32 *count_scan,
                   const Scalars *sc, u32 *root_node, u32 *parent, const u32 *abort = nullptr) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= systems || aborted(abort)) return;
  const u32 last = start[k + 1] - 1;
  const u32 r = sc->n_nodes - count_scan[last] - count[last];
  root_node[k] = r;
  parent[r] = 0xffffffffu;
}

// Sorts n <= kN values in registers (Batcher's odd-even merge network; the places
// past n hold values that stay behind all others).
template <int kN>
__device__ __forceinline__ void sort_few(u32 *v, u32 n) {
  u32 r[kN];
#pragma unroll
  for (int i = 0; i < kN; ++i) r[i] = static_cast<u32>(i) < n ? v[i] : 0xffffffffu;
#pragma unroll
  for (int p = 1; p < kN; p *= 2)
#pragma unroll
    for (int k = p; k >= 1; k /= 2)
#pragma unroll
      for (int j = k % p; j + k < kN; j += 2 * k)
#pragma unroll
        for (int i = 0; i < k; ++i)
          if (i + j + k < kN && (i + j) / (2 * p) == (i + j + k) / (2 * p)) {
            const u32 lo = min(r[i + j], r[i + j + k]), hi = max(r[i + j], r[i + j + k]);
            r[i + j] = lo;
            r[i + j + k] = hi;
          }
#pragma unroll
  for (int i = 0; i < kN; ++i)
    if (static_cast<u32>(i) < n) v[i] = r[i];
}

// Input order inside each leaf (the reference never splits a leaf's range). A
// thread's loads are issued together and its leaf sorted in registers (an
// insertion sort in memory, a chain of loads and stores, before): 5k bodies 7.5 -> 4.6
// us, 200k 13.5 -> 5.2, 2M 34 -> 10; larger leaves still so.
__global__ void __launch_bounds__(kT)
    k_leaf_order(const u8 *isleaf, const u32 *nbegin, const u32 *nend, u32 m, u32 *idx,
                 const u32 *m_dev = nullptr, const u32 *abort = nullptr) {
  grid_wait();
  const u32 p = blockIdx.x * kT + threadIdx.x;
  if (aborted(abort) || p >= bounded(m, m_dev) || !isleaf[p]) return;
  const u32 b0 = nbegin[p], b1 = nend[p];
  if (b1 - b0 <= 8) return sort_few<8>(idx + b0, b1 - b0);
  if (b1 - b0 <= 16) return sort_few<16>(idx + b0, b1 - b0);
  for (u32 i = b0 + 1; i < b1; ++i) {
    const u32 v = idx[i];
    u32 j = i;
    while (j > b0 && idx[j - 1] > v) {
      idx[j] = idx[j - 1];
      --j;
    }
    idx[j] = v;
  }
}

__global__ void __launch_bounds__(kT)
    k_tree_order(const double *pos, const double *mass, const u32 *idx, u32 n, double *tpos,
                 double *tmass, const u32 *abort = nullptr) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= n || aborted(abort)) return;
  const u64 i = idx[k];
  tpos[3ull * k] = pos[3 * i];
  tpos[3ull * k + 1] = pos[3 * i + 1];
  tpos[3ull * k + 2] = pos[3 * i + 2];
  tmass[k] = mass[i];
}

// ---------------------------------------------------------------- moments

struct MomentArrays {
  const double2 *geom;   // 2 per node: (cx, cy), (cz, half)
  const u32 *nbegin, *nend, *skip, *parent;
  const u8 *nchild;
  const uint4 *kids;     // 2 per node: the children, last octant first
  const double *tpos, *tmass;
  double2 *mom;     // 2 per node: (mx, my), (mz, mass)
  double2 *quad;    // 3 x double2 per node: xx yy | zz xy | xz yz
  double *delta;
  double *term;     // 6 per node: what it adds to its parent's quadrupole beside its own
};

__device__ __forceinline__ Dbl4 load_pair(const double2 *a, u32 p) {
  const double2 u = a[2 * p], v = a[2 * p + 1];
  return make_dbl4(u.x, u.y, v.x, v.y);
}

// The moments in two passes, with the reference's operations in its order:
// the centres of mass first (all the walk's records need), the quadrupoles
// after them, from the stored centres of mass. The walk starts after the
// first pass while the second one runs beside it.
//
// FP64 sets the time: the pipe issues one warp instruction in 16 cycles
// whatever its lanes, with a latency of 64, a division takes 560. So one lane
// works one component of a node (a centre of mass: x, y, z, mass; a
// quadrupole: six): the components of a node advance together, and a node's
// chain is its children's additions and one division.
//
// A team of lanes starts from each leaf; the last child of a node to finish
// hands the node to its own block's queue (a count per node, no waiting), and
// the block's teams work the queue together, so that the lanes of a warp are
// full while a block has work. One launch builds the whole tree: with a launch
// per depth each depth took 9 us (centres of mass) and 15 us (quadrupoles)
// however few its nodes. Centres of mass with the walk records, then the
// quadrupoles and cells: 5k bodies 113 -> 40 and 180 -> 53 us, 50k 130 -> 48 and
// 254 -> 70 us, 2M 358 -> 311 us and, beside the walk, 1.63 -> 1.10 ms.
__device__ __forceinline__ double *mom_d(const MomentArrays &a) {
  return reinterpret_cast<double *>(a.mom);
}

// A centre of mass and mass by a team of four lanes (component c: x, y, z,
// mass) from their sums: the mass in lane 3, sums of mass times position in
// the others (octree.cpp:46-54, 75-85).
__device__ __forceinline__ void finish_com(const MomentArrays &a, u32 p, int c, double sum,
                                           u32 team_mask) {
  const double m = __shfl_sync(team_mask, sum, 3, 4);
  double v = sum;
  if (c < 3) v = m > 0 ? sum / m : reinterpret_cast<const double *>(a.geom)[4ull * p + c];
  mom_d(a)[4ull * p + c] = v;
}

// kAhead bodies' loads together: small trees wait for them (5k bodies 35 -> 33
// us, 50k 41 -> 40), large ones for the FP64 pipe (2M by one 190 us, by eight 250).
template <u32 kAhead>
__device__ __forceinline__ void leaf_com(const MomentArrays &a, u32 p, int c, u32 team_mask) {
  const u32 b0 = a.nbegin[p], b1 = a.nend[p];
  double sum = 0.0;
  for (u32 k = b0; k < b1; k += kAhead) {
    double m[kAhead], x[kAhead];
#pragma unroll
    for (u32 j = 0; j < kAhead; ++j)
      if (k + j < b1) {
        m[j] = a.tmass[k + j];
        x[j] = c < 3 ? a.tpos[3ull * (k + j) + c] : 0.0;
      }
#pragma unroll
    for (u32 j = 0; j < kAhead; ++j)
      if (k + j < b1) {
        const double t = c < 3 ? m[j] * x[j] : m[j];
        sum += t;
      }
  }
  finish_com(a, p, c, sum, team_mask);
}

// A node's children, first octant first (kids lists them last octant first),
// as many as it has.
__device__ __forceinline__ int load_kids(const MomentArrays &a, u32 p, u32 ch[8]) {
  const uint4 k0 = a.kids[2ull * p], k1 = a.kids[2ull * p + 1];
  ch[0] = k0.x;
  ch[1] = k0.y;
  ch[2] = k0.z;
  ch[3] = k0.w;
  ch[4] = k1.x;
  ch[5] = k1.y;
  ch[6] = k1.z;
  ch[7] = k1.w;
  return a.nchild[p];
}

// Children finished by other blocks of the same launch are read from L2: an
// SM's L1 may hold an older copy of the line.
__device__ __forceinline__ void node_com(const MomentArrays &a, u32 p, int c, u32 team_mask) {
  u32 ch[8];
  const int nc = load_kids(a, p, ch);
  double v[8], w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < nc) {
      w[j] = __ldcg(mom_d(a) + 4ull * ch[j] + 3);
      v[j] = __ldcg(mom_d(a) + 4ull * ch[j] + c);
    }
  double sum = 0.0;
#pragma unroll
  for (int j = 7; j >= 0; --j)
    if (j < nc) {
      const double t = c < 3 ? w[j] * v[j] : w[j];
      sum += t;
    }
  finish_com(a, p, c, sum, team_mask);
}

__device__ __forceinline__ double delta_of(const Dbl4 &com, const Dbl4 &g) {  // octree.cpp:71, 101
  const double ex = com.x - g.x, ey = com.y - g.y, ez = com.z - g.z;
  return sqrt(ex * ex + ey * ey + ez * ez);
}

// Bodies whose loads a leaf's quadrupole starts together (5k bodies 17 -> 13 us, 50k
// 26 -> 18; 4 and 8 measure the same).
constexpr u32 kLeafAhead = 4;
__device__ void leaf_quad(const MomentArrays &a, u32 p) {  // octree.cpp:55-70
  const Dbl4 c = load_pair(a.mom, p);
  const double cx = c.x, cy = c.y, cz = c.z;
  const u32 b0 = a.nbegin[p], b1 = a.nend[p];
  double q0 = 0, q1 = 0, q2 = 0, q3 = 0, q4 = 0, q5 = 0;
  for (u32 k = b0; k < b1; k += kLeafAhead) {  // several bodies' loads first
    double m[kLeafAhead], x[kLeafAhead], y[kLeafAhead], z[kLeafAhead];
#pragma unroll
    for (u32 j = 0; j < kLeafAhead; ++j)
      if (k + j < b1) {
        m[j] = a.tmass[k + j];
        x[j] = a.tpos[3ull * (k + j)];
        y[j] = a.tpos[3ull * (k + j) + 1];
        z[j] = a.tpos[3ull * (k + j) + 2];
      }
#pragma unroll
    for (u32 j = 0; j < kLeafAhead; ++j)
      if (k + j < b1) {
        const double mi = m[j], dx = x[j] - cx, dy = y[j] - cy, dz = z[j] - cz;
        const double r2 = dx * dx + dy * dy + dz * dz;
        q0 += mi * (3 * dx * dx - r2);
        q1 += mi * (3 * dy * dy - r2);
        q2 += mi * (3 * dz * dz - r2);
        q3 += mi * 3 * dx * dy;
        q4 += mi * 3 * dx * dz;
        q5 += mi * 3 * dy * dz;
      }
  }
  a.quad[3 * p] = make_double2(q0, q1);
  a.quad[3 * p + 1] = make_double2(q2, q3);
  a.quad[3 * p + 2] = make_double2(q4, q5);
}

// What node p adds to its parent's quadrupole beside its own (octree.cpp:86-100:
// the parallel-axis terms). They need centres of mass only, so every node's
// are formed at once, and a node's chain is additions.
__device__ __forceinline__ void quad_term(const MomentArrays &a, u32 p) {
  const u32 q = a.parent[p];
  if (q == 0xffffffffu) return;
  const Dbl4 c = load_pair(a.mom, p), pc = load_pair(a.mom, q);
  const double dx = c.x - pc.x, dy = c.y - pc.y, dz = c.z - pc.z;
  const double r2 = dx * dx + dy * dy + dz * dz;
  double2 *t = reinterpret_cast<double2 *>(a.term + 6ull * p);
  t[0] = make_double2(c.w * (3 * dx * dx - r2), c.w * (3 * dy * dy - r2));
  t[1] = make_double2(c.w * (3 * dz * dz - r2), c.w * 3 * dx * dy);
  t[2] = make_double2(c.w * 3 * dx * dz, c.w * 3 * dy * dz);
}

// Component c (below 6) of a node's quadrupole from its children's.
__device__ __forceinline__ void node_quad(const MomentArrays &a, u32 p, int c) {
  u32 ch[8];
  const int nc = load_kids(a, p, ch);
  double *quad = reinterpret_cast<double *>(a.quad);
  double v[8], t[8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < nc) {
      v[j] = __ldcg(quad + 6ull * ch[j] + c);
      t[j] = a.term[6ull * ch[j] + c];
    }
  double sum = 0.0;
#pragma unroll
  for (int j = 7; j >= 0; --j)
    if (j < nc) sum += v[j] + t[j];
  quad[6ull * p + c] = sum;
}

// FP32 estimates of the moments, for the learned walk's decisions only: the
// same sums as the FP64 passes, in FP32 on the FP32 bodies (relative to the root centre),
// written as GTCell-layout cells plus delta.
// They take a few tens of microseconds where the FP64 moments take most of a
// millisecond, so the learned walk starts while the FP64 moments -- which
// the evaluation reads -- are still being accumulated.
struct Moment32Arrays {
  const double2 *geom;
  const u32 *nbegin, *nend;
  const u8 *nchild;
  const uint4 *kids;
  const float4 *bodies;  // tree order, relative to the root centre
  const TreeRoot *root;
  float4 *cells;         // 3 per node: (com, mass), (xx, yy, zz, xy), (xz, yz, 0, 0)
  float *delta;
};

__device__ __forceinline__ void finish_moments32(const Moment32Arrays &a, u32 p, float m, float cx,
                                                 float cy, float cz, const float *q) {
  const Dbl4 g = load_pair(a.geom, p);
  const float gx = static_cast<float>(g.x - a.root->center[0]),
              gy = static_cast<float>(g.y - a.root->center[1]),
              gz = static_cast<float>(g.z - a.root->center[2]);
  a.cells[3 * p] = make_float4(cx, cy, cz, m);
  a.cells[3 * p + 1] = make_float4(q[0], q[1], q[2], q[3]);
  a.cells[3 * p + 2] = make_float4(q[4], q[5], 0.f, 0.f);
  const float ex = cx - gx, ey = cy - gy, ez = cz - gz;
  a.delta[p] = sqrtf(ex * ex + ey * ey + ez * ez);
}

__device__ __forceinline__ float3 centre32(const Moment32Arrays &a, u32 p) {
  const Dbl4 g = load_pair(a.geom, p);
  return make_float3(static_cast<float>(g.x - a.root->center[0]),
                     static_cast<float>(g.y - a.root->center[1]),
                     static_cast<float>(g.z - a.root->center[2]));
}

// Bodies k0.. of [k0, k1), at most eight, loaded together.
__device__ __forceinline__ void bodies32(const Moment32Arrays &a, u32 k0, u32 k1, float4 (&b)[8]) {
#pragma unroll
  for (u32 j = 0; j < 8; ++j)
    if (k0 + j < k1) b[j] = a.bodies[k0 + j];
}

__device__ void leaf_moments32(const Moment32Arrays &a, u32 p) {
  const u32 b0 = a.nbegin[p], b1 = a.nend[p];
  float m = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
  float4 b[8];
  for (u32 k = b0; k < b1; k += 8) {
    bodies32(a, k, b1, b);
#pragma unroll
    for (u32 j = 0; j < 8; ++j) {
      if (k + j >= b1) break;
      m += b[j].w;
      cx += b[j].w * b[j].x;
      cy += b[j].w * b[j].y;
      cz += b[j].w * b[j].z;
    }
  }
  if (m > 0) {
    cx /= m;
    cy /= m;
    cz /= m;
  } else {
    const float3 c = centre32(a, p);
    cx = c.x;
    cy = c.y;
    cz = c.z;
  }
  float q[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (u32 k = b0; k < b1; k += 8) {
    if (b1 - b0 > 8) bodies32(a, k, b1, b);
#pragma unroll
    for (u32 j = 0; j < 8; ++j) {
      if (k + j >= b1) break;
      const float w = b[j].w, dx = b[j].x - cx, dy = b[j].y - cy, dz = b[j].z - cz;
      const float r2 = dx * dx + dy * dy + dz * dz;
      q[0] += w * (3.f * dx * dx - r2);
      q[1] += w * (3.f * dy * dy - r2);
      q[2] += w * (3.f * dz * dz - r2);
      q[3] += w * 3.f * dx * dy;
      q[4] += w * 3.f * dx * dz;
      q[5] += w * 3.f * dy * dz;
    }
  }
  finish_moments32(a, p, m, cx, cy, cz, q);
}

// The children's cells, written by other threads of the same launch, are read
// from L2 (an SM's L1 may hold an older copy of the line), all loads first.
__device__ void node_moments32(const Moment32Arrays &a, u32 p) {
  const uint4 k0 = a.kids[2ull * p], k1 = a.kids[2ull * p + 1];
  const u32 ch[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
  const int nc = a.nchild[p];
  float4 c[8], qa[8];
  float2 qb[8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < nc) {
      const float4 *cell = &a.cells[3 * ch[j]];
      c[j] = __ldcg(cell);
      qa[j] = __ldcg(cell + 1);
      qb[j] = __ldcg(reinterpret_cast<const float2 *>(cell + 2));
    }
  float m = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
#pragma unroll
  for (int j = 7; j >= 0; --j)
    if (j < nc) {
      m += c[j].w;
      cx += c[j].w * c[j].x;
      cy += c[j].w * c[j].y;
      cz += c[j].w * c[j].z;
    }
  if (m > 0) {
    cx /= m;
    cy /= m;
    cz /= m;
  } else {
    const float3 c = centre32(a, p);
    cx = c.x;
    cy = c.y;
    cz = c.z;
  }
  float q[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 7; j >= 0; --j)
    if (j < nc) {
      const float w = c[j].w, dx = c[j].x - cx, dy = c[j].y - cy, dz = c[j].z - cz;
      const float r2 = dx * dx + dy * dy + dz * dz;
      q[0] += qa[j].x + w * (3.f * dx * dx - r2);
      q[1] += qa[j].y + w * (3.f * dy * dy - r2);
      q[2] += qa[j].z + w * (3.f * dz * dz - r2);
      q[3] += qa[j].w + w * 3.f * dx * dy;
      q[4] += qb[j].x + w * 3.f * dx * dz;
      q[5] += qb[j].y + w * 3.f * dy * dz;
    }
  finish_moments32(a, p, m, cx, cy, cz, q);
}

// Leaves are bucketed by body count, so that the leaves a warp sums loop the
// same number of times: the FP64 pipe, the bound here, then issues full
// warps. The order inside a bucket does not matter, each leaf's sums run in
// the reference's order. Small trees go without (kBucketNodes).
constexpr int kLeafClasses = 9;                          // 1..8 bodies, more
constexpr int kBuckets = kLeafClasses;

struct BucketView {
  const u8 *isleaf;
  const u32 *nbegin, *nend;
};

// A leaf's bucket, -1 for an inner node.
__device__ __forceinline__ int bucket_of(const BucketView &v, u32 p) {
  if (!v.isleaf[p]) return -1;
  const u32 nb = v.nend[p] - v.nbegin[p];
  return static_cast<int>(nb < 1 ? 0u : min(nb, static_cast<u32>(kLeafClasses)) - 1);
}

// Per-block histograms in shared memory, one global atomic per bucket.
__global__ void __launch_bounds__(kT)
    k_bucket_count(BucketView v, u32 m, u32 *count, const u32 *m_dev = nullptr,
                   const u32 *abort = nullptr) {
  grid_wait();
  __shared__ u32 h[kBuckets];
  if (aborted(abort)) return;
  if (threadIdx.x < kBuckets) h[threadIdx.x] = 0;
  __syncthreads();
  const u32 p = blockIdx.x * kT + threadIdx.x;
  if (p < bounded(m, m_dev)) {
    const int b = bucket_of(v, p);
    if (b >= 0) atomicAdd(&h[b], 1u);
  }
  __syncthreads();
  if (threadIdx.x < kBuckets && h[threadIdx.x]) atomicAdd(&count[threadIdx.x], h[threadIdx.x]);
}

// Each block reserves one range per bucket behind the buckets before it, then
// places its leaves there. meta: the counts, then the places taken.
__global__ void __launch_bounds__(kT)
    k_bucket_fill(BucketView v, u32 m, u32 *meta, u32 *bucket, const u32 *m_dev = nullptr,
                  const u32 *abort = nullptr) {
  grid_wait();
  __shared__ u32 h[kBuckets], base[kBuckets];
  if (aborted(abort)) return;
  if (threadIdx.x < kBuckets) h[threadIdx.x] = 0;
  __syncthreads();
  const u32 p = blockIdx.x * kT + threadIdx.x;
  int b = -1;
  u32 local = 0;
  if (p < bounded(m, m_dev)) {
    b = bucket_of(v, p);
    if (b >= 0) local = atomicAdd(&h[b], 1u);
  }
  __syncthreads();
  if (threadIdx.x < kBuckets) {
    u32 first = 0;
    for (u32 k = 0; k < threadIdx.x; ++k) first += meta[k];
    base[threadIdx.x] =
        h[threadIdx.x] ? first + atomicAdd(&meta[kBuckets + threadIdx.x], h[threadIdx.x]) : 0u;
  }
  __syncthreads();
  if (b >= 0) bucket[base[b] + local] = p;
}

__device__ __forceinline__ u32 leaf_count(const u32 *meta) {
  u32 count = 0;
  for (int b = 0; b < kLeafClasses; ++b) count += meta[b];
  return count;
}

// The k-th leaf: from the buckets, or (bucket null) node k when it is a leaf.
// kNoNode past the last.
constexpr u32 kNoNode = 0xffffffffu;
__device__ __forceinline__ u32 nth_leaf(u64 k, const u32 *bucket, const u32 *meta,
                                        const u8 *isleaf, u32 m) {
  if (bucket) return k < leaf_count(meta) ? bucket[k] : kNoNode;
  return k < m && isleaf[k] ? static_cast<u32>(k) : kNoNode;
}

// One more of node q's children is finished (by this thread's warp, whose
// lanes' values a __syncwarp put before this): its values are visible to
// whoever counts the last one, and the others' to this thread if it does.
__device__ __forceinline__ u32 count_arrival(u32 *arrive) {
  u32 before;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;"
               : "=r"(before)
               : "l"(arrive)
               : "memory");
  return before;
}

// Bottom-up over the whole tree in one launch (above), by teams of kLanes
// lanes: the centres of mass (kQuad false) or, the leaves' quadrupoles and the
// terms being there, the quadrupoles. A block takes per_block leaves (at most
// kMostLeaves), then the nodes its queue holds, turn by turn; a turn hands over
// at most as many nodes as it worked. `arrive` counts each node's finished
// children (zero at the start).
constexpr u32 kUpThreads = 128;
constexpr u32 kMostLeaves = 128;
template <bool kQuad, u32 kAhead>
__global__ void __launch_bounds__(kUpThreads)
    k_moments_up(MomentArrays a, const u32 *bucket, const u32 *meta, const u8 *isleaf, u32 m,
                 u32 per_block, u32 *arrive, const u32 *m_dev, const u32 *abort) {
  grid_wait();
  constexpr u32 kLanes = kQuad ? 8 : 4;
  __shared__ u32 queue[2][kMostLeaves];
  __shared__ u32 queued[2];
  if (aborted(abort)) return;
  m = bounded(m, m_dev);
  const u32 teams = blockDim.x / kLanes, team = threadIdx.x / kLanes;
  const int c = static_cast<int>(threadIdx.x % kLanes);
  const u32 team_mask = ((1u << kLanes) - 1u) << (threadIdx.x & 31u & ~(kLanes - 1u));
  if (threadIdx.x < 2) queued[threadIdx.x] = 0u;
  __syncthreads();
  auto hand_over = [&](int next, u32 q, u32 children) {
    if (q != kNoNode && count_arrival(&arrive[q]) + 1u == children)
      queue[next][atomicAdd(&queued[next], 1u)] = q;
  };
  const u64 first = static_cast<u64>(blockIdx.x) * per_block;
  if (kQuad) {  // the leaves only count
    for (u32 i = threadIdx.x; i < per_block; i += blockDim.x) {
      const u32 p = nth_leaf(first + i, bucket, meta, isleaf, m);
      if (p == kNoNode) continue;
      const u32 q = a.parent[p];
      hand_over(0, q, q != kNoNode ? a.nchild[q] : 0u);
    }
  } else {
    for (u32 i = team; i < per_block; i += teams) {
      const u32 p = nth_leaf(first + i, bucket, meta, isleaf, m);
      if (p == kNoNode) continue;
      const u32 q = a.parent[p], children = q != kNoNode ? a.nchild[q] : 0u;
      leaf_com<kAhead>(a, p, c, team_mask);
      __syncwarp(team_mask);
      if (c == 0) hand_over(0, q, children);
    }
  }
  for (int turn = 0; turn <= kMaxDepth; ++turn) {
    const int cur = turn & 1;
    __syncthreads();  // this turn's queue is complete, the next one's counter clear
    const u32 count = queued[cur];
    if (count == 0) return;
    for (u32 i = team; i < count; i += teams) {
      const u32 p = queue[cur][i];
      const u32 q = a.parent[p], children = q != kNoNode ? a.nchild[q] : 0u;
      if (!kQuad) node_com(a, p, c, team_mask);
      else if (c < 6) node_quad(a, p, c);
      __syncwarp(team_mask);
      if (c == 0) hand_over(cur ^ 1, q, children);
    }
    __syncthreads();  // read by all before the counter is used again
    if (threadIdx.x == 0) queued[cur] = 0u;
  }
}

// The leaves' quadrupoles, a thread each.
constexpr u32 kLeafThreads = 64;  // small blocks: small trees spread over the SMs
__global__ void __launch_bounds__(kLeafThreads)
    k_leaf_quads(MomentArrays a, const u32 *bucket, const u32 *meta, const u8 *isleaf, u32 m,
                 const u32 *m_dev, const u32 *abort) {
  grid_wait();
  if (aborted(abort)) return;
  const u32 p = nth_leaf(static_cast<u64>(blockIdx.x) * kLeafThreads + threadIdx.x, bucket, meta,
                         isleaf, bounded(m, m_dev));
  if (p != kNoNode) leaf_quad(a, p);
}

// Every node's term in its parent's quadrupole; with `deltas` (no walk
// records, which hold them otherwise) its delta too.
__global__ void __launch_bounds__(kLeafThreads)
    k_quad_terms(MomentArrays a, u32 m, bool deltas, const u32 *m_dev, const u32 *abort) {
  grid_wait();
  const u32 p = blockIdx.x * kLeafThreads + threadIdx.x;
  if (aborted(abort) || p >= bounded(m, m_dev)) return;
  quad_term(a, p);
  if (deltas) a.delta[p] = delta_of(load_pair(a.mom, p), load_pair(a.geom, p));
}

// All of the FP32 moments in one launch, bottom-up: a thread per leaf (in
// the leaf buckets' order) computes its leaf, then climbs while it is the
// last child of its parent to finish, computing that parent from its
// children in child order as node_moments32 does. So every node is computed
// once, after all its children; the climb ends at the root or at a parent a sibling
// will finish (at most kMaxDepth steps).
__global__ void __launch_bounds__(kT)
    k_moments32_up(Moment32Arrays a, const u32 *bucket, const u32 *meta, const u32 *parent,
                   u32 *arrive) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= leaf_count(meta)) return;
  u32 p = bucket[k];
  leaf_moments32(a, p);
  for (int step = 0; step <= kMaxDepth; ++step) {
    const u32 q = parent[p];
    if (q == 0xffffffffu) return;
    if (count_arrival(&arrive[q]) + 1u != a.nchild[q]) return;
    node_moments32(a, q);
    p = q;
  }
}

__global__ void k_root_mass(const float4 *cells32, double2 *rootmom) {
  grid_wait();
  rootmom[0] = make_double2(0.0, 0.0);
  rootmom[1] = make_double2(0.0, static_cast<double>(cells32[0].w));
}

// A graph replay's checks after the node count: an error so far (positions that
// are not finite), deeper keys needed, or a leaf below the sorted levels (bit
// 1), or more nodes than the node arrays hold (bit 2). The host looks at the error
// first; the abort keeps the later kernels from writing results.
__global__ void k_check_tree_graph(Scalars *sc, u32 cap, int sorted_levels) {
  grid_wait();
  if (sc->error || sc->deep > 0 || static_cast<int>(sc->depth) > sorted_levels) sc->abort |= 1u;
  if (sc->n_nodes > cap) sc->abort |= 2u;
}

// --------------------------------------------------------------- packing

// Walk records (FP32 and FP64) of every node (group_lists.cpp:59-61) and the
// deltas: they need the centres of mass only, so they are packed after the
// first moment pass.
__global__ void __launch_bounds__(kT)
    k_pack_walk(const double2 *geom, const double2 *mom, double *delta, const u32 *nbegin,
                const u32 *nend, const u32 *skip, const u8 *isleaf, u32 m, const TreeRoot *root,
                double inv_theta, WalkRec32 *walk32, WalkRec64 *walk64,
                const u32 *m_dev = nullptr, const u32 *abort = nullptr,
                const u16 *sys = nullptr) {
  grid_wait();
  const u32 p = blockIdx.x * kT + threadIdx.x;
  if (aborted(abort) || p >= bounded(m, m_dev)) return;
  if (sys) root += sys[nbegin[p]];  // a forest: relative to the node's system's root
  const Dbl4 g = load_pair(geom, p), c = load_pair(mom, p);
  const double d = delta_of(c, g);
  delta[p] = d;
  const double crit = 2.0 * g.w * inv_theta + d;
  WalkRec64 r;
  r.cx = g.x;
  r.cy = g.y;
  r.cz = g.z;
  r.slack = g.w * 1.0001;
  r.mx = c.x;
  r.my = c.y;
  r.mz = c.z;
  r.crit2 = crit * crit;
  walk64[p] = r;
  const double ox = root->center[0], oy = root->center[1], oz = root->center[2];
  WalkRec32 f;
  f.cx = static_cast<float>(g.x - ox);
  f.cy = static_cast<float>(g.y - oy);
  f.cz = static_cast<float>(g.z - oz);
  f.slack = static_cast<float>(r.slack);
  f.mx = static_cast<float>(c.x - ox);
  f.my = static_cast<float>(c.y - oy);
  f.mz = static_cast<float>(c.z - oz);
  f.crit2 = static_cast<float>(r.crit2);
  f.skip = skip[p];
  f.nbody_leaf = (nend[p] - nbegin[p]) | (isleaf[p] ? 0x80000000u : 0u);
  f.begin = nbegin[p];
  // magnitude bound of this record's FP32 values, rounded up
  const float mag = fmaxf(fmaxf(fmaxf(fabsf(f.cx), fabsf(f.cy)), fmaxf(fabsf(f.cz), fabsf(f.mx))),
                          fmaxf(fabsf(f.my), fabsf(f.mz)));
  f.bound = (mag + f.slack) * (1.0f + 1.0f / (1 << 20));
  walk32[p] = f;
}

// FP32 cell of every node, after the quadrupole pass (group_lists.cpp:52-58).
__global__ void __launch_bounds__(kT)
    k_pack_cells(const double2 *mom, const double2 *quad, const u32 *nbegin, u32 m,
                 const TreeRoot *root, float4 *cells, const u32 *m_dev = nullptr,
                 const u32 *abort = nullptr, const u16 *sys = nullptr) {
  grid_wait();
  const u32 p = blockIdx.x * kT + threadIdx.x;
  if (aborted(abort) || p >= bounded(m, m_dev)) return;
  if (sys) root += sys[nbegin[p]];
  const Dbl4 c = load_pair(mom, p);
  const double ox = root->center[0], oy = root->center[1], oz = root->center[2];
  const double2 qa = quad[3 * p], qb = quad[3 * p + 1], qc = quad[3 * p + 2];
  cells[3 * p] = make_float4(static_cast<float>(c.x - ox), static_cast<float>(c.y - oy),
                             static_cast<float>(c.z - oz), static_cast<float>(c.w));
  cells[3 * p + 1] = make_float4(static_cast<float>(qa.x), static_cast<float>(qa.y),
                                 static_cast<float>(qb.x), static_cast<float>(qb.y));
  cells[3 * p + 2] = make_float4(static_cast<float>(qc.x), static_cast<float>(qc.y), 0.0f, 0.0f);
}

// A forest's FP32 bodies, each relative to its system's root centre.
__global__ void __launch_bounds__(kT)
    k_pack_bodies_forest(const double *tpos, const double *tmass, u32 n, const u16 *sys,
                         const TreeRoot *roots, float4 *bodies, const u32 *abort = nullptr) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= n || aborted(abort)) return;
  const double *o = roots[sys[k]].center;
  bodies[k] = make_float4(static_cast<float>(tpos[3ull * k] - o[0]),
                          static_cast<float>(tpos[3ull * k + 1] - o[1]),
                          static_cast<float>(tpos[3ull * k + 2] - o[2]),
                          static_cast<float>(tmass[k]));
}

// FP32 bodies relative to `origin` (group_lists.cpp:46-50, gravity_backends.cpp:15-23).
__global__ void __launch_bounds__(kT)
    k_pack_bodies(const double *tpos, const double *tmass, u32 n, const double *origin,
                  float4 *bodies, const u32 *abort = nullptr) {
  grid_wait();
  const u32 k = blockIdx.x * kT + threadIdx.x;
  if (k >= n || aborted(abort)) return;
  bodies[k] = make_float4(static_cast<float>(tpos[3ull * k] - origin[0]),
                          static_cast<float>(tpos[3ull * k + 1] - origin[1]),
                          static_cast<float>(tpos[3ull * k + 2] - origin[2]),
                          static_cast<float>(tmass[k]));
}

const double *root_centre(const TreeRoot *root) {
  return reinterpret_cast<const double *>(reinterpret_cast<const char *>(root) +
                                          offsetof(TreeRoot, center));
}

// (The counts read back size buffers and the scans behind them give places: neither
// is used after an error.)
void read_scalars(Workspace &ws, Scalars *host, cudaStream_t s) {
  GTC_CUDA(cudaMemcpyAsync(host, ws.scalars.ptr, sizeof(Scalars), cudaMemcpyDeviceToHost, s));
  GTC_CUDA(cudaStreamSynchronize(s));
  check_device_error(host->error);
}

}  // namespace

void bbox_root(Workspace &ws, const double *pos, u64 n, cudaStream_t s, bool split) {
  const u32 nparts = std::min<u32>(1024, std::max<u32>(1, ceil_div(n, kT)));
  ws.bbox_part.ensure(6 * sizeof(u64) * nparts);
  ws.root.ensure(sizeof(TreeRoot));
  if (!ws.bbox_ticket.ptr) {
    ws.bbox_ticket.ensure(sizeof(u32));
    GTC_CUDA(cudaMemsetAsync(ws.bbox_ticket.ptr, 0, sizeof(u32), s));
  }
  if (split) ws.split.ensure(3ull * kSplitSize * sizeof(double));
  launch(k_bbox, nparts, kT, 0, s, pos, n, ws.bbox_part.as<u64>(), ws.bbox_ticket.as<u32>(),
         ws.root.as<TreeRoot>(), split ? ws.split.as<double>() : nullptr);
  GTC_LAUNCH_CHECK();
}

void pack_bodies_bbox(Workspace &ws, const double *pos, const double *mass, u64 n,
                      cudaStream_t s) {
  bbox_root(ws, pos, n, s, false);
  ws.bodies.ensure(n * sizeof(float4));
  const TreeRoot *root = ws.root.as<TreeRoot>();
  launch(k_pack_bodies, ceil_div(n, kT), kT, 0, s, pos, mass, static_cast<u32>(n),
         root_centre(root), ws.bodies.as<float4>());
  GTC_LAUNCH_CHECK();
}

void ensure_side(Workspace &ws) {
  if (ws.side) return;
  GTC_CUDA(cudaStreamCreateWithFlags(&ws.side, cudaStreamNonBlocking));
  GTC_CUDA(cudaEventCreateWithFlags(&ws.side_fork, cudaEventDisableTiming));
  GTC_CUDA(cudaEventCreateWithFlags(&ws.side_done, cudaEventDisableTiming));
  GTC_CUDA(cudaEventCreateWithFlags(&ws.side_walk, cudaEventDisableTiming));
}

cudaStream_t fork_side(Workspace &ws, cudaStream_t s) {
  ensure_side(ws);
  GTC_CUDA(cudaEventRecord(ws.side_fork, s));
  GTC_CUDA(cudaStreamWaitEvent(ws.side, ws.side_fork, 0));
  ws.side_pending = true;
  ws.walk_pending = false;
  return ws.side;
}

void join_side(Workspace &ws, cudaStream_t s) {
  ws.walk_pending = false;
  if (!ws.side_pending) return;
  ws.side_pending = false;
  if (cudaEventRecord(ws.side_done, ws.side) == cudaSuccess)
    cudaStreamWaitEvent(s, ws.side_done, 0);
}

void mark_walk_ready(Workspace &ws, cudaStream_t side) {
  ws.stage(Workspace::kStMomW, side);
  GTC_CUDA(cudaEventRecord(ws.side_walk, side));
  ws.walk_pending = true;
}

void join_walk(Workspace &ws, cudaStream_t s) {
  if (!ws.walk_pending) {
    join_side(ws, s);  // no walk mark: all of the side stream's work
    return;
  }
  ws.walk_pending = false;
  GTC_CUDA(cudaStreamWaitEvent(s, ws.side_walk, 0));
}

namespace {
// The first key word of every body.
void make_keys(Workspace &ws, const double *pos, u32 n, const TreeRoot *root, cudaStream_t s) {
  launch(k_keys, ceil_div(n, kT), kT, 0, s, pos, n, ws.forest.sys, root, ws.key0.as<u64>(),
         ws.idx.as<u32>(), ws.tiny.as<u8>(), &ws.scalars.as<Scalars>()->error);
  GTC_LAUNCH_CHECK();
}

// Sorts the (key, body) pairs on the first `levels` levels of the first key
// word, rounded up to whole 8-bit passes (21 or more: the whole word), and
// returns the levels the order is exact for. Bodies that share those levels
// keep their input order, which is all the tree needs while no leaf lies
// deeper. A forest's pairs are then sorted by system, stably: (system,
// key), each system at its own bodies' positions.
int sort_top_levels(Workspace &ws, u32 n, int levels, cudaStream_t s) {
  const int passes = levels >= kLevelsPerWord ? 8 : (3 * std::max(levels, 1) + 7) / 8;
  const int low = std::max(0, 3 * kLevelsPerWord - 8 * passes);
  ws.sort_passes = passes;
  u32 *err = &ws.scalars.as<Scalars>()->error;
  radix_sort_pairs(ws.key0.as<u64>(), ws.idx.as<u32>(), ws.key0_alt.as<u64>(),
                   ws.idx_alt.as<u32>(), n, 3 * kLevelsPerWord - low, ws.radix, s, low, err);
  if (ws.forest) {
    const ForestView &fv = ws.forest;
    ws.dkey.ensure(n * 8ull);
    ws.dkey_alt.ensure(n * 8ull);
    ws.drec.ensure(n * 4ull);
    ws.drec_alt.ensure(n * 4ull);
    u64 *skey = ws.dkey.as<u64>();
    u32 *spos = ws.drec.as<u32>();
    const u32 nb = ceil_div(n, kT);
    launch(k_forest_sys_keys, nb, kT, 0, s, ws.key0.as<u64>(), ws.idx.as<u32>(), fv.sys, n, skey,
           spos, ws.key0_alt.as<u64>(), ws.idx_alt.as<u32>(), err);
    GTC_LAUNCH_CHECK();
    int bits = 1;
    while (bits < 16 && (1u << bits) < fv.systems) ++bits;
    radix_sort_pairs(skey, spos, ws.dkey_alt.as<u64>(), ws.drec_alt.as<u32>(), n, bits, ws.radix,
                     s, 0, err);
    launch(k_forest_gather, nb, kT, 0, s, spos, ws.key0_alt.as<u64>(), ws.idx_alt.as<u32>(), n,
           ws.key0.as<u64>(), ws.idx.as<u32>(), err);
    GTC_LAUNCH_CHECK();
  }
  return low == 0 ? kLevelsPerWord : (3 * kLevelsPerWord - low) / 3;
}

// A forest's root cubes and split tables (one per system).
void forest_roots_and_tables(Workspace &ws, const double *pos, cudaStream_t s) {
  const ForestView &fv = ws.forest;
  ws.bbox_part.ensure(6 * sizeof(u64) * fv.bbox_nblocks);
  ws.split.ensure((3ull * fv.systems << fv.split_levels) * sizeof(double));
  launch(k_bbox_forest, fv.bbox_nblocks, kT, 0, s, pos, fv.bbox_blocks, fv.start,
         ws.bbox_part.as<u64>());
  GTC_LAUNCH_CHECK();
  launch(k_root_forest, fv.systems, kT, 0, s, ws.bbox_part.as<u64>(), fv.sys_blocks, fv.roots,
         fv.split_levels, ws.split.as<double>());
  GTC_LAUNCH_CHECK();
}

void forest_roots(Workspace &ws, const u32 *abort, cudaStream_t s) {
  const ForestView &fv = ws.forest;
  launch(k_forest_roots, ceil_div(fv.systems, kT), kT, 0, s, fv.start, fv.systems,
         ws.count.as<u32>(), ws.count_scan.as<u32>(), ws.scalars.as<Scalars>(), fv.root_node,
         ws.parent.as<u32>(), abort);
  GTC_LAUNCH_CHECK();
}

void pack_bodies_tree(Workspace &ws, u32 n, const TreeRoot *root, const u32 *abort,
                      cudaStream_t s) {
  if (ws.forest) {
    launch(k_pack_bodies_forest, ceil_div(n, kT), kT, 0, s, ws.tpos.as<double>(),
           ws.tmass.as<double>(), n, ws.forest.sys, ws.forest.roots, ws.bodies.as<float4>(),
           abort);
  } else {
    launch(k_pack_bodies, ceil_div(n, kT), kT, 0, s, ws.tpos.as<double>(), ws.tmass.as<double>(),
           n, root_centre(root), ws.bodies.as<float4>(), abort);
  }
  GTC_LAUNCH_CHECK();
}

// A build's moment launches: m nodes (a replay: at most; the count and the
// abort word on the device).
struct MomentPlan {
  MomentArrays ma;
  const u32 *bucket, *meta;  // null: small trees take their leaves in node order
  u32 m;
  u32 *arrive;               // two counts per node, one for each pass
  const u32 *m_dev, *abort;
};

// Below this many nodes the three launches that sort the leaves by size cost
// more than the warps' uneven loops.
constexpr u32 kBucketNodes = 65536;

u64 arrive_bytes(u64 m) { return 2 * m * sizeof(u32); }

MomentPlan plan_moments(Workspace &ws, u32 m, bool buckets, cudaStream_t s,
                        const u32 *m_dev = nullptr, const u32 *abort = nullptr) {
  MomentPlan p{};
  p.m = m;
  p.m_dev = m_dev;
  p.abort = abort;
  p.ma = MomentArrays{ws.geom.as<double2>(), ws.nbegin.as<u32>(), ws.nend.as<u32>(),
                      ws.skip.as<u32>(), ws.parent.as<u32>(), ws.nchild.as<u8>(),
                      ws.kids.as<uint4>(), ws.tpos.as<double>(), ws.tmass.as<double>(),
                      ws.mom.as<double2>(), ws.quad.as<double2>(), ws.delta.as<double>(),
                      ws.qterm.as<double>()};
  p.arrive = ws.climb.as<u32>();
  const bool use_buckets = buckets || m >= kBucketNodes;
  clear({{p.arrive, arrive_bytes(m)},
         {ws.arrive.ptr, use_buckets ? 2 * kBuckets * sizeof(u32) : 0}},
        s);
  if (use_buckets) {
    u32 *meta = ws.arrive.as<u32>(), *bucket = ws.bucket.as<u32>();
    const BucketView bv{ws.isleaf.as<u8>(), ws.nbegin.as<u32>(), ws.nend.as<u32>()};
    launch(k_bucket_count, ceil_div(m, kT), kT, 0, s, bv, m, meta, m_dev, abort);
    GTC_LAUNCH_CHECK();
    launch(k_bucket_fill, ceil_div(m, kT), kT, 0, s, bv, m, meta, bucket, m_dev, abort);
    GTC_LAUNCH_CHECK();
    p.bucket = bucket;
    p.meta = meta;
  }
  return p;
}

// Many leaves to a block keep its queue full on the way up; few spread a
// small tree over the SMs. (2M: blocks of 512, 256, 128 threads with a leaf per
// thread take 0.39, 0.33, 0.31 ms for the centres of mass and walk records.)
template <bool kQuad>
void launch_up(const Workspace &ws, const MomentPlan &p, u32 *arrive, cudaStream_t s) {
  const u32 per_block = p.m >= kBucketNodes ? kMostLeaves : 32u;
  launch(p.bucket ? k_moments_up<kQuad, 1> : k_moments_up<kQuad, kQuad ? 1 : 8>,
         ceil_div(p.m, per_block), kUpThreads, 0, s, p.ma, p.bucket, p.meta, ws.isleaf.as<u8>(),
         p.m, per_block, arrive, p.m_dev, p.abort);
  GTC_LAUNCH_CHECK();
}

void launch_coms(const Workspace &ws, const MomentPlan &p, cudaStream_t s) {
  launch_up<false>(ws, p, p.arrive, s);
}

void launch_pack_walk(Workspace &ws, const MomentPlan &p, const TreeRoot *root, double theta,
                      cudaStream_t s) {
  launch(k_pack_walk, ceil_div(p.m, kT), kT, 0, s, ws.geom.as<double2>(), ws.mom.as<double2>(),
         ws.delta.as<double>(), ws.nbegin.as<u32>(), ws.nend.as<u32>(), ws.skip.as<u32>(),
         ws.isleaf.as<u8>(), p.m, root, 1.0 / theta, ws.walk32.as<WalkRec32>(),
         ws.walk64.as<WalkRec64>(), p.m_dev, p.abort, ws.forest.sys);
  GTC_LAUNCH_CHECK();
}

// The quadrupoles, from the centres of mass, and the FP32 cells.
void launch_quads(Workspace &ws, const MomentPlan &p, const TreeRoot *root, bool deltas,
                  cudaStream_t s) {
  const u32 blocks = ceil_div(p.m, kLeafThreads);
  launch(k_leaf_quads, blocks, kLeafThreads, 0, s, p.ma, p.bucket, p.meta, ws.isleaf.as<u8>(),
         p.m, p.m_dev, p.abort);
  GTC_LAUNCH_CHECK();
  launch(k_quad_terms, blocks, kLeafThreads, 0, s, p.ma, p.m, deltas, p.m_dev, p.abort);
  GTC_LAUNCH_CHECK();
  launch_up<true>(ws, p, p.arrive + p.m, s);
  launch(k_pack_cells, ceil_div(p.m, kT), kT, 0, s, ws.mom.as<double2>(), ws.quad.as<double2>(),
         ws.nbegin.as<u32>(), p.m, root, ws.cells.as<float4>(), p.m_dev, p.abort, ws.forest.sys);
  GTC_LAUNCH_CHECK();
}
}  // namespace

void reserve_bodies(Workspace &ws, u64 n) {
  ws.key0.ensure(n * 8);
  ws.key0_alt.ensure(n * 8);
  ws.idx.ensure(n * 4);
  ws.idx_alt.ensure(n * 4);
  ws.tiny.ensure(n);
  ws.lcp.ensure(n);
  ws.leafdepth.ensure(n);
  ws.count.ensure(n * 4);
  ws.count_scan.ensure(n * 4);
  ws.tpos.ensure(n * 24);
  ws.tmass.ensure(n * 8);
  ws.bodies.ensure(n * sizeof(float4));
  ws.scalars.ensure(sizeof(Scalars));
}

void reserve_nodes(Workspace &ws, u64 m) {
  ws.geom.ensure(m * 2 * sizeof(double2));
  ws.mom.ensure(m * 2 * sizeof(double2));
  ws.quad.ensure(m * 3 * sizeof(double2));
  ws.delta.ensure(m * 8);
  ws.nbegin.ensure(m * 4);
  ws.nend.ensure(m * 4);
  ws.skip.ensure(m * 4);
  ws.parent.ensure(m * 4);
  ws.depth.ensure(m);
  ws.nchild.ensure(m);
  ws.kids.ensure(m * 8 * sizeof(u32));
  ws.isleaf.ensure(m);
  ws.arrive.ensure(2 * kBuckets * sizeof(u32));
  ws.climb.ensure(arrive_bytes(m));
  ws.qterm.ensure(m * 6 * sizeof(double));
  ws.bucket.ensure(m * 4);
  ws.walk32.ensure(m * sizeof(WalkRec32));
  ws.walk64.ensure(m * sizeof(WalkRec64));
  ws.cells.ensure(m * 3 * sizeof(float4));
}

void build_tree(Workspace &ws, const double *pos, const double *mass, u64 n,
                const SolverParams &sp, cudaStream_t s, Scalars *host, bool walk_records) {
  ws.n = n;
  ws.n_nodes = 0;
  ws.key_words = 1;
  if (n == 0) return;
  const u32 n32 = static_cast<u32>(n);
  const u32 nb = ceil_div(n, kT);
  const int L = std::max(1, sp.leaf_size);

  reserve_bodies(ws, n);
  join_side(ws, s);  // nothing of an earlier call may still write the buffers
  Scalars *sc = ws.scalars.as<Scalars>();
  clear({{sc, sizeof(Scalars)}}, s);

  ws.stage(Workspace::kStBuild, s);
  const ForestView &fv = ws.forest;
  if (fv) forest_roots_and_tables(ws, pos, s);
  else bbox_root(ws, pos, n, s, true);
  const TreeRoot *root = fv ? fv.roots : ws.root.as<TreeRoot>();
  u64 *key0 = ws.key0.as<u64>();
  u32 *idx = ws.idx.as<u32>();
  u8 *tiny = ws.tiny.as<u8>();
  make_keys(ws, pos, n32, root, s);
  // the levels the last tree needed first; all of them when a leaf lies
  // deeper (sorting the partly sorted pairs again gives the full order)
  ws.stage(Workspace::kStSort0, s);
  const int sorted = sort_top_levels(ws, n32, ws.sort_levels > 0 ? ws.sort_levels : kLevelsPerWord, s);
  ws.stage(Workspace::kStSort1, s);

  KeyView kv{key0, nullptr, nullptr, 1, fv.sys};
  signed char *lcp_next = ws.lcp.as<signed char>();
  u8 *leafdepth = ws.leafdepth.as<u8>();
  // Node numbering: count the nodes ending at each sorted position (with
  // the levels, so that one read back serves both).
  u32 *count = ws.count.as<u32>(), *cscan = ws.count_scan.as<u32>();
  auto count_nodes = [&] {
    exclusive_scan_u32(count, cscan, n, &sc->n_nodes, ws.scan_tmp, s, &sc->error);
  };
  launch(k_levels, nb, kT, 0, s, kv, idx, tiny, n32, L, lcp_next, leafdepth, count, sc);
  GTC_LAUNCH_CHECK();
  count_nodes();
  read_scalars(ws, host, s);
  if (sorted < kLevelsPerWord && static_cast<int>(host->depth) > sorted) {
    sort_top_levels(ws, n32, kLevelsPerWord, s);
    GTC_CUDA(cudaMemsetAsync(&sc->deep, 0, sizeof(u32), s));
    GTC_CUDA(cudaMemsetAsync(&sc->depth, 0, sizeof(u32), s));
    launch(k_levels, nb, kT, 0, s, kv, idx, tiny, n32, L, lcp_next, leafdepth, count, sc);
    GTC_LAUNCH_CHECK();
    count_nodes();
    read_scalars(ws, host, s);
  }
  const bool had_deep = host->deep > 0;

  // Deeper key words for bodies whose leaves lie below the words so far.
  while (host->deep > 0 && kv.words < 3) {
    const int limit = kLevelsPerWord * kv.words;
    DeviceBuffer &wbuf = kv.words == 1 ? ws.key1 : ws.key2;
    wbuf.ensure(n * 8);
    GTC_CUDA(cudaMemsetAsync(wbuf.ptr, 0, n * 8, s));
    ws.flags.ensure(n * 4);
    ws.flags_scan.ensure(n * 4);
    u32 *flag = ws.flags.as<u32>(), *fscan = ws.flags_scan.as<u32>();
    launch(k_deep_flags, nb, kT, 0, s, leafdepth, n32, limit, flag);
    GTC_LAUNCH_CHECK();
    exclusive_scan_u32(flag, fscan, n, &sc->deep, ws.scan_tmp, s, &sc->error);
    read_scalars(ws, host, s);
    const u32 nd = host->deep;
    ws.dpos.ensure(nd * 4ull);
    ws.dkey.ensure(nd * 8ull);
    ws.dkey_alt.ensure(nd * 8ull);
    ws.drec.ensure(nd * 4ull);
    ws.drec_alt.ensure(nd * 4ull);
    const u64 idx_bytes = (nd * 4ull + 15) & ~15ull;
    ws.dtmp.ensure(idx_bytes + nd * 8ull);
    u32 *dpos = ws.dpos.as<u32>(), *drec = ws.drec.as<u32>();
    u32 *didx = ws.dtmp.as<u32>();
    u64 *dword = reinterpret_cast<u64 *>(ws.dtmp.as<char>() + idx_bytes);
    const u32 ndb = ceil_div(nd, kT);
    launch(k_compact, nb, kT, 0, s, flag, fscan, n32, dpos);
    GTC_LAUNCH_CHECK();
    launch(k_deep_keys, ndb, kT, 0, s, kv, dpos, nd, idx, pos, root, tiny, dword, drec, didx);
    GTC_LAUNCH_CHECK();
    // order records by (segment, new word, input order): sort by the word,
    // then stably by segment number
    u64 *dkey = ws.dkey.as<u64>();
    GTC_CUDA(cudaMemcpyAsync(dkey, dword, nd * 8ull, cudaMemcpyDeviceToDevice, s));
    radix_sort_pairs(dkey, drec, ws.dkey_alt.as<u64>(), ws.drec_alt.as<u32>(), nd, 63, ws.radix, s,
                     0, &sc->error);
    u32 *sflag = ws.flags.as<u32>(), *sscan = ws.flags_scan.as<u32>();
    launch(k_deep_segments, ndb, kT, 0, s, kv, dpos, nd, sflag);
    GTC_LAUNCH_CHECK();
    exclusive_scan_u32(sflag, sscan, nd, &sc->aux, ws.scan_tmp, s, &sc->error);
    read_scalars(ws, host, s);
    int seg_bits = 1;
    while (seg_bits < 32 && (1ull << seg_bits) <= host->aux) ++seg_bits;
    launch(k_seg_keys, ndb, kT, 0, s, drec, sscan, sflag, nd, dkey, &sc->error);
    GTC_LAUNCH_CHECK();
    radix_sort_pairs(dkey, drec, ws.dkey_alt.as<u64>(), ws.drec_alt.as<u32>(), nd, seg_bits,
                     ws.radix, s, 0, &sc->error);
    launch(k_deep_scatter, ndb, kT, 0, s, dpos, drec, didx, dword, nd, idx, wbuf.as<u64>(),
           &sc->error);
    GTC_LAUNCH_CHECK();
    if (kv.words == 1) kv.w1 = ws.key1.as<u64>();
    else kv.w2 = ws.key2.as<u64>();
    kv.words += 1;
    GTC_CUDA(cudaMemsetAsync(&sc->deep, 0, sizeof(u32), s));
    launch(k_levels, nb, kT, 0, s, kv, idx, tiny, n32, L, lcp_next, leafdepth, count, sc);
    GTC_LAUNCH_CHECK();
    read_scalars(ws, host, s);
  }
  if (host->deep > 0) throw RuntimeError("octree deeper than the depth cap");
  ws.key_words = kv.words;
  ws.sort_levels = kv.words == 1 ? static_cast<int>(host->depth) + 1 : 0;
  if (had_deep) {  // new key words: count again
    count_nodes();
    read_scalars(ws, host, s);
  }
  const u32 m = host->n_nodes;
  ws.n_nodes = m;
  ws.tree_depth = static_cast<int>(host->depth);
  reserve_nodes(ws, m);
  const u32 mb = ceil_div(m, kT);

  launch(k_nodes, nb, kT, 0, s, kv, lcp_next, leafdepth, count, cscan, n32, sc, root,
         ws.split.as<double>(), ws.geom.as<double2>(), ws.nbegin.as<u32>(), ws.nend.as<u32>(),
         ws.skip.as<u32>(), ws.depth.as<u8>(), ws.isleaf.as<u8>(),
         fv ? fv.split_levels : kSplitLevels, nullptr);
  GTC_LAUNCH_CHECK();
  launch(k_children, mb, kT, 0, s, ws.skip.as<u32>(), ws.isleaf.as<u8>(), m, ws.parent.as<u32>(),
         ws.nchild.as<u8>(), ws.kids.as<uint4>());
  GTC_LAUNCH_CHECK();
  if (fv) forest_roots(ws, nullptr, s);
  launch(k_leaf_order, mb, kT, 0, s, ws.isleaf.as<u8>(), ws.nbegin.as<u32>(), ws.nend.as<u32>(),
         m, idx);
  GTC_LAUNCH_CHECK();
  launch(k_tree_order, nb, kT, 0, s, pos, mass, idx, n32, ws.tpos.as<double>(),
         ws.tmass.as<double>());
  GTC_LAUNCH_CHECK();
  ws.stage(Workspace::kStTopo, s);

  // the moments and node records on the side stream, beside the group choice
  // (which needs none of it): the centres of mass first and the walk records
  // from them (the walk waits for these only), then the quadrupoles and the
  // cells beside the walk
  const MomentPlan mp = plan_moments(ws, m, !walk_records, s);
  cudaStream_t ms = fork_side(ws, s);
  ws.stage(Workspace::kStMom0, ms);
  launch_coms(ws, mp, ms);
  if (walk_records) launch_pack_walk(ws, mp, root, sp.theta, ms);
  mark_walk_ready(ws, ms);
  launch_quads(ws, mp, root, !walk_records, ms);
  ws.stage(Workspace::kStMom1, ms);
  pack_bodies_tree(ws, n32, root, nullptr, s);
}

void moments32(Workspace &ws, float4 *cells32, float *delta32, double2 *rootmom,
               cudaStream_t s) {
  const u32 m = static_cast<u32>(ws.n_nodes);
  if (m == 0) return;
  const Moment32Arrays a{ws.geom.as<double2>(), ws.nbegin.as<u32>(), ws.nend.as<u32>(),
                         ws.nchild.as<u8>(),   ws.kids.as<uint4>(), ws.bodies.as<float4>(),
                         ws.root.as<TreeRoot>(), cells32, delta32};
  const u32 *meta = ws.arrive.as<u32>(), *bucket = ws.bucket.as<u32>();
  ws.up_arrive.ensure(m * sizeof(u32));
  clear({{ws.up_arrive.ptr, m * sizeof(u32)}}, s);
  launch(k_moments32_up, ceil_div(m, kT), kT, 0, s, a, bucket, meta, ws.parent.as<u32>(),
         ws.up_arrive.as<u32>());
  GTC_LAUNCH_CHECK();
  launch(k_root_mass, 1, 1, 0, s, cells32, rootmom);
  GTC_LAUNCH_CHECK();
}

void build_tree_graph(Workspace &ws, const double *pos, const double *mass, u64 n,
                      const SolverParams &sp, const GraphCaps &caps, cudaStream_t s) {
  ws.n = n;
  ws.key_words = 1;
  const u32 n32 = static_cast<u32>(n), mcap = caps.nodes;
  const u32 nb = ceil_div(n, kT), mb = ceil_div(mcap, kT);
  const int L = std::max(1, sp.leaf_size);
  Scalars *sc = ws.scalars.as<Scalars>();
  u32 *abort = &sc->abort;
  clear({{sc, sizeof(Scalars)}}, s);
  const ForestView &fv = ws.forest;
  if (fv) forest_roots_and_tables(ws, pos, s);
  else bbox_root(ws, pos, n, s, true);
  const TreeRoot *root = fv ? fv.roots : ws.root.as<TreeRoot>();
  u64 *key0 = ws.key0.as<u64>();
  u32 *idx = ws.idx.as<u32>();
  u8 *tiny = ws.tiny.as<u8>();
  make_keys(ws, pos, n32, root, s);
  // the levels the captured depth allows: a deeper tree aborts the replay
  const int sorted = sort_top_levels(ws, n32, caps.depth + 1, s);
  const KeyView kv{key0, nullptr, nullptr, 1, fv.sys};
  signed char *lcp_next = ws.lcp.as<signed char>();
  u8 *leafdepth = ws.leafdepth.as<u8>();
  u32 *count = ws.count.as<u32>(), *cscan = ws.count_scan.as<u32>();
  launch(k_levels, nb, kT, 0, s, kv, idx, tiny, n32, L, lcp_next, leafdepth, count, sc);
  GTC_LAUNCH_CHECK();
  exclusive_scan_u32(count, cscan, n, &sc->n_nodes, ws.scan_tmp, s, &sc->error);
  launch(k_check_tree_graph, 1, 1, 0, s, sc, mcap, sorted);
  GTC_LAUNCH_CHECK();
  const u32 *m_dev = &sc->n_nodes;
  launch(k_nodes, nb, kT, 0, s, kv, lcp_next, leafdepth, count, cscan, n32, sc, root,
         ws.split.as<double>(), ws.geom.as<double2>(), ws.nbegin.as<u32>(), ws.nend.as<u32>(),
         ws.skip.as<u32>(), ws.depth.as<u8>(), ws.isleaf.as<u8>(),
         fv ? fv.split_levels : kSplitLevels, abort);
  GTC_LAUNCH_CHECK();
  launch(k_children, mb, kT, 0, s, ws.skip.as<u32>(), ws.isleaf.as<u8>(), mcap,
         ws.parent.as<u32>(), ws.nchild.as<u8>(), ws.kids.as<uint4>(), m_dev, abort);
  GTC_LAUNCH_CHECK();
  if (fv) forest_roots(ws, abort, s);
  launch(k_leaf_order, mb, kT, 0, s, ws.isleaf.as<u8>(), ws.nbegin.as<u32>(), ws.nend.as<u32>(),
         mcap, idx, m_dev, abort);
  GTC_LAUNCH_CHECK();
  launch(k_tree_order, nb, kT, 0, s, pos, mass, idx, n32, ws.tpos.as<double>(),
         ws.tmass.as<double>(), abort);
  GTC_LAUNCH_CHECK();
  // the moments on the side stream, as in the eager build (the walk waits for
  // the walk records, the caller joins the rest before the evaluation)
  const MomentPlan mp = plan_moments(ws, mcap, false, s, m_dev, abort);
  cudaStream_t ms = fork_side(ws, s);
  launch_coms(ws, mp, ms);
  launch_pack_walk(ws, mp, root, sp.theta, ms);
  mark_walk_ready(ws, ms);
  launch_quads(ws, mp, root, false, ms);
  pack_bodies_tree(ws, n32, root, abort, s);
}

}  // namespace gtc
