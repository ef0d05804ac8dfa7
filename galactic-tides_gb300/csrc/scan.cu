// Device-wide exclusive prefix sums, in one launch: node numbering, group
// offsets, list offsets.
//
// Up to kSmall elements one block scans all of them. Beyond, a block takes the
// next tile from a counter, publishes the tile's sum, and finds the sum of the
// earlier tiles by looking back over what they published, 32 at a time: each
// tile's own sum first, then, once known, the running sum up to and including
// it, at which a look-back stops (Merrill and Garland, "Single-pass parallel
// prefix scan with decoupled look-back", 2016). A look-back waits only on
// tiles taken earlier, whose blocks publish before they wait; each wait is
// bounded all the same, and past the bound sets error bit 16. Sums of tiles,
// their scan and the addition as three launches took 10 us where one takes 4.

#include <algorithm>

#include "common.cuh"

namespace gtc {
namespace {

constexpr int kThreads = 256;
constexpr int kItems = 8;
constexpr u32 kTile = kThreads * kItems;

template <class T>
__device__ T warp_inclusive(T v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T t = __shfl_up_sync(kFullMask, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Exclusive scan of one value per thread across the block; *total gets the sum.
template <int kThreads, class T>
__device__ T block_exclusive(T v, T *warp_sums, T *total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T incl = warp_inclusive(v);
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    T w = lane < kThreads / 32 ? warp_sums[lane] : T(0);
    w = warp_inclusive(w);
    if (lane < kThreads / 32) warp_sums[lane] = w;
  }
  __syncthreads();
  const T before = warp > 0 ? warp_sums[warp - 1] : T(0);
  *total = warp_sums[kThreads / 32 - 1];
  __syncthreads();
  return before + incl - v;
}

constexpr u64 kAggregate = 1ull << 62;  // a tile's own sum
constexpr u64 kInclusive = 2ull << 62;  // the sum of it and every earlier tile
constexpr u64 kValueMask = (1ull << 62) - 1;
constexpr u32 kSpinLimit = 1u << 22;    // polls before giving up
constexpr u32 kScanTimeout = 16u;       // error bit

__device__ __forceinline__ u64 load_relaxed(const u64 *p) {
  u64 v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_relaxed(u64 *p, u64 v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The sum of the tiles before `tile`, by one warp.
__device__ u64 look_back(const u64 *status, u32 tile, u32 *error) {
  const int lane = threadIdx.x & 31;
  u64 sum = 0;
  for (long long t = static_cast<long long>(tile) - 1; t >= 0; t -= 32) {
    const long long mine = t - lane;
    u64 v = kInclusive;  // (before the first tile: zero)
    for (u32 spin = 0;; ++spin) {
      if (mine >= 0) v = load_relaxed(status + mine);
      if (__all_sync(kFullMask, (v >> 62) != 0)) break;
      if (spin == kSpinLimit) {  // the same for every lane
        if (lane == 0) atomicOr(error, kScanTimeout);
        return sum;
      }
    }
    const unsigned running = __ballot_sync(kFullMask, (v >> 62) == 2);
    const int stop = running ? __ffs(static_cast<int>(running)) - 1 : 31;
    u64 part = lane <= stop ? v & kValueMask : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(kFullMask, part, o);
    sum += part;
    if (running) break;
  }
  return sum;
}

template <class T>
__global__ void __launch_bounds__(kThreads)
    k_scan(const T *in, T *out, u64 n, T *total_dev, u64 *status, u32 *counter, u32 *error) {
  grid_wait();
  __shared__ T ws[kThreads / 32];
  __shared__ u32 tile_s;
  __shared__ u64 before_s;
  if (threadIdx.x == 0) tile_s = atomicAdd(counter, 1u);
  __syncthreads();
  const u32 tile = tile_s;
  const u64 base = static_cast<u64>(tile) * kTile + static_cast<u64>(threadIdx.x) * kItems;
  T v[kItems];
  T local = 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const u64 i = base + k;
    v[k] = i < n ? in[i] : T(0);
    local += v[k];
  }
  T total;
  T run = block_exclusive<kThreads>(local, ws, &total);
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0)
      store_relaxed(status + tile, (tile == 0 ? kInclusive : kAggregate) | static_cast<u64>(total));
    const u64 before = look_back(status, tile, error);
    if (threadIdx.x == 0) {
      if (tile > 0) store_relaxed(status + tile, kInclusive | (before + static_cast<u64>(total)));
      before_s = before;
    }
  }
  __syncthreads();
  run += static_cast<T>(before_s);
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const u64 i = base + k;
    if (i < n) out[i] = run;
    run += v[k];
  }
  if (total_dev && tile == gridDim.x - 1 && threadIdx.x == kThreads - 1) *total_dev = run;
}

constexpr int kSmallThreads = 1024;
constexpr u64 kSmall = kSmallThreads * kItems;

template <class T>
__global__ void __launch_bounds__(kSmallThreads)
    k_scan_small(const T *in, T *out, u32 n, T *total_dev) {
  grid_wait();
  __shared__ T ws[kSmallThreads / 32];
  const u32 base = threadIdx.x * kItems;
  T v[kItems];
  T local = 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    v[k] = base + k < n ? in[base + k] : T(0);
    local += v[k];
  }
  T total;
  T run = block_exclusive<kSmallThreads>(local, ws, &total);
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (total_dev && threadIdx.x == kSmallThreads - 1) *total_dev = run;
}

struct ClearRanges {
  u32 *ptr[kClearRanges];
  u64 words[kClearRanges];
};
__global__ void __launch_bounds__(kThreads) k_clear(ClearRanges r) {
  grid_wait();
  const u64 first = blockIdx.x * static_cast<u64>(kThreads) + threadIdx.x,
            stride = static_cast<u64>(gridDim.x) * kThreads;
#pragma unroll
  for (int k = 0; k < kClearRanges; ++k) {
    u32 *p = r.ptr[k];
    const u64 words = r.words[k];
    const u64 vectors = (reinterpret_cast<uintptr_t>(p) & 15) == 0 ? words / 4 : 0;
    for (u64 i = first; i < vectors; i += stride)
      reinterpret_cast<uint4 *>(p)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (u64 i = 4 * vectors + first; i < words; i += stride) p[i] = 0u;
  }
}

// Scratch: the tiles' words, their counter and an error word.
u64 scratch_bytes(u64 n) { return (n + kTile - 1) / kTile * sizeof(u64) + 4 * sizeof(u32); }

template <class T>
void scan_impl(const T *in, T *out, u64 n, T *total_dev, DeviceBuffer &tmp, cudaStream_t s,
               u32 *error) {
  if (n == 0) {
    if (total_dev) GTC_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(T), s));
    return;
  }
  if (n <= kSmall) {
    launch(k_scan_small<T>, 1, kSmallThreads, 0, s, in, out, static_cast<u32>(n), total_dev);
    GTC_LAUNCH_CHECK();
    return;
  }
  const u32 tiles = ceil_div(n, kTile);
  tmp.ensure(scratch_bytes(n));
  u64 *status = tmp.as<u64>();
  u32 *counter = reinterpret_cast<u32 *>(status + tiles);
  clear({{tmp.ptr, scratch_bytes(n)}}, s);
  launch(k_scan<T>, tiles, kThreads, 0, s, in, out, n, total_dev, status, counter,
         error ? error : counter + 1);
  GTC_LAUNCH_CHECK();
}

}  // namespace

void clear(std::initializer_list<ClearRange> ranges, cudaStream_t s) {
  ClearRanges r{};
  u64 most = 0;
  int k = 0;
  for (const ClearRange &c : ranges) {
    if (k == kClearRanges || c.bytes % 4) throw RuntimeError("clear: ranges");
    r.ptr[k] = static_cast<u32 *>(c.ptr);
    r.words[k++] = c.bytes / 4;
    most = std::max(most, c.bytes);
  }
  if (most == 0) return;
  launch(k_clear, static_cast<u32>(std::min<u64>(1024, (most + 4095) / 4096)), kThreads, 0, s, r);
  GTC_LAUNCH_CHECK();
}

void exclusive_scan_u32(const u32 *in, u32 *out, u64 n, u32 *total_dev, DeviceBuffer &tmp,
                        cudaStream_t s, u32 *error) {
  scan_impl<u32>(in, out, n, total_dev, tmp, s, error);
}

void exclusive_scan_u64(const u64 *in, u64 *out, u64 n, u64 *total_dev, DeviceBuffer &tmp,
                        cudaStream_t s, u32 *error) {
  scan_impl<u64>(in, out, n, total_dev, tmp, s, error);
}

void reserve_scans(DeviceBuffer &tmp, u64 n) { tmp.ensure(scratch_bytes(n)); }

}  // namespace gtc
