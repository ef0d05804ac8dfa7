// Stable LSD radix sort of (u64 key, u32 value) pairs, 8 bits per pass, in
// one sweep per pass (after Adinets and Merrill, "Onesweep: a faster least
// significant digit radix sort for GPUs", 2022).
//
// One launch counts the digits of every pass at once (the keys are read
// once for all passes) and one small launch scans them into each digit's
// start in each pass. Then each pass is a single launch: a block takes the
// next tile (2048 pairs) from a counter, ranks its keys stably (each warp
// by ballots and a warp-private histogram, equal digits in input
// order), publishes its digit counts, and finds how many pairs of each digit
// the earlier tiles hold by looking back over their published counts --
// each tile publishes first its own counts, then, once it knows them, the
// running totals up to and including it, so a look-back stops at the first
// running total it meets. The tile is put in digit order in shared memory
// and written out in that order (consecutive threads, consecutive places of
// a digit's run). Per pass a pair is read once and written once (12 B each
// way), with no histogram read or scan launch of its own.
//
// (Time at 2M, six passes: 248 us with __match_any_sync and each load beside its
// ranking, 238 with the loads first, 215 with ballots; 35 us a pass, bound by
// the latencies of a tile's stages. Look-backs of 1 to 16 words a time measure
// the same.)
//
// A look-back waits only on tiles taken earlier from the counter, whose
// blocks are running or done and publish their counts before waiting
// themselves, so the waits end. Each wait is bounded all the same: past the
// limit the kernel records error bit 16 (and the pass's output is garbage, which
// the solve does not use).
//
// Up to kClusterItems pairs a CTA of one thread-block cluster (16 CTAs where the
// GPU takes such clusters, else 8) the whole sort is one launch: the pairs stay
// in registers, a pass ranks them as above, the CTAs write their digit counts
// into each other's shared memory, and each pair goes straight to its place in
// the shared memory of the CTA that will hold it. Two cluster barriers a pass
// replace the counting launches, the look-back and a launch per pass: five
// passes of 5k pairs 64 -> 22 us, of 50k 68 -> 53 us. (One more at the start, after
// which every CTA's shared memory may be written, measures nothing: it is waited
// for behind the first ranking.) With eight pairs a thread
// (to 131072) the one cluster is the slower: a solve of 65k bodies took the same
// either way, one of 80k 0.537 ms against 0.504 in sweeps, of 131072 0.705 and
// 0.661.

#include <utility>

#include "common.cuh"

namespace gtc {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kPerLane = 8;                  // keys per lane per tile
constexpr u32 kTile = kThreads * kPerLane;   // 2048 keys per tile
constexpr u32 kPerWarp = 32 * kPerLane;      // contiguous keys per warp
constexpr int kBins = 256;
constexpr int kMaxPasses = 8;
static_assert(kThreads == kBins, "the scatter gives each thread one digit");

// A tile's published word per digit: flag in the top two bits, count below.
constexpr u64 kAggregate = 1ull << 62;       // this tile's own count
constexpr u64 kInclusive = 2ull << 62;       // the count of this and every earlier tile
constexpr u64 kCountMask = (1ull << 62) - 1;
constexpr int kBack = 4;                     // words a look-back loads at once
constexpr u32 kSpinLimit = 1u << 22;         // polls of one word before giving up
constexpr u32 kSortTimeout = 16u;            // error bit

__device__ __forceinline__ u64 load_relaxed(const u64 *p) {
  u64 v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_relaxed(u64 *p, u64 v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The lanes with digit d among those with a key: one ballot per bit. (Eight
// ballots and their logic are some 24 instructions of a few cycles each;
// __match_any_sync works through the warp's distinct values in turn.)
__device__ __forceinline__ unsigned peers_of(u32 d, bool ok) {
  unsigned peers = __ballot_sync(kFullMask, ok);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const bool bit = (d >> b) & 1u;
    const unsigned m = __ballot_sync(kFullMask, bit);
    peers &= bit ? m : ~m;
  }
  return peers;
}

// Digit counts of every pass: hist[p][d] += pairs whose digit p is d.
__global__ void __launch_bounds__(kThreads)
    k_digit_counts(const u64 *keys, u32 n, int low_bit, int passes, u32 *hist) {
  grid_wait();
  __shared__ u32 h[kMaxPasses][kBins];
  for (int p = 0; p < passes; ++p) h[p][threadIdx.x] = 0;
  __syncthreads();
  for (u64 i = static_cast<u64>(blockIdx.x) * kThreads + threadIdx.x; i < n;
       i += static_cast<u64>(gridDim.x) * kThreads) {
    const u64 k = keys[i];
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(k >> (low_bit + 8 * p)) & 0xff], 1u);
  }
  __syncthreads();
  for (int p = 0; p < passes; ++p)
    if (h[p][threadIdx.x]) atomicAdd(&hist[p * kBins + threadIdx.x], h[p][threadIdx.x]);
}

// Each pass's digit starts: an exclusive scan of its 256 counts (block p).
__global__ void __launch_bounds__(kThreads) k_digit_starts(const u32 *hist, u32 *start) {
  grid_wait();
  __shared__ u32 wsum[kWarps];
  const int d = threadIdx.x, lane = d & 31, warp = d >> 5;
  const u32 c = hist[blockIdx.x * kBins + d];
  u32 incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 v = __shfl_up_sync(kFullMask, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  u32 before = 0;
  for (int w = 0; w < warp; ++w) before += wsum[w];
  start[blockIdx.x * kBins + d] = before + incl - c;
}

__global__ void __launch_bounds__(kThreads)
    k_onesweep(const u64 *keys, const u32 *vals, u64 *keys_out, u32 *vals_out, u32 n, int shift,
               const u32 *digit_start, u64 *status, u32 *tile_counter, u32 *error) {
  grid_wait();
  __shared__ u32 wh[kWarps][kBins];     // per-warp running counts
  __shared__ u32 woff[kWarps][kBins];   // per-warp start within the tile's digit run
  __shared__ u32 dstart[kBins];         // start of each digit's run inside the tile
  __shared__ u64 gout[kBins];           // where each digit's run goes in the output
  __shared__ u64 skey[kTile];           // the tile, sorted by digit
  __shared__ u32 sval[kTile];
  __shared__ u32 wsum[kWarps];
  __shared__ u32 tile_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) tile_s = atomicAdd(tile_counter, 1u);  // tiles in start order
  for (int b = lane; b < kBins; b += 32) wh[warp][b] = 0;
  __syncthreads();
  const u32 tile = tile_s;
  const unsigned lt = (1u << lane) - 1u;
  const u64 tile0 = static_cast<u64>(tile) * kTile;
  const u64 base = tile0 + static_cast<u64>(warp) * kPerWarp;

  u64 key[kPerLane];
  u32 val[kPerLane];
  u32 rank[kPerLane];
  // (all loads first: the ranking's warp barriers would put them in series)
#pragma unroll
  for (int c = 0; c < kPerLane; ++c) {
    const u64 i = base + static_cast<u64>(c) * 32 + lane;
    key[c] = i < n ? keys[i] : 0;
    val[c] = i < n ? vals[i] : 0;
  }
#pragma unroll
  for (int c = 0; c < kPerLane; ++c) {
    const bool ok = base + static_cast<u64>(c) * 32 + lane < n;
    const u32 d = static_cast<u32>((key[c] >> shift) & 0xff);
    const unsigned peers = peers_of(d, ok);
    u32 before = 0;
    if (ok) before = wh[warp][d];
    __syncwarp();
    if (ok && (peers & lt) == 0) wh[warp][d] = before + __popc(peers);
    __syncwarp();
    rank[c] = before + __popc(peers & lt);
  }
  __syncthreads();
  {
    const int d = threadIdx.x;  // kThreads == kBins
    u32 run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      woff[w][d] = run;
      run += wh[w][d];
    }
    // this tile's count of digit d, then the earlier tiles' by looking back
    u64 *mine = status + static_cast<u64>(tile) * kBins + d;
    store_relaxed(mine, (tile == 0 ? kInclusive : kAggregate) | run);
    // Back over the earlier tiles, kBack words at a time: a hop costs an L2 round
    // trip, and the first wave's tiles find few running totals.
    u64 excl = 0;
    bool stop = false;
    for (u32 t = tile; t > 0 && !stop;) {
      u64 v[kBack];
#pragma unroll
      for (int k = 0; k < kBack; ++k)
        v[k] = static_cast<u32>(k) < t
                   ? load_relaxed(status + static_cast<u64>(t - 1 - k) * kBins + d)
                   : kInclusive;
#pragma unroll
      for (int k = 0; k < kBack; ++k) {
        if (stop) continue;
        for (u32 spin = 0; (v[k] >> 62) == 0; ++spin) {
          if (spin == kSpinLimit) {
            atomicOr(error, kSortTimeout);
            v[k] = kInclusive;  // give up: count 0, stop
            break;
          }
          v[k] = load_relaxed(status + static_cast<u64>(t - 1 - k) * kBins + d);
        }
        excl += v[k] & kCountMask;
        stop = (v[k] >> 62) == 2;  // a running total: done
      }
      t = t > kBack ? t - kBack : 0;
    }
    if (tile > 0) store_relaxed(mine, kInclusive | (excl + run));
    gout[d] = digit_start[d] + excl;
    // the digit runs' starts inside the tile: exclusive scan of run
    u32 incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 v = __shfl_up_sync(kFullMask, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    u32 before = 0;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    dstart[d] = before + incl - run;
  }
  __syncthreads();
  // the tile in digit order in shared memory
#pragma unroll
  for (int c = 0; c < kPerLane; ++c) {
    const u64 i = base + static_cast<u64>(c) * 32 + lane;
    if (i >= n) continue;
    const u32 d = static_cast<u32>((key[c] >> shift) & 0xff);
    const u32 local = dstart[d] + woff[warp][d] + rank[c];
    skey[local] = key[c];
    sval[local] = val[c];
  }
  __syncthreads();
  // out in order: consecutive threads write consecutive places of a digit's run
  const u32 count = static_cast<u32>(n - tile0 < kTile ? n - tile0 : kTile);
  for (u32 j = threadIdx.x; j < count; j += kThreads) {
    const u64 k = skey[j];
    const u32 d = static_cast<u32>((k >> shift) & 0xff);
    const u64 dst = gout[d] + (j - dstart[d]);
    keys_out[dst] = k;
    vals_out[dst] = sval[j];
  }
}

// ------------------------------------------- one cluster, all passes

constexpr int kCT = 1024;
constexpr int kCWarps = kCT / 32;
constexpr int kMaxCtas = 16;
constexpr int kMostPerThread = 4;
constexpr u32 kClusterItems = kCT * kMostPerThread;  // pairs per CTA at most

__device__ __forceinline__ u32 cluster_rank() {
  u32 r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_sync() {
  cluster_arrive();
  cluster_wait();
}
// Address of this CTA's shared `p` in CTA `rank` of the cluster.
__device__ __forceinline__ u32 remote(const void *p, u32 rank) {
  u32 a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a)
      : "r"(static_cast<u32>(__cvta_generic_to_shared(p))), "r"(rank));
  return a;
}
__device__ __forceinline__ void put(u32 addr, u32 v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void put(u32 addr, u64 v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

template <int kPer>
struct ClusterSort {
  u64 key[kCT * kPer];
  u32 val[kCT * kPer];
  u32 wh[kCWarps][kBins];      // per-warp digit counts, then starts within a quarter
  u32 quarter[4][kBins];       // eight warps' counts, then starts within the CTA
  u32 table[kMaxCtas][kBins];  // every CTA's digit counts
  u32 start[kBins];            // where this CTA's pairs of each digit go
  u32 wsum[kBins / 32];
};

// CTA r holds the pairs [r kCT kPer, (r + 1) kCT kPer) at the start of every
// pass, item c of a lane at warp * 32 kPer + 32 c + lane of them.
template <int kPer>
__global__ void __launch_bounds__(kCT)
    k_sort_cluster(u64 *keys, u32 *vals, u32 n, u32 ctas, int low_bit, int passes) {
  grid_wait();
  // (a CTA's shared memory may be written once it runs: waited for before the first
  // write into another's, behind the loads and the first ranking)
  cluster_arrive();
  extern __shared__ __align__(16) unsigned char raw[];
  ClusterSort<kPer> &sm = *reinterpret_cast<ClusterSort<kPer> *>(raw);
  constexpr u32 kShare = kCT * kPer;
  const u32 rank = cluster_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const u32 local0 = static_cast<u32>(warp) * 32 * kPer + lane;
  const u32 base = rank * kShare + local0;
  u64 key[kPer];
  u32 val[kPer], place[kPer];
#pragma unroll
  for (int c = 0; c < kPer; ++c) {
    const u32 i = base + 32 * c;
    key[c] = i < n ? keys[i] : 0;
    val[c] = i < n ? vals[i] : 0;
  }
  for (int p = 0; p < passes; ++p) {
    const int shift = low_bit + 8 * p;
    for (int b = lane; b < kBins; b += 32) sm.wh[warp][b] = 0;
    __syncwarp();
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
      const bool ok = base + 32 * c < n;
      const u32 d = static_cast<u32>(key[c] >> shift) & 0xff;
      const unsigned peers = peers_of(d, ok);
      u32 before = 0;
      if (ok) before = sm.wh[warp][d];
      __syncwarp();
      if (ok && (peers & lt) == 0) sm.wh[warp][d] = before + __popc(peers);
      __syncwarp();
      place[c] = before + __popc(peers & lt);
    }
    __syncthreads();
    {  // starts of each warp's pairs of digit d: within eight warps ...
      const u32 d = threadIdx.x & (kBins - 1), q = threadIdx.x / kBins;
      u32 run = 0;
#pragma unroll
      for (int k = 0; k < kCWarps / 4; ++k) {
        const u32 v = sm.wh[q * (kCWarps / 4) + k][d];
        sm.wh[q * (kCWarps / 4) + k][d] = run;
        run += v;
      }
      sm.quarter[q][d] = run;
    }
    __syncthreads();
    if (p == 0) cluster_wait();
    if (threadIdx.x < kBins) {  // ... within the CTA, whose counts all CTAs get
      const u32 d = threadIdx.x;
      u32 run = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const u32 v = sm.quarter[q][d];
        sm.quarter[q][d] = run;
        run += v;
      }
      for (u32 r = 0; r < ctas; ++r) put(remote(&sm.table[rank][d], r), run);
    }
    cluster_sync();
    u32 total = 0, before = 0, incl = 0;
    if (threadIdx.x < kBins) {  // digit starts over the cluster
      for (u32 r = 0; r < ctas; ++r) {
        const u32 v = sm.table[r][threadIdx.x];
        if (r < rank) before += v;
        total += v;
      }
      incl = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 v = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) sm.wsum[warp] = incl;
    }
    __syncthreads();
    if (threadIdx.x < kBins) {
      for (int w = 0; w < warp; ++w) before += sm.wsum[w];
      sm.start[threadIdx.x] = before + incl - total;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
      if (base + 32 * c >= n) continue;
      const u32 d = static_cast<u32>(key[c] >> shift) & 0xff;
      const u32 to = sm.start[d] + sm.quarter[warp / (kCWarps / 4)][d] + sm.wh[warp][d] + place[c];
      const u32 cta = to / kShare, at = to % kShare;
      put(remote(&sm.key[at], cta), key[c]);
      put(remote(&sm.val[at], cta), val[c]);
    }
    cluster_sync();
    // (the pairs are read before the next barrier, behind which the next pass
    // writes)
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
      key[c] = sm.key[local0 + 32 * c];
      val[c] = sm.val[local0 + 32 * c];
    }
  }
#pragma unroll
  for (int c = 0; c < kPer; ++c) {
    const u32 i = base + 32 * c;
    if (i < n) {
      keys[i] = key[c];
      vals[i] = val[c];
    }
  }
}

template <int kPer>
cudaLaunchConfig_t cluster_config(u32 ctas, cudaLaunchAttribute *attr, cudaStream_t s) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = ctas;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kCT);
  cfg.dynamicSmemBytes = sizeof(ClusterSort<kPer>);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

template <int kPer>
void allow_cluster(bool sixteen) {
  GTC_CUDA(cudaFuncSetAttribute(k_sort_cluster<kPer>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(sizeof(ClusterSort<kPer>))));
  if (sixteen)
    GTC_CUDA(cudaFuncSetAttribute(k_sort_cluster<kPer>,
                                  cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

// The CTAs a cluster of the largest kind may have here: 16, 8, or 0 (no such
// cluster fits the GPU).
int cluster_ctas() {
  for (int ctas : {16, 8}) {
    allow_cluster<kMostPerThread>(ctas == 16);
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg =
        cluster_config<kMostPerThread>(static_cast<u32>(ctas), &attr, nullptr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k_sort_cluster<kMostPerThread>, &cfg) ==
            cudaSuccess &&
        clusters > 0)
      return ctas;
    (void)cudaGetLastError();
  }
  return 0;
}

template <int kPer>
void launch_cluster(u64 *keys, u32 *vals, u32 n, int low_bit, int passes, bool sixteen,
                    cudaStream_t s) {
  allow_cluster<kPer>(sixteen);
  u32 ctas = 1;
  while (ctas * kCT * kPer < n) ctas *= 2;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = cluster_config<kPer>(ctas, attr, s);
  add_early_start(cfg, attr);
  GTC_CUDA(cudaLaunchKernelEx(&cfg, k_sort_cluster<kPer>, keys, vals, n, ctas, low_bit, passes));
  GTC_LAUNCH_CHECK();
}

}  // namespace

void radix_sort_pairs(u64 *keys, u32 *vals, u64 *alt_keys, u32 *alt_vals, u32 n, int bits,
                      RadixScratch &scratch, cudaStream_t s, int low_bit, u32 *error) {
  if (n <= 1 || bits <= 0) return;
  const u32 ntiles = ceil_div(n, kTile);
  const int passes = (bits + 7) / 8;
  if (passes > kMaxPasses) throw InvalidArgument("radix sort: more than 64 key bits");
  if (scratch.cluster_ctas < 0) scratch.cluster_ctas = cluster_ctas();
  const u32 ctas = static_cast<u32>(scratch.cluster_ctas);
  if (n <= ctas * kClusterItems) {  // the fewest pairs per thread that fit
    const bool wide = ctas == 16;
    if (n <= ctas * kCT) launch_cluster<1>(keys, vals, n, low_bit, passes, wide, s);
    else if (n <= ctas * kCT * 2) launch_cluster<2>(keys, vals, n, low_bit, passes, wide, s);
    else launch_cluster<4>(keys, vals, n, low_bit, passes, wide, s);
    return;
  }
  // scratch, sized for the most passes whatever this call needs (so that a
  // captured sort of more levels than the eager one finds it allocated):
  // per pass the status words of every tile, then the digit counts, digit
  // starts and tile counters of every pass and an error word; the parts
  // this call uses are zeroed
  const u64 status_max = static_cast<u64>(kMaxPasses) * ntiles * kBins;
  const u64 small = 2ull * kMaxPasses * kBins + kMaxPasses + 2;
  scratch.counts.ensure(status_max * sizeof(u64) + small * sizeof(u32));
  u64 *status = scratch.counts.as<u64>();
  u32 *hist = reinterpret_cast<u32 *>(status + status_max);
  u32 *start = hist + kMaxPasses * kBins;
  u32 *tiles = start + kMaxPasses * kBins;
  u32 *own_error = tiles + kMaxPasses;
  clear({{status, static_cast<u64>(passes) * ntiles * kBins * sizeof(u64)},
         {hist, small * sizeof(u32)}},
        s);
  int dev = 0, sms = 0;
  GTC_CUDA(cudaGetDevice(&dev));
  GTC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const u32 hblocks = std::min<u32>(ceil_div(n, kThreads), 4u * static_cast<u32>(sms));
  launch(k_digit_counts, hblocks, kThreads, 0, s, keys, n, low_bit, passes, hist);
  GTC_LAUNCH_CHECK();
  launch(k_digit_starts, passes, kThreads, 0, s, hist, start);
  GTC_LAUNCH_CHECK();

  // Ping-pong between the two buffers; an odd number of passes ends with
  // one copy back.
  u64 *src_k = keys, *dst_k = alt_keys;
  u32 *src_v = vals, *dst_v = alt_vals;
  for (int p = 0; p < passes; ++p) {
    launch(k_onesweep, ntiles, kThreads, 0, s, src_k, src_v, dst_k, dst_v, n, low_bit + 8 * p,
           start + p * kBins, status + static_cast<u64>(p) * ntiles * kBins, tiles + p,
           error ? error : own_error);
    GTC_LAUNCH_CHECK();
    std::swap(src_k, dst_k);
    std::swap(src_v, dst_v);
  }
  if (src_k != keys) {
    GTC_CUDA(cudaMemcpyAsync(keys, src_k, static_cast<u64>(n) * sizeof(u64),
                             cudaMemcpyDeviceToDevice, s));
    GTC_CUDA(cudaMemcpyAsync(vals, src_v, static_cast<u64>(n) * sizeof(u32),
                             cudaMemcpyDeviceToDevice, s));
  }
}

}  // namespace gtc
