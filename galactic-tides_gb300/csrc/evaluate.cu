// Warp-per-group evaluation of grouped interaction lists, FP32.
//
// Same arithmetic as the reference's shared kernels (gt_body / gt_cell,
// include/galactic_tides/kernels/gravity_kernels.h:71-135) and the same
// order -- all cells in list order, then all bodies in list order, skipping
// the target itself (gt_group_accel, :162-170) -- with FMA contraction and
// the SFU reciprocal square root (rsqrtf; in the packed kernel the SFU
// instruction itself, rsqrt_normal, as every softened r^2 is a normal
// float) instead of 1/sqrt.
//
// Packed FP32x2: a lane holds two targets of its group, one in each half of
// its float2 registers, and every FFMA2 / FMUL2 / FADD2 works one list entry
// against both. Entries (48-byte cells, 16-byte bodies) are copied from
// global to shared memory by cp.async, two per lane and round, a round ahead
// of the arithmetic; a slot past the list is filled with zeros, whose zero
// mass and quadrupole add exactly zero to a softened sum. The staged entries
// come back as broadcast loads, and the factor G multiplies the sums once.
//
// What bounds the kernel is the FP32 FMA pipe: 33 packed instructions per
// cell and target pair, 13 per body. A packed instruction holds the pipe two
// cycles when its operands allow; with three different register pairs it
// takes three (measured in a loop of them: 3.1 cycles, 2.3 with two pairs),
// so the inner loop alone runs at 80 cycles for 66 of arithmetic. Scalar
// FFMAs measured no faster (88 cycles: issue). Pairing two targets instead of
// two entries halves the shared-memory bytes per interaction (the pipe to
// shared memory was 83% busy, now 43%), and the copies a round ahead take
// the list's latency off the warps, so 5 blocks of 4 warps (96 registers)
// serve better than 32 warps per SM did. Copies through L1 (.ca) gain 1% over
// copies past it: neighbouring groups share cells.
//
// Lane fill: a group of T targets has P = ceil(T / 2) target pairs. Its lists
// are cut into S slices, and the (slice, pair) slots v = s P + q go to the
// lanes 32 at a time, a pass each, so that ceil(S P / 32) passes keep nearly
// every lane busy whatever T is (94% of the lanes' work is real at 200k). S is
// chosen per group from T and the list lengths alone (choose_slices). Each
// target's partial sums are added in slice order, so the result does not
// depend on which warp ran which pass.
//
// With many groups one warp works a group's passes one after another (groups
// handed out by an atomic counter). Below kTeamGroups the four warps of a
// block share a group's passes, so that long lists do not run alone at the
// end. From there to kWarpGroups a warp still has only a few groups to work,
// and a group whose box spans much of the system (its list several times the
// mean) ran on alone when the rest was done: such long groups are worked
// first, by teams, and the others by a warp each. 200k bodies with one list of
// 8765 entries (mean 1340): 0.415 -> 0.343 ms; with none above twice the mean 0.335
// -> 0.342, 400k (17.7k groups) 0.637 -> 0.659, where it is not used.
//
// Kernel times against a kernel pairing two entries for one target, a warp per
// group, the next round's entries loaded only when needed (seed 1 galaxies,
// quadrupoles): 5k bodies 139 -> 32 us (86 with a warp per group), 50k 140 -> 101
// us (133), 200k (8.9k groups) 359 -> 332 us (359 with all in teams), 2M 3.26 -> 3.21
// ms; monopoles only (a scalar kernel before) 200k 276 -> 219 us, 2M 2.39 -> 1.97 ms.

#include <algorithm>

#include "pipeline.cuh"

namespace gtc {
namespace {

constexpr int kWarpsPerBlock = 4;
constexpr int kT = 32 * kWarpsPerBlock;
constexpr int kBlocksPerSm = 5;   // 96 registers: 2M 3.21 ms; 4: 3.24, 6: 3.26, 7: 3.4 ms
constexpr float kSoftEps2 = 1e-14f;  // eps^-5 stays below 1e35
constexpr int kNoGroups = 0, kAllGroups = 1, kLongGroups = 2;  // worked by teams
constexpr u32 kNone = 0xffffffffu;
constexpr u32 kMaxSlices = 32;    // slices per group at most
constexpr u32 kStage = 64;        // entries a warp stages per round, two per lane
constexpr int kPer = kStage / 32;    // entries a lane stages per round
constexpr u32 kChunk = 256;       // entries a slice holds at most (up to kMaxSlices slices)

// Target i's results (tree order) into eo: the FP32 record, and the caller's
// FP64 arrays (FP32 -> FP64 exactly) and |a| when eo asks for them.
__device__ __forceinline__ void write_target(const EvalOut &eo, u32 i, float4 a) {
  eo.out[i] = a;
  if (!eo.acc) return;
  const u64 j = eo.order[i];
  eo.acc[3 * j] = a.x;
  eo.acc[3 * j + 1] = a.y;
  eo.acc[3 * j + 2] = a.z;
  eo.pot[j] = a.w;
  if (eo.amag) eo.amag[j] = sqrtf(__fmaf_rn(a.x, a.x, __fmaf_rn(a.y, a.y, __fmul_rn(a.z, a.z))));
}

// Slices for a group of T targets with ec cells and eb bodies (warp-uniform):
// of the S in 1..32 whose slices hold at most kChunk entries, the one that
// minimises passes x (entries per slice + pass_cost); 32 when the lists are
// longer than that. pass_cost is a pass's fixed cost in entries worked
// against one target: half as many against the lane's two.
__device__ __forceinline__ u32 choose_slices(u32 T, u32 ec, u32 eb, int lane, u32 pass_cost) {
  const u32 P = (T + 1) / 2;
  const u32 S = static_cast<u32>(lane) + 1u;
  const u32 passes = (S * P + 31u) / 32u;
  const u32 each = (ec + S - 1) / S + (eb + S - 1) / S;
  const u32 cost = each <= kChunk ? passes * (each + pass_cost / 2u) : (1u << 26);
  // ties: the most slices
  return kMaxSlices - (__reduce_min_sync(kFullMask, cost << 5 | (kMaxSlices - S)) & 31u);
}

// 16 (8) bytes from global to shared memory without a register in between;
// zeros where `real` is false.
__device__ __forceinline__ void copy_async16(void *dst, const void *src, bool real) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<u32>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(real ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copy_async8(void *dst, const void *src, bool real) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                   static_cast<u32>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(real ? 8 : 0)
               : "memory");
}
template <bool kQuad>
__device__ __forceinline__ void copy_cell(float4 *dst, const float4 *cells, u32 c) {
  const bool real = c != kNone;
  const float4 *src = cells + 3ull * (real ? c : 0u);
  copy_async16(dst, src, real);
  if (kQuad) {
    copy_async16(dst + 1, src + 1, real);
    copy_async8(dst + 2, src + 2, real);
  }
}

// A list of e entries cut into S nearly equal slices: the entry slice s
// starts at.
struct Cut {
  u32 base, rest;
  __device__ __forceinline__ Cut(u32 e, u32 S) : base(e / S), rest(e % S) {}
  __device__ __forceinline__ u32 at(u32 s) const { return base * s + min(s, rest); }
  __device__ __forceinline__ u32 longest() const { return base + (rest ? 1u : 0u); }
};

// a / b for a below 2^12, from r = 1 / b: (a + 1/2) / b is at least 1 / 2b from
// a whole number, far more than the roundings.
__device__ __forceinline__ u32 small_div(u32 a, float r) {
  return static_cast<u32>((static_cast<float>(a) + 0.5f) * r);
}

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

// A lane's two targets, one in each half of the pairs, and what has been
// summed onto them.
struct Targets {
  float2 px, py, pz;
  float2 ax, ay, az, pot;
};

// One staged body (or monopole) against the lane's targets, without the
// factor -G (applied once to the sums): d = source - target; without
// softening, self0 / self1 leave the target itself out.
template <bool kSoft>
__device__ __forceinline__ void add_body(Targets &a, const float4 b, const float2 e2,
                                         bool self0 = false, bool self1 = false) {
  const float2 dx = __fadd2_rn(dup(b.x), a.px), dy = __fadd2_rn(dup(b.y), a.py),
               dz = __fadd2_rn(dup(b.z), a.pz);
  float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
  float2 m = dup(b.w);
  if (!kSoft) {
    r2 = f2(self0 ? 1.f : r2.x, self1 ? 1.f : r2.y);
    m = f2(self0 ? 0.f : m.x, self1 ? 0.f : m.y);
  }
  const float2 inv = kSoft ? f2(rsqrt_normal(r2.x), rsqrt_normal(r2.y))
                           : f2(rsqrtf(r2.x), rsqrtf(r2.y));
  const float2 mr = __fmul2_rn(m, inv);                     // m / r
  const float2 mr3 = __fmul2_rn(mr, __fmul2_rn(inv, inv));  // m / r^3
  a.ax = __ffma2_rn(mr3, dx, a.ax);
  a.ay = __ffma2_rn(mr3, dy, a.ay);
  a.az = __ffma2_rn(mr3, dz, a.az);
  a.pot = __fadd2_rn(a.pot, mr);
}

// One staged cell with its quadrupole (q: Qxx, Qyy, Qzz, Qxy; w: Qxz, Qyz),
// d = source - target: a / G = m d / r^3 - Q d / r^5 + 5/2 (d.Q.d) d / r^7, phi
// / -G = m / r + 1/2 d.Q.d / r^5; r.Q.r / r^5 once for both.
template <bool kSoft>
__device__ __forceinline__ void add_cell(Targets &a, const float4 c, const float4 q,
                                         const float2 w, const float2 e2) {
  const float2 dx = __fadd2_rn(dup(c.x), a.px), dy = __fadd2_rn(dup(c.y), a.py),
               dz = __fadd2_rn(dup(c.z), a.pz);
  const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
  const float2 inv = kSoft ? f2(rsqrt_normal(r2.x), rsqrt_normal(r2.y))
                           : f2(rsqrtf(r2.x), rsqrtf(r2.y));
  const float2 m = dup(c.w), qxy = dup(q.w), qxz = dup(w.x), qyz = dup(w.y);
  const float2 inv2 = __fmul2_rn(inv, inv), inv3 = __fmul2_rn(inv, inv2);
  const float2 qx = __ffma2_rn(dup(q.x), dx, __ffma2_rn(qxy, dy, __fmul2_rn(qxz, dz)));
  const float2 qy = __ffma2_rn(qxy, dx, __ffma2_rn(dup(q.y), dy, __fmul2_rn(qyz, dz)));
  const float2 qz = __ffma2_rn(qxz, dx, __ffma2_rn(qyz, dy, __fmul2_rn(dup(q.z), dz)));
  const float2 rqr = __ffma2_rn(dx, qx, __ffma2_rn(dy, qy, __fmul2_rn(dz, qz)));
  const float2 inv5 = __fmul2_rn(inv3, inv2), rqr5 = __fmul2_rn(rqr, inv5);
  const float2 along = __ffma2_rn(__fmul2_rn(dup(2.5f), rqr5), inv2, __fmul2_rn(m, inv3));
  const float2 n5 = f2(-inv5.x, -inv5.y);
  a.ax = __ffma2_rn(along, dx, __ffma2_rn(qx, n5, a.ax));
  a.ay = __ffma2_rn(along, dy, __ffma2_rn(qy, n5, a.ay));
  a.az = __ffma2_rn(along, dz, __ffma2_rn(qz, n5, a.az));
  a.pot = __ffma2_rn(dup(0.5f), rqr5, __ffma2_rn(m, inv, a.pot));
}

// kSoft: eps2 at least kSoftEps2. Every target appears exactly once in
// its own group's body list (each body is covered once and no accepted cell
// holds a target), and with softening its self term adds exactly zero
// acceleration (d = 0) and a known -G m_i / eps to the potential, so the
// loop needs no self test and the self potential is taken back out at the
// end; nor do the zeros past a list's end need one. Otherwise the self term
// is singular, or powers of 1/eps overflow: each entry is tested as in the
// reference, and only real entries are worked (kU = 1).
// kTeam: the groups whose passes the block's warps share (else a warp per group).
// kU: staged entries a lane works per inner-loop iteration (1 or 2, a
// context option searched by gtc_autotune_eval): their arithmetic is
// independent up to the accumulation, which stays in list order, so results
// do not depend on it.
// Staged entries, per warp and round parity: slice area a of the pass holds W
// entries from float4 a (kF4 W + 1) on (3 float4 per quadrupole cell, else 1); W
// is even and the 16-byte gap puts the areas on different banks. Per warp
// (kAllGroups: per slice) and target: the running sum (a, potential). (Arrays of
// their own: one struct of them all ran 1.5% slower.)
template <typename Stage, typename Sj, typename Sums>
struct EvalShared {
  Stage &stage;
  Sj &sj;  // staged body indices (self test)
  Sums &sums;
};

// Group g: by the warp (kNoGroups) or by the block's warps.
template <bool kQuad, bool kSoft, int kTeam, int kU, typename Shared>
__device__ __forceinline__ void eval_group(const Shared &sm, const float4 *__restrict__ bodies,
                                           const float4 *__restrict__ cells,
                                           const u32 *__restrict__ cell_list,
                                           const u32 *__restrict__ body_list,
                                           const uint4 *__restrict__ groups, u32 g, float G,
                                           float eps2, const float2 e2, const EvalOut &eo,
                                           u32 pass_cost) {
  constexpr u32 kF4 = kQuad ? 3 : 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint4 q0 = groups[4ull * g], q1 = groups[4ull * g + 1], q2 = groups[4ull * g + 2],
              q3 = groups[4ull * g + 3];
  const SegView cs = cell_segs(q1, q2), bs = body_segs(q2, q3);  // list entry -> index
  const u32 T = q0.y - q0.x, P = (T + 1) / 2;
  const u32 ec = q0.z, eb = q0.w;
  u32 S = 0;
  float4 *sum = sm.sums[kTeam == kNoGroups ? warp : 0];
  if (T > 0) {
    S = choose_slices(T, ec, eb, lane, pass_cost);
    const u32 slots = S * P;
    const u32 passes = (slots + 31u) / 32u;
    const float per_P = 1.f / static_cast<float>(P);
    const Cut cut_c(ec, S), cut_b(eb, S);
    if (kTeam != kAllGroups) {
      if (kTeam == kNoGroups || warp == 0) sum[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
      __syncwarp();
    }
    // (kLongGroups: every warp of a team takes each turn's barriers)
    const u32 ahead = kTeam == kLongGroups ? warp : 0u;
    for (u32 p = kTeam != kNoGroups ? warp : 0u; p - ahead < passes;
         p += kTeam != kNoGroups ? kWarpsPerBlock : 1u) {
      const bool works = kTeam != kLongGroups || p < passes;
      const u32 v = 32u * p + static_cast<u32>(lane);
      const bool computes = works && v < slots;
      const u32 slice = small_div(v, per_P), t0 = 2u * (v - slice * P),
                t1 = min(t0 + 1u, T - 1u);
      // the slices of the pass, and each one's share of the staging area
      const u32 s_lo = __shfl_sync(kFullMask, slice, 0);
      const u32 nsp = min(S - 1u, __shfl_sync(kFullMask, slice, 31)) - s_lo + 1u;
      const u32 W = small_div(kStage, 1.f / static_cast<float>(nsp)) & ~1u;  // 2..64
      const float per_W = 1.f / static_cast<float>(W);
      const u32 area = slice - s_lo;
      const float4 b0 = bodies[q0.x + (computes ? t0 : 0u)],
                   b1 = bodies[q0.x + (computes ? t1 : 0u)];
      Targets tg{f2(-b0.x, -b1.x), f2(-b0.y, -b1.y), f2(-b0.z, -b1.z),
                 dup(0.f), dup(0.f), dup(0.f), dup(0.f)};
      // The lane's two staging places (slice area and position in it) and
      // the list entries that go there round by round: cells, then bodies.
      u32 to_c[kPer], to_b[kPer], next[2][kPer], last[2][kPer];
#pragma unroll
      for (int h = 0; h < kPer; ++h) {
        const u32 e = static_cast<u32>(lane) + 32u * h, a = small_div(e, per_W), pos = e - a * W;
        to_c[h] = a < nsp ? a * (kF4 * W + 1u) + kF4 * pos : kNone;
        to_b[h] = a * (W + 1u) + pos;
#pragma unroll
        for (int l = 0; l < 2; ++l) {
          const Cut &cut = l ? cut_b : cut_c;
          next[l][h] = cut.at(s_lo + a) + pos;
          last[l][h] = a < nsp ? cut.at(s_lo + a + 1u) : 0u;
        }
      }
      const u32 cell_rounds = works ? (cut_c.longest() + W - 1u) / W : 0u;
      const u32 rounds = works ? cell_rounds + (cut_b.longest() + W - 1u) / W : 0u;
      // the list indices of round r, kNone past the slice's end
      u32 idx[kPer];
      auto load_indices = [&](u32 r) {
#pragma unroll
        for (int h = 0; h < kPer; ++h) {
          idx[h] = kNone;
          if (r < cell_rounds) {
            if (next[0][h] < last[0][h]) idx[h] = cell_list[cs.at(next[0][h])];
            next[0][h] += W;
          } else if (r < rounds) {
            if (next[1][h] < last[1][h]) idx[h] = body_list[bs.at(next[1][h])];
            next[1][h] += W;
          }
        }
      };
      // starts the copies of the entries idx names into round r's buffer
      auto stage_round = [&](u32 r) {
        if (r < rounds) {
          float4 *buf = sm.stage[warp][r & 1u];
#pragma unroll
          for (int h = 0; h < kPer; ++h) {
            if (to_c[h] == kNone) continue;
            if (r < cell_rounds) {
              copy_cell<kQuad>(buf + to_c[h], cells, idx[h]);
            } else {
              copy_async16(buf + to_b[h], bodies + (idx[h] == kNone ? 0u : idx[h]),
                           idx[h] != kNone);
              if (!kSoft) sm.sj[warp][r & 1u][to_b[h]] = idx[h];
            }
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      load_indices(0);
      stage_round(0);
      load_indices(1);
      u32 left_c = cut_c.base + (slice < cut_c.rest ? 1u : 0u),
          left_b = cut_b.base + (slice < cut_b.rest ? 1u : 0u);
      if (!computes) left_c = left_b = 0u;
      for (u32 r = 0; r < rounds; ++r) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();  // every lane's copies of round r; round r - 1 read
        stage_round(r + 1u);
        load_indices(r + 2u);
        const float4 *buf = sm.stage[warp][r & 1u];
        if (r < cell_rounds) {
          const u32 cnt = min(W, left_c);
          left_c -= cnt;
          const float4 *mine = buf + area * (kF4 * W + 1u);
          for (u32 j = 0; j < cnt; j += kU) {
#pragma unroll
            for (int u = 0; u < kU; ++u) {
              const float4 c = mine[kF4 * u];
              if (kQuad) {
                const float4 q = mine[kF4 * u + 1];
                const float2 w = *reinterpret_cast<const float2 *>(&mine[kF4 * u + 2]);
                add_cell<kSoft>(tg, c, q, w, e2);
              } else {
                add_body<kSoft>(tg, c, e2);
              }
            }
            mine += kF4 * kU;
          }
        } else {
          const u32 cnt = min(W, left_b);
          left_b -= cnt;
          const float4 *mine = buf + area * (W + 1u);
          for (u32 j = 0; j < cnt; j += kU) {
#pragma unroll
            for (int u = 0; u < kU; ++u) {
              const float4 b = mine[u];
              u32 self = kNone;  // the entry's target, if it is one
              if (!kSoft) self = sm.sj[warp][r & 1u][kSoft ? 0u : area * (W + 1u) + j + u] - q0.x;
              add_body<kSoft>(tg, b, e2, !kSoft && self == t0, !kSoft && self == t1);
            }
            mine += kU;
          }
        }
      }
      __syncwarp();  // the last round is read before the next pass stages
      // this pass's partial sums onto the targets', slice by slice
      const float4 r0 = make_float4(tg.ax.x, tg.ay.x, tg.az.x, tg.pot.x),
                   r1 = make_float4(tg.ax.y, tg.ay.y, tg.az.y, tg.pot.y);
      if (kTeam == kAllGroups) {
        if (computes) {
          sm.sums[slice][t0] = r0;
          if (t1 != t0) sm.sums[slice][t1] = r1;
        }
      }
      const int turns = kTeam == kAllGroups ? 0 : kTeam == kLongGroups ? kWarpsPerBlock : 1;
      for (int turn = 0; turn < turns; ++turn) {
        if (kTeam == kLongGroups) {  // the team's warps in pass order
          __syncthreads();
          if (turn != warp || !works) continue;
        }
        for (u32 a = 0; a < nsp; ++a) {
          if (computes && area == a) {
            float4 &u = sum[t0];
            u = make_float4(u.x + r0.x, u.y + r0.y, u.z + r0.z, u.w + r0.w);
            if (t1 != t0) {
              float4 &w = sum[t1];
              w = make_float4(w.x + r1.x, w.y + r1.y, w.z + r1.z, w.w + r1.w);
            }
          }
          __syncwarp();
        }
      }
    }
  }
  if (kTeam != kNoGroups) __syncthreads();
  if (static_cast<u32>(lane) < T && (kTeam == kNoGroups || warp == 0)) {
    const u32 i = q0.x + static_cast<u32>(lane);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kTeam == kAllGroups) {
      for (u32 s = 0; s < S; ++s) {
        const float4 u = sm.sums[s][lane];
        acc = make_float4(acc.x + u.x, acc.y + u.y, acc.z + u.z, acc.w + u.w);
      }
    } else {
      acc = sum[lane];
    }
    // the self term (softened), taken back once
    if (kSoft) acc.w -= __fmul_rn(bodies[i].w, rsqrtf(eps2));
    write_target(eo, i, make_float4(G * acc.x, G * acc.y, G * acc.z, -G * acc.w));
  }
  if (kTeam != kNoGroups) __syncthreads();  // the sums are read before the next group's
}

template <bool kQuad, bool kSoft, int kTeam, int kU>
__global__ void __launch_bounds__(kT, kBlocksPerSm)
    k_eval(const float4 *__restrict__ bodies, const float4 *__restrict__ cells,
           const u32 *__restrict__ cell_list, const u32 *__restrict__ body_list,
           const uint4 *__restrict__ groups, u32 ngroups, float G, float eps2, EvalOut eo,
           u32 *next_group, const u32 *ng_dev, const u32 *abort, u32 pass_cost,
           const unsigned long long *interactions) {
  grid_wait();
  __shared__ float4 stage[kWarpsPerBlock][2][kStage * (kQuad ? 3 : 1) + 32];
  __shared__ u32 sj[kWarpsPerBlock][2][kSoft ? 1 : kStage + 32];
  __shared__ float4 sums[kTeam == kAllGroups ? kMaxSlices : kWarpsPerBlock][32];
  __shared__ u32 team_group;
  const EvalShared<decltype(stage), decltype(sj), decltype(sums)> sm{stage, sj, sums};
  const int lane = threadIdx.x & 31;
  if (abort && *abort) return;
  if (ng_dev) ngroups = min(ngroups, *ng_dev);
  const float2 e2 = dup(eps2);
  if (kTeam == kAllGroups) {
    for (;;) {
      if (threadIdx.x == 0) team_group = atomicAdd(next_group, 1u);
      __syncthreads();
      const u32 g = team_group;
      if (g >= ngroups) return;
      eval_group<kQuad, kSoft, kAllGroups, kU>(
          sm, bodies, cells, cell_list, body_list, groups, g, G, eps2, e2, eo, pass_cost);
    }
  }
  // A group's work: targets x (entries, a cell counted as so much of a body). Long:
  // more than three quarters of a warp's share of it all.
  constexpr u64 kCellCost = kQuad ? 5 : 2, kBodyCost = 2;
  u64 long_work = ~0ull;
  auto is_long = [&](const uint4 &q) {
    return static_cast<u64>(q.y - q.x) * (kCellCost * q.z + kBodyCost * q.w) > long_work;
  };
  if (kTeam == kLongGroups) {
    long_work = (kCellCost * interactions[0] + kBodyCost * interactions[1]) * 3ull /
                (4ull * gridDim.x * kWarpsPerBlock);
    // the long ones among the block's share, every gridDim.x-th group
    for (u64 share = blockIdx.x; share < ngroups;) {
      const u64 mine = share + static_cast<u64>(threadIdx.x) * gridDim.x;
      if (threadIdx.x == 0) team_group = kNone;
      __syncthreads();
      if (mine < ngroups && is_long(groups[4ull * mine]))
        atomicMin(&team_group, static_cast<u32>(mine));
      __syncthreads();
      const u32 g = team_group;
      __syncthreads();
      if (g == kNone) {
        share += static_cast<u64>(kT) * gridDim.x;
        continue;
      }
      eval_group<kQuad, kSoft, kLongGroups, kU>(
          sm, bodies, cells, cell_list, body_list, groups, g, G, eps2, e2, eo, pass_cost);
      share = static_cast<u64>(g) + gridDim.x;
    }
  }
  for (;;) {
    u32 g = 0;
    if (lane == 0) g = atomicAdd(next_group, 1u);
    g = __shfl_sync(kFullMask, g, 0);
    if (g >= ngroups) return;
    if (kTeam == kLongGroups && is_long(groups[4ull * g])) continue;
    eval_group<kQuad, kSoft, kNoGroups, kU>(sm, bodies, cells, cell_list, body_list, groups, g, G,
                                            eps2, e2, eo, pass_cost);
  }
}

// What evaluate_lists' launches share.
struct EvalArgs {
  const float4 *bodies, *cells;
  const u32 *cell_list, *body_list;
  const uint4 *groups;
  u64 n_groups;  // groups at most
  float G, eps2;
  EvalOut eo;
  u32 *counter;
  EvalShape shape;
  const Scalars *sc;  // a graph replay: the group count and the abort word
  const unsigned long long *interactions;  // the lists' totals: cells, bodies
};

template <bool kQuad, bool kSoft, int kTeam, int kU>
void launch_shape(const EvalArgs &a, int sms, cudaStream_t s) {
  int per_sm = 0;
  GTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &per_sm, k_eval<kQuad, kSoft, kTeam, kU>, kT, 0));
  const u64 want = kTeam == kAllGroups ? a.n_groups : (a.n_groups + kWarpsPerBlock - 1) / kWarpsPerBlock;
  const u32 grid =
      static_cast<u32>(std::min<u64>(want, static_cast<u64>(sms) * std::max(1, per_sm)));
  launch(k_eval<kQuad, kSoft, kTeam, kU>, grid, kT, 0, s, a.bodies, a.cells, a.cell_list,
         a.body_list, a.groups, static_cast<u32>(a.n_groups), a.G, a.eps2, a.eo, a.counter,
         a.sc ? &a.sc->n_groups : nullptr, a.sc ? &a.sc->abort : nullptr, a.shape.pass_cost,
         a.interactions);
  GTC_LAUNCH_CHECK();
}

// Groups below which a block's warps share every group, and below which they
// share the long ones (above).
constexpr u64 kTeamGroups = 6000, kWarpGroups = 12000;

template <bool kQuad, bool kSoft>
void launch_eval(const EvalArgs &a, u64 groups_hint, cudaStream_t s) {
  constexpr int kTwo = kSoft ? 2 : 1;  // (an unsoftened slice is worked without padding)
  int dev = 0, sms = 0;
  GTC_CUDA(cudaGetDevice(&dev));
  GTC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const bool one = a.shape.pairs == 1;
  if (groups_hint < kTeamGroups) {
    if (one) launch_shape<kQuad, kSoft, kAllGroups, 1>(a, sms, s);
    else launch_shape<kQuad, kSoft, kAllGroups, kTwo>(a, sms, s);
  } else if (groups_hint < kWarpGroups && a.interactions) {
    if (one) launch_shape<kQuad, kSoft, kLongGroups, 1>(a, sms, s);
    else launch_shape<kQuad, kSoft, kLongGroups, kTwo>(a, sms, s);
  } else {
    if (one) launch_shape<kQuad, kSoft, kNoGroups, 1>(a, sms, s);
    else launch_shape<kQuad, kSoft, kNoGroups, kTwo>(a, sms, s);
  }
}

void launch_any(const EvalArgs &a, bool quadrupole, u64 groups_hint, cudaStream_t s) {
  if (a.n_groups == 0) return;
  const bool soft = a.eps2 >= kSoftEps2;
  if (quadrupole && soft) launch_eval<true, true>(a, groups_hint, s);
  else if (quadrupole) launch_eval<true, false>(a, groups_hint, s);
  else if (soft) launch_eval<false, true>(a, groups_hint, s);
  else launch_eval<false, false>(a, groups_hint, s);
}

}  // namespace

void evaluate_lists(const float4 *bodies, const float4 *cells, const u32 *cell_list,
                    const u32 *body_list, const uint4 *groups, u64 n_groups, float G, float eps2,
                    bool quadrupole, const EvalOut &eo, u32 *counter, cudaStream_t s,
                    const EvalShape &shape, const unsigned long long *interactions) {
  launch_any(EvalArgs{bodies, cells, cell_list, body_list, groups, n_groups, G, eps2, eo, counter,
                      shape, nullptr, interactions},
             quadrupole, n_groups, s);
}

void evaluate_lists_graph(const float4 *bodies, const float4 *cells, const u32 *cell_list,
                          const u32 *body_list, const uint4 *groups, u64 max_groups,
                          u64 groups_hint, const Scalars *sc, float G, float eps2,
                          bool quadrupole, const EvalOut &eo, u32 *counter, cudaStream_t s,
                          const EvalShape &shape) {
  launch_any(EvalArgs{bodies, cells, cell_list, body_list, groups, max_groups, G, eps2, eo,
                      counter, shape, sc, &sc->cell_interactions},
             quadrupole, groups_hint, s);
}

}  // namespace gtc
