// The per-particle tree walk: Octree::accel_pot (src/octree.cpp:275-344) for
// every body, the reference's `gravity = tree` solver (compute_gravity_tree,
// src/gravity.cpp:7-26), on the device tree.
//
// FP64 with every product and sum rounded on its own (compiled -fmad=false)
// and the reference's operand order, on nodes identical to the reference's:
// the walk visits nodes in the reference's stack order (the device numbers
// nodes that way, so the stack becomes a forward scan with skip links), the
// opening test is the Barnes (1994) offset criterion -- a cell is accepted
// when the body lies outside its slackened cube and r^2 > (2 h / theta +
// delta)^2 -- and accepted cells add monopole and quadrupole terms; opened
// leaves add their bodies, skipping the body itself. CUDA's FP64 division
// and square root round correctly, as the host's do, so the forces are the
// reference's bit for bit.
//
// One lane per body in tree order (neighbours walk alike), results to the
// caller's order. Bound: the FP64 pipe, which issues a warp's instruction
// in the same time whether one lane or all take part. So a warp works in two
// turns. Walk: every lane follows its own walk, deciding each opening test
// in FP32 with an error band (walk_test.cuh; the body is a box of no extent)
// and in FP64 only within the band, and lists what it met -- accepted cells
// and leaf bodies, in visit order -- in shared memory, until each lane holds
// kList entries or is done. Evaluate: the lanes work through their lists
// entry by entry together, so that the FP64 instructions run with full
// warps. Each body still adds the same terms in the same order. With one
// FP64 test and one FP64 interaction per visit and lane, a warp issued the
// interaction for every visit any lane accepted: 200k bodies of the benchmark
// galaxy took 63 ms; in turns 32 ms (87 FP64 instructions per 32
// interactions, the pipe 84% busy). Their products, the root and the quotient
// then went to the integer pipes (wide.cuh), rounded alike, which leaves the
// 25 sums: 11.7 ms, the FP64 pipe near 70% busy, the integer and multiply
// pipes near 60%. Ten blocks an SM (96 registers, none spilled) 11.7 ms,
// unbounded (114) 12.4; blocks of 128 and lists of 16 to 48 measure the same.

#include "pipeline.cuh"
#include "walk_test.cuh"
#include "wide.cuh"

namespace gtc {
namespace {

constexpr int kT = 64;
constexpr int kBlocks = 10;        // per SM: 96 registers, none spilled
constexpr u32 kList = 32;          // entries a lane lists before they are evaluated
constexpr u32 kBodyBit = 1u << 31; // entry: a body's tree position, else a node index

struct TreeWalkArgs {
  const WalkRec32 *walk32;
  const double2 *geom;  // (cx, cy), (cz, half)
  const double2 *mom;   // (mx, my), (mz, mass)
  const double2 *quad;  // xx yy | zz xy | xz yz
  const double *delta;
  const double *tpos, *tmass;  // tree order
  const u32 *order;            // tree position -> caller index
  const TreeRoot *root;
  u32 n, m;
  double G, eps2, inv_theta;
  double *acc, *pot;           // caller order
  unsigned long long *counts;  // cell, particle interactions
  Scalars *sc;
};

// The opening test of octree.cpp:275-344 in FP64, as the reference has it.
__device__ __noinline__ bool accepts64(const TreeWalkArgs &a, u32 i, double x, double y,
                                       double z) {
  const double2 g0 = a.geom[2ull * i], g1 = a.geom[2ull * i + 1];
  const double2 c0 = a.mom[2ull * i], c1 = a.mom[2ull * i + 1];
  const double half = g1.y;
  const double dx = x - c0.x, dy = y - c0.y, dz = z - c1.x;
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double crit = 2.0 * half * a.inv_theta + a.delta[i];
  const double slack = half * 1.0001;
  const bool inside = fabs(x - g0.x) <= slack && fabs(y - g0.y) <= slack &&
                      fabs(z - g1.x) <= slack;
  return !inside && r2 > crit * crit;
}

// The bounds on lengths' components, and on masses and moments, within which
// every product of an interaction is a normal number.
constexpr int kStepExp = -110, kMassExp = -300;
constexpr u32 kSteps = kWord<90> - kWord<kStepExp>, kMasses = kWord<450> - kWord<kMassExp>;

// What one entry adds to its body: fx .. fp are taken from the sums, then ux ..
// uz added and up taken (quadrupole; cells only).
struct Terms {
  double fx, fy, fz, fp, ux, uy, uz, up;
};

// As the reference writes them, in FP64. CUDA's division and square root round
// correctly, as the host's do.
template <bool kQuad>
__device__ __noinline__ void terms64(const TreeWalkArgs &a, bool body, u32 j, double dx, double dy,
                                     double dz, double r2s, double mass, Terms &t) {
  const double gm = a.G * mass;
  const double inv = 1.0 / sqrt(r2s);
  const double inv3 = inv * inv * inv;
  // the reference's operand order differs: G m inv inv inv for a body,
  // G m (inv inv inv) for a cell
  const double gm3 = body ? gm * inv * inv * inv : gm * inv3;
  t.fx = gm3 * dx;
  t.fy = gm3 * dy;
  t.fz = gm3 * dz;
  t.fp = gm * inv;
  if (kQuad && !body) {
    const double2 qa = a.quad[3ull * j], qb = a.quad[3ull * j + 1], qc = a.quad[3ull * j + 2];
    const double qx = qa.x * dx + qb.y * dy + qc.x * dz;
    const double qy = qb.y * dx + qa.y * dy + qc.y * dz;
    const double qz = qc.x * dx + qc.y * dy + qb.x * dz;
    const double rqr = dx * qx + dy * qy + dz * qz;
    const double inv5 = inv3 * inv * inv;
    const double inv7 = inv5 * inv * inv;
    t.ux = a.G * (qx * inv5 - 2.5 * rqr * dx * inv7);
    t.uy = a.G * (qy * inv5 - 2.5 * rqr * dy * inv7);
    t.uz = a.G * (qz * inv5 - 2.5 * rqr * dz * inv7);
    t.up = 0.5 * a.G * rqr * inv5;
  }
}

// kUnitG: G is 1, and a factor of it changes nothing.
template <bool kQuad, bool kUnitG>
__global__ void __launch_bounds__(kT, kBlocks) k_tree_walk(TreeWalkArgs a) {
  grid_wait();
  __shared__ u32 lists[kT / 32][kList][32];
  const int lane = threadIdx.x & 31;
  u32 (*list)[32] = lists[threadIdx.x >> 5];
  const u32 t = blockIdx.x * kT + threadIdx.x;
  const bool valid = t < a.n;
  u32 ncell = 0, npart = 0;
  double x = 0, y = 0, z = 0;
  if (valid) {
    x = a.tpos[3ull * t];
    y = a.tpos[3ull * t + 1];
    z = a.tpos[3ull * t + 2];
  }
  const float gf[3] = {static_cast<float>(x - a.root->center[0]),
                       static_cast<float>(y - a.root->center[1]),
                       static_cast<float>(z - a.root->center[2])};
  const float hf[3] = {0.f, 0.f, 0.f};
  const float gbound = fmaxf(fmaxf(fabsf(gf[0]), fabsf(gf[1])), fabsf(gf[2])) *
                       (1.0f + 1.0f / (1 << 20));
  double ax = 0, ay = 0, az = 0, phi = 0;
  u32 i = valid ? 0u : a.m;
  u32 k = 0, kend = 0;  // the rest of an opened leaf
  for (;;) {
    u32 cnt = 0;
    while (cnt < kList && (k < kend || i < a.m)) {
      if (k < kend) {
        if (k != t) {
          list[cnt++][lane] = k | kBodyBit;
          ++npart;
        }
        ++k;
        continue;
      }
      const WalkRec32 r = load32(a.walk32, i);
      int verdict = accept32(r, gf, hf, gbound);
      if (verdict == 2) verdict = accepts64(a, i, x, y, z) ? 1 : 0;
      const bool leaf = (r.nbody_leaf >> 31) != 0;
      if (verdict == 1) {
        list[cnt++][lane] = i;
        ++ncell;
      } else if (leaf) {
        k = r.begin;
        kend = r.begin + (r.nbody_leaf & 0x7fffffffu);
      }
      if (verdict == 1 || leaf) {
        if (r.skip <= i) {  // malformed tree: never loop
          atomicOr(&a.sc->error, 1u);
          i = a.m;
        } else {
          i = r.skip;
        }
      } else {
        ++i;  // the children follow, in the reference's stack order
      }
    }
    __syncwarp();
    const u32 most = __reduce_max_sync(kFullMask, cnt);
    if (most == 0) break;
    for (u32 e = 0; e < most; ++e) {
      if (e >= cnt) continue;
      const u32 q = list[e][lane];
      const bool body = (q & kBodyBit) != 0;
      const u32 j = q & ~kBodyBit;
      double dx, dy, dz, mass;
      if (body) {
        dx = a.tpos[3ull * j];
        dy = a.tpos[3ull * j + 1];
        dz = a.tpos[3ull * j + 2];
        mass = a.tmass[j];
      } else {
        const double2 c0 = a.mom[2ull * j], c1 = a.mom[2ull * j + 1];
        dx = c0.x;
        dy = c0.y;
        dz = c1.x;
        mass = c1.y;
      }
      dx = x - dx;
      dy = y - dy;
      dz = z - dz;
      // The same operations, bit for bit, with the products, the root and the
      // quotient on the integer pipes. Lengths within 2^+-80 (steps from 2^-110),
      // masses and moments from 2^-300 to 2^450, and zeros, keep every product
      // normal; others are worked in FP64.
      const Factor mx = factor(dx), my = factor(dy), mz = factor(dz);
      const double r2s = product(mx, mx) + product(my, my) + product(mz, mz) + a.eps2;
      const double gm = kUnitG ? mass : a.G * mass;
      const u32 step = above<kStepExp>(dx, above<kStepExp>(dy, above<kStepExp>(dz, 0u)));
      const u32 r2w = static_cast<u32>(__double2hiint(r2s)) - kWord<-160> / 2;
      u32 far = above<kMassExp>(gm, 0u);
      Terms w;
      if (step >= kSteps || r2w >= kWord<160> / 2 - kWord<-160> / 2 || far >= kMasses) {
        terms64<kQuad>(a, body, j, dx, dy, dz, dx * dx + dy * dy + dz * dz + a.eps2, mass, w);
        ax -= w.fx;
        ay -= w.fy;
        az -= w.fz;
        phi -= w.fp;
        if (kQuad && !body) {
          ax += w.ux;
          ay += w.uy;
          az += w.uz;
          phi -= w.up;
        }
        continue;
      }
      const Factor inv = factor<true>(recip_sqrt(r2s));
      const Factor inv2 = factor<true>(product<true>(inv, inv));
      const Factor inv3 = factor<true>(product<true>(inv2, inv));
      const Factor m = factor(gm);
      const double gm1 = product(m, inv);
      Factor head = m, tail = inv3;
      if (body) {
        head = factor(product(factor(gm1), inv));
        tail = inv;
      }
      const Factor gm3 = factor(product(head, tail));
      ax -= product(gm3, mx);
      ay -= product(gm3, my);
      az -= product(gm3, mz);
      phi -= gm1;
      if (kQuad && !body) {
        const double2 qa = a.quad[3ull * j], qb = a.quad[3ull * j + 1], qc = a.quad[3ull * j + 2];
        const Factor xx = factor(qa.x), yy = factor(qa.y), zz = factor(qb.x), xy = factor(qb.y),
                     xz = factor(qc.x), yz = factor(qc.y);
        const double qx = product(xx, mx) + product(xy, my) + product(xz, mz);
        const double qy = product(xy, mx) + product(yy, my) + product(yz, mz);
        const double qz = product(xz, mx) + product(yz, my) + product(zz, mz);
        const Factor vx = factor(qx), vy = factor(qy), vz = factor(qz);
        const double rqr = product(mx, vx) + product(my, vy) + product(mz, vz);
        far = above<kMassExp>(qa.x, above<kMassExp>(qa.y, above<kMassExp>(qb.x, far)));
        far = above<kMassExp>(qb.y, above<kMassExp>(qc.x, above<kMassExp>(qc.y, far)));
        const double u = kUnitG ? rqr : a.G * rqr;
        far = above<kMassExp>(qx, above<kMassExp>(qy, above<kMassExp>(qz, far)));
        far = above<kMassExp>(rqr, above<kMassExp>(u, far));
        if (far < kMasses) {
          const Factor inv5 = factor<true>(product<true>(
              factor<true>(product<true>(inv3, inv)), inv));
          const Factor inv7 = factor<true>(product<true>(
              factor<true>(product<true>(inv5, inv)), inv));
          Factor half5 = inv5;  // exact: 0.5 G rqr inv5 = (G rqr) (inv5 / 2)
          half5.se -= 0x100000u;
          const Factor v = factor(product(factor(rqr), factor<true>(2.5)));
          w.ux = product(vx, inv5) - product(factor(product(v, mx)), inv7);
          w.uy = product(vy, inv5) - product(factor(product(v, my)), inv7);
          w.uz = product(vz, inv5) - product(factor(product(v, mz)), inv7);
          if (!kUnitG) {
            w.ux = a.G * w.ux;
            w.uy = a.G * w.uy;
            w.uz = a.G * w.uz;
          }
          w.up = product(factor(u), half5);
        } else {
          terms64<kQuad>(a, body, j, dx, dy, dz, r2s, mass, w);
        }
        ax += w.ux;
        ay += w.uy;
        az += w.uz;
        phi -= w.up;
      }
    }
    __syncwarp();
  }
  if (valid) {
    const u32 self = a.order[t];
    a.acc[3ull * self] = ax;
    a.acc[3ull * self + 1] = ay;
    a.acc[3ull * self + 2] = az;
    a.pot[self] = phi;
  }
  // interaction counters: one atomic per warp
  ncell = __reduce_add_sync(kFullMask, ncell);
  npart = __reduce_add_sync(kFullMask, npart);
  if (lane == 0) {
    atomicAdd(&a.counts[0], static_cast<unsigned long long>(ncell));
    atomicAdd(&a.counts[1], static_cast<unsigned long long>(npart));
  }
}

}  // namespace

void tree_walk_forces(Workspace &ws, const SolverParams &sp, double *acc, double *pot,
                      unsigned long long *counts, cudaStream_t s) {
  if (ws.n == 0) return;
  const TreeWalkArgs a{ws.walk32.as<WalkRec32>(), ws.geom.as<double2>(), ws.mom.as<double2>(),
                       ws.quad.as<double2>(), ws.delta.as<double>(), ws.tpos.as<double>(),
                       ws.tmass.as<double>(), ws.idx.as<u32>(), ws.root.as<TreeRoot>(),
                       static_cast<u32>(ws.n), static_cast<u32>(ws.n_nodes), sp.G,
                       sp.eps * sp.eps, 1.0 / sp.theta, acc, pot, counts,
                       ws.scalars.as<Scalars>()};
  const bool unit = sp.G == 1.0;
  const auto kernel = sp.quadrupole ? (unit ? k_tree_walk<true, true> : k_tree_walk<true, false>)
                                    : (unit ? k_tree_walk<false, true> : k_tree_walk<false, false>);
  launch(kernel, ceil_div(ws.n, kT), kT, 0, s, a);
  GTC_LAUNCH_CHECK();
}

}  // namespace gtc
