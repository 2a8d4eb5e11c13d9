// gx_walk.cu -- warp-cooperative Barnes-Hut tree walk.
//
// Reference: solvers/src/lbvh.rs:469-524 (LbvhFlat::accel: skip the subtree of a
// massless node; a leaf adds the Plummer-softened pair term unless it is the target
// itself; an internal node is accepted as a monopole iff the target is not inside
// its AABB and theta*(d - delta) >= s, s = 2*max(half extents); otherwise it is
// opened) and :673-675 (result times G).
//
// FP32 walk (k_walk_f32): one warp walks the tree for 8, 16 or 32 Morton-consecutive targets
// of one system. It pops up to 32 nodes at a time from a stack in shared memory, one a lane,
// decides each node's two children for all its targets against the targets' box, and lists
// what they take; the lists are evaluated a batch at a time. Decisions that the box leaves
// open are made for every target. Node centres of mass and leaf positions are float-float
// (hi + lo), ~48 bits of the f64 coordinates; the opening test compares d^2 with
// rcrit^2 = (s/theta + delta)^2 and re-decides in FP64 with the reference's exact expression
// whenever the FP32 value lies within a relative 4e-6 band of the threshold (or touches the
// AABB within 2^-20), so every opening decision equals the reference's. Terms are
// accumulated in FP32 with Kahan compensation; the sums leave FP32 compensated.
// FP64 walk (k_walk_f64): every lane walks the tree for its own target, without a stack (a
// record names the node that follows its subtree), with the reference's arithmetic,
// operation for operation and in its depth-first order, so accelerations are
// bit-identical to the reference's CPU walk.
// Bounds: the FP32 stack cannot pass kWalkStack, and the steps of either walk are limited by
// the system's nodes; a tree that breaks them raises the device error word.
#include "gx_kernels.h"

namespace gx {

namespace {

// The reference's decision for internal node gi (solvers/src/lbvh.rs:485-514) in f64
// on the node's f64 aggregate, geometry derived as in reference_flatten
// (lbvh.rs:602-613): 1 = take the monopole, 0 = open, -1 = skip (massless subtree).
__device__ __noinline__ int exact_decision(const Agg64* __restrict__ agg, uint32_t gi, const double x[3],
                                           double theta) {
  const Agg64& a = agg[gi];
  if (!(a.m > 0.0)) return -1;
  double ctr[3], hf[3], dv[3], dx[3];
  bool inside = true;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    ctr[c] = dmul(dadd(a.mn[c], a.mx[c]), 0.5);
    hf[c] = dmul(dsub(a.mx[c], a.mn[c]), 0.5);
    dv[c] = dsub(a.com[c], ctr[c]);
    inside = inside && (fabs(dsub(x[c], ctr[c])) <= hf[c]);
    dx[c] = dsub(a.com[c], x[c]);
  }
  const double delta = dsqrt(dlen2(dv[0], dv[1], dv[2]));
  const double d2 = dlen2(dx[0], dx[1], dx[2]);
  const double s = dmul(2.0, fmax(hf[0], fmax(hf[1], hf[2])));
  const double d = dsqrt(d2);
  return (!inside && dmul(theta, dsub(d, delta)) >= s) ? 1 : 0;
}

__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace

// The FP64 walk's records, made once a tree, one thread a sorted position: the internal node of that index
// and the leaf. The node after a subtree in depth-first order is the right child of the
// first ancestor that the subtree lies to the left of, two steps up on average. The
// thresholds bracket the reference's test theta (d - delta) >= s on d^2 by 1e-9 (its
// rounding is a few 1e-16), and from kInsideTheta on the upper one is also beyond the box's
// corners, so that what is taken is outside the box; in between, and with NaN thresholds
// (a zero-size box, a square out of range), the exact decision is made. At theta = 0 every
// box of some size is opened. (With the exact decision for every node taken from
// kInsideTheta on, or at theta = 0, which divergent lanes make one after another, the walk
// stage of 30,011 of a disk at theta 1.2 took 679 us against 279, 3,000 of a Plummer sphere at
// theta 0 4.0 ms against 2.0; one walk a warp 610 us and 3.4 ms.)
// `split` CTAs a tile: with one, a thread climbs for 16 positions one after another (30,011
// particles 49 us against 10).
__global__ void __launch_bounds__(kTileThreads) k_walk_records64(StepBufs b, int split) {
  const TileDesc t = tile_part(b.tiles, split);
  const SysDesc sd = b.sys[t.sys];
  const uint32_t n_total = b.n, int_lo = n_total + sd.off;
  auto next_of = [&](uint32_t u) {
    for (int level = 0; level <= kMaxDepth; ++level) {
      const uint32_t p = b.parent[u];
      if (p - int_lo >= sd.n - 1u) return kWalkEnd;  // the root
      const uint2 kd = b.kids[p - n_total];
      if (kd.x == u) return kd.y;
      u = p;
    }
    raise_err(b.ctl, kErrClimb);
    return kWalkEnd;
  };
  for (uint32_t k = t.begin + threadIdx.x; k < t.end; k += kTileThreads) {
    if (sd.n < 2) continue;
    b.leaf_next[k] = next_of(k);
    if (k == sd.off + sd.n - 1u) continue;  // one internal node fewer than leaves
    const Agg64& a = b.agg64[k];
    Rec64 r;
    double hf[3], dv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      r.com[c] = a.com[c];
      hf[c] = dmul(dsub(a.mx[c], a.mn[c]), 0.5);
      dv[c] = dsub(a.com[c], dmul(dadd(a.mn[c], a.mx[c]), 0.5));
    }
    r.m = a.m;
    const double s = dmul(2.0, fmax(hf[0], fmax(hf[1], hf[2])));
    const double delta = dsqrt(dlen2(dv[0], dv[1], dv[2]));
    const double rc = s / sd.theta + delta;
    // a target inside the box is at most its half diagonal and delta from the centre of mass
    const double far = sd.theta < kInsideTheta ? rc : fmax(rc, dsqrt(dlen2(hf[0], hf[1], hf[2])) + delta);
    const bool ok = sd.theta > 0.0 && s > 0.0 && rc * rc > 1e-280 && far * far < 1e280;
    const double none = sd.theta == 0.0 && s > 0.0 ? INFINITY : __longlong_as_double(0x7fffffffffffffffll);
    r.lo2 = ok ? rc * rc * (1.0 - 1e-9) : none;
    r.hi2 = ok ? far * far * (1.0 + 1e-9) : none;
    r.left = b.kids[k].x;
    r.next = next_of(n_total + k);
    r.pad[0] = r.pad[1] = 0u;
    b.rec64[k] = r;
  }
}

namespace {

// Nodes that the walks of a warp's targets visit, each counted once (the statistic
// warp_node_visits): the warp goes through the tree in depth-first order, and a lane waits
// until the warp is at the next node of its own walk.
__device__ __noinline__ uint32_t warp_visits(const StepBufs& b, const SysDesc& sd, const double x[3], bool valid) {
  const uint32_t n_total = b.n, int_lo = n_total + sd.off, max_steps = 2u * sd.n;
  uint32_t mine = valid ? int_lo : kWalkEnd, count = 0;
  uint32_t u = __any_sync(0xffffffffu, valid) ? int_lo : kWalkEnd;
  while (count < max_steps && (u - sd.off < sd.n || u - int_lo < sd.n - 1u)) {
    ++count;
    const bool leaf = u < n_total, at = mine == u;
    const uint32_t next = leaf ? b.leaf_next[u] : b.rec64[u - n_total].next;
    const uint32_t left = leaf ? kWalkEnd : b.rec64[u - n_total].left;
    const bool open = at && !leaf && exact_decision(b.agg64, u - n_total, x, sd.theta) == 0;
    if (at) mine = open ? left : next;
    u = __any_sync(0xffffffffu, open) ? left : next;
  }
  return count;
}

}  // namespace

// Exact FP64 walk: every lane walks the tree for its own target in strict depth-first,
// left-before-right order and adds its terms in that order with the reference's arithmetic.
// A record names its successor for either decision, so there is no stack, and the next
// record is loaded before the current one's term (a square root and a division) is
// evaluated. Bound by the latency of one record per step; the lanes' walks are
// independent. (One walk a warp, over the union of its 32 targets' nodes, with the exact
// test and a ballot per node: N = 30,011 Plummer, theta 0.5: 9.3 ms; this one 3.1 ms; 262,144 of a
// collision: 7.8 and 6.6 ms.)
template <bool STATS, bool LIST>
__global__ void __launch_bounds__(kWalkThreads) k_walk_f64(StepBufs b, int persistent) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps_total = (gridDim.x * blockDim.x) >> 5;
  uint32_t item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t n_total = b.n;
  while (item < b.nitems) {
    const WalkItem it = b.items[item];
    const SysDesc sd = b.sys[it.sys];
    const uint32_t end = sd.off + sd.n;
    // a target list (active-subset walk) names the item's targets; else they are the
    // 32 sorted positions from it.begin
    const uint32_t li = it.begin + lane;
    const bool valid = LIST ? (lane < static_cast<int>(b.group) && li < *b.ntargets) : li < end;
    const uint32_t k = LIST ? (valid ? b.targets[li] : 0u) : li;
    double a64[3] = {0.0, 0.0, 0.0};
    unsigned long long n_leaf = 0, n_far = 0, n_open = 0;
    if (sd.n > 1 && valid) {
      const double eps2 = dmul(sd.eps, sd.eps);
      const double4 x = b.leaf64[k];
      const double x3[3] = {x.x, x.y, x.z};
      const uint32_t max_steps = 2u * sd.n;
      const uint32_t int_lo = n_total + sd.off, int_n = sd.n - 1;
      double4 p;          // the current node: centre of mass (or leaf position) and mass
      double lo2, hi2;    // its thresholds (a leaf is always taken)
      uint32_t left, next;
      auto fetch = [&](uint32_t u) {
        const bool leaf = u < n_total;
        const double4* q = leaf ? &b.leaf64[u] : reinterpret_cast<const double4*>(&b.rec64[u - n_total]);
        p = *q;
        lo2 = hi2 = -1.0;
        left = next = kWalkEnd;
        if (leaf) {
          next = b.leaf_next[u];
        } else {
          const double2 th = *reinterpret_cast<const double2*>(q + 1);
          const uint2 ln = *reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(q + 1) + 16);
          lo2 = th.x;
          hi2 = th.y;
          left = ln.x;
          next = ln.y;
        }
      };
      uint32_t u = int_lo;
      fetch(u);
      for (uint32_t step = 0;; ++step) {
        if (step >= max_steps) {
          raise_err(b.ctl, kErrBadIndex);
          break;
        }
        const double dx = dsub(p.x, x3[0]), dy = dsub(p.y, x3[1]), dz = dsub(p.z, x3[2]);
        const double d2 = dlen2(dx, dy, dz);
        const double m = p.w;
        bool take = d2 > hi2, open = d2 < lo2;
        if (!(m > 0.0)) {
          take = open = false;
        } else if (!take && !open) {
          const int dec = u < n_total ? 1 : exact_decision(b.agg64, u - n_total, x3, sd.theta);
          take = dec == 1;
          open = dec == 0;
        }
        const bool self = u == k;
        if (STATS) {
          n_leaf += take && u < n_total && !self ? 1 : 0;
          n_far += take && u >= n_total ? 1 : 0;
          n_open += open ? 1 : 0;
        }
        u = open ? left : next;
        const bool more = u != kWalkEnd;
        if (more) {
          if (u - sd.off >= sd.n && u - int_lo >= int_n) {
            raise_err(b.ctl, kErrBadIndex);
            break;
          }
          fetch(u);
        }
        if (take && !self) {
          const double r2 = dadd(d2, eps2);
          const double f = ddiv(m, dmul(r2, dsqrt(r2)));
          a64[0] = dadd(a64[0], dmul(dx, f));
          a64[1] = dadd(a64[1], dmul(dy, f));
          a64[2] = dadd(a64[2], dmul(dz, f));
        }
        if (!more) break;
      }
    }
    __syncwarp();
    if (valid) {
      const uint32_t o = b.order[k];
#pragma unroll
      for (int c = 0; c < 3; ++c) b.acc[3 * (size_t)o + c] = sd.n > 1 ? dmul(a64[c], sd.g) : 0.0;
    }
    if (STATS) {
      const double4 xv = valid ? b.leaf64[k] : make_double4(0.0, 0.0, 0.0, 0.0);
      const double x3[3] = {xv.x, xv.y, xv.z};
      const uint32_t n_vis = sd.n > 1 ? warp_visits(b, sd, x3, valid) : 0u;
      n_leaf = warp_sum64(n_leaf);
      n_far = warp_sum64(n_far);
      n_open = warp_sum64(n_open);
      if (lane == 0) {
        atomicAdd(&b.ctl->stats[0], n_leaf);
        atomicAdd(&b.ctl->stats[1], n_far);
        atomicAdd(&b.ctl->stats[2], n_open);
        atomicAdd(&b.ctl->stats[4], static_cast<unsigned long long>(n_vis));
      }
    }
    if (persistent) {
      uint32_t nxt = 0;
      if (lane == 0) nxt = atomicAdd(&b.counters[kWalkItemCounter], 1u) + warps_total;
      item = __shfl_sync(0xffffffffu, nxt, 0);
    } else {
      item = b.nitems;
    }
  }
}

namespace {

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// Opening test for theta >= kInsideTheta: the target inside the child's AABB must open it.
// Returns the adjusted (take, open, amb) of a child whose distance test said "take".
__device__ __forceinline__ void inside_test(const StepBufs& b, const float xh[3], uint32_t gi, bool& take, bool& open,
                                            bool& amb) {
  const float4 nc = __ldg(&b.nodeC[gi]);
  const float4 nd4 = __ldg(&b.nodeD[gi]);
  const float q0 = fabsf(xh[0] - nc.x) - nd4.x;
  const float q1 = fabsf(xh[1] - nc.y) - nd4.y;
  const float q2 = fabsf(xh[2] - nc.z) - nd4.z;
  const float t0 = 0x1p-20f * (fabsf(nc.x) + nd4.x) + 1e-30f;
  const float t1 = 0x1p-20f * (fabsf(nc.y) + nd4.y) + 1e-30f;
  const float t2 = 0x1p-20f * (fabsf(nc.z) + nd4.z) + 1e-30f;
  const bool near_face = fabsf(q0) <= t0 || fabsf(q1) <= t1 || fabsf(q2) <= t2;
  const bool inside = q0 < 0.f && q1 < 0.f && q2 < 0.f;
  const bool t = take;
  take = t && !near_face && !inside;
  open = open || (t && !near_face && inside);
  amb = amb || (t && near_face);
}

// True when internal node gi's AABB (FP32 centre / half extents, rounded from FP64) and
// the targets' padded box (negated faces nlo, nhi) are apart along some axis by more than
// the rounding of the FP32 box, so that no target is inside the node.
__device__ __forceinline__ bool boxes_apart(const StepBufs& b, uint32_t gi, const float2 nlo[3], const float2 nhi[3]) {
  const float4 nc = __ldg(&b.nodeC[gi]);
  const float4 nd = __ldg(&b.nodeD[gi]);
  const float c[3] = {nc.x, nc.y, nc.z}, h[3] = {nd.x, nd.y, nd.z};
  bool apart = false;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float m = 0x1p-20f * (fabsf(c[a]) + h[a]) + 1e-30f;
    const float lo = -nlo[a].x, hi = -nhi[a].x;
    apart = apart || lo > c[a] + h[a] + m || hi < c[a] - h[a] - m;
  }
  return apart;
}

// FP64 decision of an undecided child with record code c (a leaf is undecided only
// when massless: skip).
__device__ __forceinline__ void resolve(const StepBufs& b, uint32_t k, double theta, uint32_t c, bool& take,
                                        bool& open) {
  int dec = -1;
  if (!(c & kLeafCode)) {
    const double4 p = b.leaf64[k];
    const double x[3] = {p.x, p.y, p.z};
    dec = exact_decision(b.agg64, c, x, theta);
  }
  take = dec == 1;
  open = dec == 0;
}

}  // namespace

#ifndef GX_WALK_MINB
#define GX_WALK_MINB 4  // resident kWalkThreads-thread blocks per SM (shared memory bounds it at 4)
#endif

namespace {

// Margins of the warp-wide (group) opening test. A child is taken for every target of
// the warp when the squared distance from its centre of mass to the targets' bounding
// box, times (1 - 2^-20), exceeds the child's take threshold, and opened for every
// target when the squared distance to the box's farthest corner, times (1 + 2^-20),
// is below its open threshold. The box is padded by 2^-21 of its coordinates, which
// covers the float-float split of every target, and the margins cover the FP32
// rounding of the box distances (a few ulps), so a group decision is the decision
// the reference's exact test makes for each target: the thresholds already hold the
// 4e-6 band around rcrit^2.
constexpr float kGroupLo = 1.0f - 0x1p-20f;
// Per-warp stack and list sizes of the FP32 walk (see WarpLists).
constexpr int kWalkStack = 384;  // stack entries
constexpr int kWalkDeep = kWalkStack - kMaxDepth - 36;  // stack entries the wide rounds may fill
constexpr int kWalkList = 96;    // entries per list: at most 31 left after an evaluation + 64 a round
constexpr int kWalkFlush = 32;   // a list is evaluated once it holds this many entries
// Undecided and near entries together: at most 31 of each are left over, a round adds at most
// 64 undecided ones and a batch of those moves at most its own number to the near list.
constexpr int kWalkPool = 128;
static_assert(31 + 31 + 64 <= kWalkPool, "undecided and near entries");
// What some targets of an undecided entry take is evaluated relative to the centre of the
// targets' box when the box's far corner is at most sqrt(kNearRatio) times as far from the
// entry as any target that takes it. The four roundings of the two relative coordinates are
// then within 2 sqrt(kNearRatio) 2^-24 (1.9e-6) of the distance, at the rule's edge; most
// entries lie far inside it. Nearer entries keep float-float coordinates, whose difference is
// exact to 2^-24 of itself. Measured over spheres, disks, collisions, cubes and clumps of 1,000
// to 600,000 particles at theta 0.3 to 1, 784 walks against the FP64 walk, errors over those
// of the walk that kept all undecided entries float-float, geometric means of the
// largest / median error of a walk's particles: ratio 4 1.00 / 0.78, 16 1.00 / 0.80, 64 1.00 /
// 0.81, 256 1.00 / 0.82 (the sums leave FP32 compensated, which that walk's did not), no near
// list 1.60 / 1.01, and up to 160 times the largest. Walk of the collision of 2^20, of 16,384
// with quadrupoles, us: 3977, 209; 3904, 201; 3881, 195; 3865, 193.
constexpr float kNearRatio = 256.f;
constexpr uint32_t kNearCode = 0x40000000u;  // flag of an undecided entry's code (indices are below 2^30)
constexpr float kGroupHi = 1.0f + 0x1p-20f;

// Order-preserving map of a float onto a signed int (for warp min / max reductions).
__device__ __forceinline__ int ford(float f) {
  const int i = __float_as_int(f);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float fdeord(int i) { return __int_as_float(i ^ ((i >> 31) & 0x7fffffff)); }

// Two list entries share each float4: entry e is half (e & 1) of float4 e >> 1, so a
// broadcast load of one float4 yields (entry 2p, entry 2p + 1) operand pairs for the
// packed FP32 instructions.
__device__ __forceinline__ void put2(float4* a, int e, float v0, float v1) {
  float* p = reinterpret_cast<float*>(a + (e >> 1)) + (e & 1);
  p[0] = v0;
  p[2] = v1;
}

}  // namespace

// Per-warp shared memory of the FP32 walk.
//   stk: (internal node, target mask) -- the node was opened for the targets in the mask
//        and its two children are still to be decided for them;
//   dense list: children every target of their mask takes, evaluated with no per-target
//        decision, in FP32 coordinates relative to the centre of the warp's target box;
//        two entries share each float4: entry e is half (e & 1) of float4 e >> 1;
//   undecided list: children some targets take and others open (or that need the FP64
//        re-decision), one field an array: a lane decides one entry for every target;
//   near list: once undecided children that some targets take, so close to the targets, for
//        the size of the targets' box, that coordinates relative to its centre would lose
//        bits (kNearRatio): they keep float-float coordinates. It grows down from the end
//        of the undecided list's arrays;
//   targets: the float-float coordinates of the warp's targets, negated, two a float4, so
//        that one broadcast load serves the packed instructions of two targets.
struct WarpLists {
  uint2 stk[kWalkStack];
  float4 da[kWalkList / 2], db[kWalkList / 2];  // (x, y) (z, m) relative to the box centre
  uint2 dm[kWalkList / 2];                      // target masks
  uint32_t dcode[kWalkList];                    // child codes (quadrupole terms, statistics)
  float uxh[kWalkPool], uyh[kWalkPool], uzh[kWalkPool], uxl[kWalkPool], uyl[kWalkPool], uzl[kWalkPool];
  float um[kWalkPool], utake[kWalkPool], uopen[kWalkPool];
  uint32_t ucode[kWalkPool], umask[kWalkPool];
  float4 ta[16], tb[16], tc[16];  // (xh,yh) (zh,xl) (yl,zl) of targets 2i, 2i + 1, negated
  // The targets' padded box as negated faces (lo, hi) and its negated centre o, each
  // duplicated for packed pairs: warp-uniform, read by the rounds only (kept here rather
  // than in 18 registers of every lane).
  float2 nlo[3], nhi[3], no[3];
  float2 pad;
};
static_assert(sizeof(WarpLists) % 16 == 0, "warp lists keep 16-byte alignment");

// Bound of the stack: a popped entry leads to at most two pushes, at once or from the
// undecided list, so a round of kk entries raises stacked + undecided entries by at most kk;
// a round takes no more than keep them within kWalkDeep. At that height it takes one entry
// and decides its undecided children at once: the stack then grows like a depth-first
// walk, by at most one entry per tree level. 384 entries: the collisions fill about 250
// often (320 entries: 20% slower); more only take room from the L1 (512: the walk of a
// 16,384-particle sphere with quadrupoles 209 us against 190).
static_assert(kWalkDeep >= 128 && kWalkDeep + kMaxDepth + 4 <= kWalkStack, "walk stack bound");

// Quadrupole mode: each dense internal node's traceless moments, fetched once by the lane
// that lists it and stored with the two entries of a pair side by side, as the packed
// evaluation reads them: a = (xx, xx', xy, xy'), b = (xz, xz', yy, yy'), c = (yz, yz', zz, zz').
// Slots of leaf entries are never written: the evaluation gives them a zero inverse
// distance, and the arrays are cleared at the kernel's start so that every slot holds
// finite values.
struct WarpQuads {
  float4 dqa[kWalkList / 2], dqb[kWalkList / 2], dqc[kWalkList / 2];
};

static_assert(kWalkCtas * ((kWalkThreads / 32) * sizeof(WarpLists) + 1024) <= 227 * 1024 &&
                  kWalkCtasQuad * ((kWalkThreads / 32) * (sizeof(WarpLists) + sizeof(WarpQuads)) + 1024) <= 227 * 1024,
              "resident walk blocks");

size_t walk_smem_bytes(int block, bool quad) {
  return static_cast<size_t>(block / 32) * (sizeof(WarpLists) + (quad ? sizeof(WarpQuads) : 0));
}

namespace {

// Plummer-softened monopole terms of two entries for one target: t += d m / (d^2 + eps^2)^1.5
// where the target takes the entry (t0, t1). r^2 is clamped at 1e-24 so that a zero
// distance (the target's own leaf) gives an exact zero term even without softening.
__device__ __forceinline__ void mono2(float2 dx, float2 dy, float2 dz, float2 m, float2 eps2, bool t0, bool t1,
                                      float2& tx, float2& ty, float2& tz, float& i0, float& i1) {
  const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
  const float2 r2s = __fadd2_rn(d2, eps2);
  i0 = rsqrtf(fmaxf(r2s.x, 1e-24f));
  i1 = rsqrtf(fmaxf(r2s.y, 1e-24f));
  const float2 inv = f2(i0, i1);
  const float2 inv3 = __fmul2_rn(inv, __fmul2_rn(inv, inv));
  float2 f = __fmul2_rn(m, inv3);
  f.x = t0 ? f.x : 0.f;
  f.y = t1 ? f.y : 0.f;
  tx = __ffma2_rn(dx, f, tx);
  ty = __ffma2_rn(dy, f, ty);
  tz = __ffma2_rn(dz, f, tz);
}

// Stores entry e's moments (xx, xy, xz, yy), (yz, zz) into the pair layout of WarpQuads.
__device__ __forceinline__ void put_quad(float4* qa, float4* qb, float4* qc, int e, const float4& a, const float4& c) {
  const int p = e >> 1, h = e & 1;
  float* A = reinterpret_cast<float*>(qa + p) + h;
  float* B = reinterpret_cast<float*>(qb + p) + h;
  float* C = reinterpret_cast<float*>(qc + p) + h;
  A[0] = a.x;
  A[2] = a.y;
  B[0] = a.z;
  B[2] = a.w;
  C[0] = c.x;
  C[2] = c.y;
}

// Quadrupole terms of the two entries of a pair for one target, packed FP32, added to the
// monopole accumulator: with r = x - com = -d, a += Q r / r^5 - 2.5 (r.Q r) r / r^7
// = -(Q d) / r^5 + 2.5 (d.Q d) d / r^7, r^2 softened like the monopole. inv is the
// inverse distance of an entry the target takes as an internal node, else 0.
__device__ __forceinline__ void quad2(float2 dx, float2 dy, float2 dz, float2 inv, const float4& qa, const float4& qb,
                                      const float4& qc, float2& tx, float2& ty, float2& tz) {
  const float2 xx = f2(qa.x, qa.y), xy = f2(qa.z, qa.w), xz = f2(qb.x, qb.y);
  const float2 yy = f2(qb.z, qb.w), yz = f2(qc.x, qc.y), zz = f2(qc.z, qc.w);
  const float2 qx = __ffma2_rn(xx, dx, __ffma2_rn(xy, dy, __fmul2_rn(xz, dz)));
  const float2 qy = __ffma2_rn(xy, dx, __ffma2_rn(yy, dy, __fmul2_rn(yz, dz)));
  const float2 qz = __ffma2_rn(xz, dx, __ffma2_rn(yz, dy, __fmul2_rn(zz, dz)));
  const float2 dqd = __ffma2_rn(dx, qx, __ffma2_rn(dy, qy, __fmul2_rn(dz, qz)));
  const float2 inv2 = __fmul2_rn(inv, inv);
  const float2 ninv5 = __fmul2_rn(__fmul2_rn(inv2, inv2), f2(-inv.x, -inv.y));      // -1 / r^5
  const float2 c7 = __fmul2_rn(__fmul2_rn(f2(-2.5f, -2.5f), dqd), __fmul2_rn(ninv5, inv2));  // 2.5 dQd / r^7
  tx = __ffma2_rn(dx, c7, __ffma2_rn(qx, ninv5, tx));
  ty = __ffma2_rn(dy, c7, __ffma2_rn(qy, ninv5, ty));
  tz = __ffma2_rn(dz, c7, __ffma2_rn(qz, ninv5, tz));
}

}  // namespace

// FP32 walk: one warp per G Morton-consecutive targets (G = 8, 16 or 32: the system's
// grouping, or the target list's), R = 32 / G lanes a target; the warp visits the union
// of their walks (each node is decided once for every target that reached it) but not
// one node at a time. A round pops up to 32 opened nodes from the warp's stack, one per
// lane, loads each one's sibling-pair record (both children: float-float centre of mass,
// mass, FP32 take / open thresholds, child codes) and decides each child for the whole
// warp against the padded bounding box of the warp's targets:
//   - taken by every target (or a leaf): appended to the dense list;
//   - opened by every target: pushed back on the stack with the same target mask;
//   - otherwise: appended to the undecided list.
// An undecided batch of 32 entries is decided one entry a lane, for every target in turn
// (two at a time, packed FP32 on float-float coordinates read from shared memory; FP64
// re-decision in the band, the inside test for theta >= kInsideTheta): the masks of the
// targets that take and that open the entry build up in the lane's registers. (Deciding
// an entry for a target a lane costs six shared loads, two ballots and a vote an entry;
// this way none: the collision of 2^20 at theta 0.5, 6.0 -> 4.5 ms.) An entry
// some targets open goes back on the stack for them, one some targets take goes on the
// dense list for them. The dense list is evaluated a target a lane (the R lanes of a
// target take turns over its entries), four entries a lane-iteration with packed FP32 and
// no decisions. Rounds, lists and entries are independent of one another, so the walk has
// no dependent chain of one record per step. Rounds narrow as the stack fills (kWalkDeep),
// which bounds it within kWalkStack. Every target takes exactly the reference's
// set of terms; only the order of summation differs from the FP64 walk. Terms are summed
// four at a time into a Kahan-compensated accumulator. Node indices are clamped into the
// record array and the number of records a warp visits is bounded by the system's node
// count, so even a corrupt tree cannot read out of bounds or loop; a clamp, an exhausted
// budget or a full stack raises the device error word.
template <bool QUAD, bool KAHAN, bool STATS, bool INSIDE, bool LIST>
__global__ void __launch_bounds__(kWalkThreads, GX_WALK_MINB) k_walk_f32(StepBufs b, int persistent) {
  extern __shared__ __align__(16) unsigned char s_walk_raw[];
  WarpLists& L = reinterpret_cast<WarpLists*>(s_walk_raw)[threadIdx.x >> 5];
  WarpQuads& Q = reinterpret_cast<WarpQuads*>(s_walk_raw + (blockDim.x >> 5) * sizeof(WarpLists))[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t warps_total = (gridDim.x * blockDim.x) >> 5;
  uint32_t item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t n_total = b.n;
  const float4* __restrict__ pairs = b.pairs;
  if (QUAD) {
    float4* z = reinterpret_cast<float4*>(&Q);
    for (int i = lane; i < static_cast<int>(sizeof(WarpQuads) / sizeof(float4)); i += 32) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();
  }
  while (item < b.nitems) {
    const WalkItem it = b.items[item];
    const SysDesc sd = b.sys[it.sys];
    const uint32_t end = sd.off + sd.n;
    // G targets a warp, R = 32 / G lanes a target: lane = sub * G + target, so the lanes of
    // one sub-lane index hold contiguous ballot bits. Masks have one bit per target.
    const uint32_t G = LIST ? b.group : sd.group;
    const int lg = __ffs(G) - 1;
    const uint32_t gmask = G == 32 ? 0xffffffffu : (1u << G) - 1u;
    const int tg = lane & (G - 1), sl = lane >> lg, R = 32 >> lg;
    const uint32_t tbit = 1u << tg;
    // a target list (active-subset walk) names the item's G targets; else they are the
    // G sorted positions from it.begin
    const uint32_t li = it.begin + tg;
    const bool valid = LIST ? li < *b.ntargets : li < end;
    const uint32_t k = LIST ? (valid ? b.targets[li] : 0u) : li;
    const uint32_t vmask = __ballot_sync(0xffffffffu, valid) & gmask;
    // Kahan state: (x, y) packed, z scalar.
    float2 sxy = f2(0.f, 0.f), cxy = f2(0.f, 0.f);
    float sz = 0.f, cz = 0.f;
    unsigned long long n_leaf = 0, n_far = 0, n_open = 0, n_re = 0, n_vis = 0;
    bool bad = false;
    // The root's box is the system's box, so every target is inside it and every target
    // opens it -- unless the whole system is massless, when nothing is added.
    const uint32_t root = sd.off;  // internal node 0 of the system
    if (sd.n > 1 && vmask && __ldg(&b.agg64[root].m) > 0.0) {
      const float eps2f = __double2float_rn(dmul(sd.eps, sd.eps));
      const float2 eps2 = f2(eps2f, eps2f);
      // The inside rule (a target inside a node's box opens it) can only bind from
      // kInsideTheta on; it follows the system's own theta (as the single-system
      // handle's choice of kernel does), so a system's terms and their order do not
      // depend on the other systems of a batch.
      const bool inside_rule = INSIDE && sd.theta >= kInsideTheta;
      float xh[3] = {0.f, 0.f, 0.f}, xl[3] = {0.f, 0.f, 0.f};
      if (valid) {
        const double4 p = b.leaf64[k];
        split_ff(p.x, xh[0], xl[0]);
        split_ff(p.y, xh[1], xl[1]);
        split_ff(p.z, xh[2], xl[2]);
      }
      if (sl == 0) {
        float* A = reinterpret_cast<float*>(L.ta + (tg >> 1)) + (tg & 1);
        float* B = reinterpret_cast<float*>(L.tb + (tg >> 1)) + (tg & 1);
        float* C = reinterpret_cast<float*>(L.tc + (tg >> 1)) + (tg & 1);
        A[0] = -xh[0];
        A[2] = -xh[1];
        B[0] = -xh[2];
        B[2] = -xl[0];
        C[0] = -xl[1];
        C[2] = -xl[2];
      }
      // The targets' padded bounding box as negated faces (lo, hi), duplicated, and its
      // centre o (an FP32 value): dense entries and targets are stored relative to o. A
      // target that is not finite turns the box into all of space: no group decisions.
      const bool fin = isfinite(xh[0]) && isfinite(xh[1]) && isfinite(xh[2]);
      const bool all_fin = __all_sync(0xffffffffu, !valid || fin);
      float xr[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        float l = fdeord(__reduce_min_sync(0xffffffffu, valid ? ford(xh[c]) : 0x7fffffff));
        float h = fdeord(__reduce_max_sync(0xffffffffu, valid ? ford(xh[c]) : static_cast<int>(0x80000000u)));
        const float o = all_fin ? 0.5f * l + 0.5f * h : 0.f;
        const float pad = (fabsf(l) + fabsf(h)) * 0x1p-21f + 1e-30f;
        l = all_fin ? l - pad : -INFINITY;
        h = all_fin ? h + pad : INFINITY;
        if (lane == 0) {
          L.nlo[c] = f2(-l, -l);
          L.nhi[c] = f2(-h, -h);
          L.no[c] = f2(-o, -o);
        }
        xr[c] = (xh[c] - o) + xl[c];  // the target relative to o
      }
      const float2 nxr = f2(-xr[0], -xr[0]), nyr = f2(-xr[1], -xr[1]), nzr = f2(-xr[2], -xr[2]);
      const uint32_t gmax = n_total - 1;
      const uint32_t max_pairs = sd.n + 64u;
      uint32_t pairs_done = 0;
      int sp = 1, dl = 0, ul = 0, nl = 0;  // heights of the stack and the dense, undecided, near lists
      if (lane == 0) L.stk[0] = make_uint2(root, vmask);
      __syncwarp();
      float2 tx = f2(0.f, 0.f), ty = f2(0.f, 0.f), tz = f2(0.f, 0.f);  // per-entry term sums
      // add the term sums of the last entries to the lane's compensated accumulator
      auto fold = [&]() {
        const float2 txy = f2(tx.x + tx.y, ty.x + ty.y);
        const float tzz = tz.x + tz.y;
        if (KAHAN) {
          const float2 y = __fadd2_rn(txy, f2(-cxy.x, -cxy.y));
          const float2 u = __fadd2_rn(sxy, y);
          cxy = __fadd2_rn(__fadd2_rn(u, f2(-sxy.x, -sxy.y)), f2(-y.x, -y.y));
          sxy = u;
          const float yz = tzz - cz;
          const float uz = sz + yz;
          cz = (uz - sz) - yz;
          sz = uz;
        } else {
          sxy = __fadd2_rn(sxy, txy);
          sz += tzz;
        }
        tx = ty = tz = f2(0.f, 0.f);
      };
      auto put_dense = [&](int e, float x_, float y_, float z_, float m_, uint32_t mask, uint32_t code) {
        put2(L.da, e, x_, y_);
        put2(L.db, e, z_, m_);
        reinterpret_cast<uint32_t*>(L.dm + (e >> 1))[e & 1] = mask;
        L.dcode[e] = code;
      };
      auto put_und = [&](int e, float xh_, float yh_, float zh_, float m_, float xl_, float yl_, float zl_,
                         float take, float open, uint32_t code, uint32_t mask) {
        L.uxh[e] = xh_;
        L.uyh[e] = yh_;
        L.uzh[e] = zh_;
        L.um[e] = m_;
        L.uxl[e] = xl_;
        L.uyl[e] = yl_;
        L.uzl[e] = zl_;
        L.utake[e] = take;
        L.uopen[e] = open;
        L.ucode[e] = code;
        L.umask[e] = mask;
      };
      // One round: the top kk stack entries, one per lane, each child decided for the
      // whole warp and appended to a list or pushed back.
      auto round = [&](int kk) {
        const bool act = lane < kk;
        uint32_t g = 0, M = 0;
        if (act) {
          const uint2 e = L.stk[sp - kk + lane];
          g = e.x;
          M = e.y;
        }
        sp -= kk;
        __syncwarp();  // popped before the pushes below overwrite the slots
        bad |= act && g > gmax;
        g = min(g, gmax);
        float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0, r2 = r0, r3 = r0, r4 = r0;
        if (act) {
          const float4* pr = pairs + 5 * (size_t)g;
          r0 = __ldg(pr);
          r1 = __ldg(pr + 1);
          r2 = __ldg(pr + 2);
          r3 = __ldg(pr + 3);
          r4 = __ldg(pr + 4);
        }
        const uint32_t cL = __float_as_uint(r4.z), cR = __float_as_uint(r4.w);
        const float2 nlo[3] = {L.nlo[0], L.nlo[1], L.nlo[2]}, nhi[3] = {L.nhi[0], L.nhi[1], L.nhi[2]};
        const float2 chx = f2(r0.x, r0.y), chy = f2(r0.z, r0.w), chz = f2(r1.x, r1.y);
        const float2 clx = f2(r2.x, r2.y), cly = f2(r2.z, r2.w), clz = f2(r3.x, r3.y);
        // c - lo and c - hi per axis, both children at once
        const float2 lx = __fadd2_rn(__fadd2_rn(chx, nlo[0]), clx), hx = __fadd2_rn(__fadd2_rn(chx, nhi[0]), clx);
        const float2 ly = __fadd2_rn(__fadd2_rn(chy, nlo[1]), cly), hy = __fadd2_rn(__fadd2_rn(chy, nhi[1]), cly);
        const float2 lz = __fadd2_rn(__fadd2_rn(chz, nlo[2]), clz), hz = __fadd2_rn(__fadd2_rn(chz, nhi[2]), clz);
        // distance to the box (0 inside) and to its farthest corner, per axis
        const float2 nx = f2(fmaxf(fmaxf(-lx.x, hx.x), 0.f), fmaxf(fmaxf(-lx.y, hx.y), 0.f));
        const float2 ny = f2(fmaxf(fmaxf(-ly.x, hy.x), 0.f), fmaxf(fmaxf(-ly.y, hy.y), 0.f));
        const float2 nz = f2(fmaxf(fmaxf(-lz.x, hz.x), 0.f), fmaxf(fmaxf(-lz.y, hz.y), 0.f));
        const float2 fx = f2(fmaxf(lx.x, -hx.x), fmaxf(lx.y, -hx.y));
        const float2 fy = f2(fmaxf(ly.x, -hy.x), fmaxf(ly.y, -hy.y));
        const float2 fz = f2(fmaxf(lz.x, -hz.x), fmaxf(lz.y, -hz.y));
        const float2 dmin2 = __ffma2_rn(nx, nx, __ffma2_rn(ny, ny, __fmul2_rn(nz, nz)));
        const float2 dmax2 = __ffma2_rn(fx, fx, __ffma2_rn(fy, fy, __fmul2_rn(fz, fz)));
        bool accL = act && dmin2.x * kGroupLo > r3.z, accR = act && dmin2.y * kGroupLo > r3.w;
        if (inside_rule) {
          // A target inside a node's box opens it: a node is taken for the whole warp only
          // when its box and the targets' box are apart along some axis.
          if (accL && !(cL & kLeafCode)) accL = boxes_apart(b, cL, nlo, nhi);
          if (accR && !(cR & kLeafCode)) accR = boxes_apart(b, cR, nlo, nhi);
        }
        const bool opnL = act && !accL && dmax2.x * kGroupHi < r4.x;
        const bool opnR = act && !accR && dmax2.y * kGroupHi < r4.y;
        const bool undL = act && !accL && !opnL, undR = act && !accR && !opnR;
        // undecided and too near for box-relative coordinates: what is taken is farther than
        // dmin, and than the take threshold
        const bool nearL = dmax2.x > kNearRatio * fmaxf(dmin2.x, r3.z), nearR = dmax2.y > kNearRatio * fmaxf(dmin2.y, r3.w);
        const uint32_t bAL = __ballot_sync(0xffffffffu, accL), bAR = __ballot_sync(0xffffffffu, accR);
        const uint32_t bUL = __ballot_sync(0xffffffffu, undL), bUR = __ballot_sync(0xffffffffu, undR);
        const uint32_t bOL = __ballot_sync(0xffffffffu, opnL), bOR = __ballot_sync(0xffffffffu, opnR);
        const int eAL = dl + __popc(bAL & lt), eAR = dl + __popc(bAL) + __popc(bAR & lt);
        const int eUL = ul + __popc(bUL & lt), eUR = ul + __popc(bUL) + __popc(bUR & lt);
        if (QUAD) {
          // the moments of the listed internal children, loaded side by side
          const bool qL = accL && !(cL & kLeafCode), qR = accR && !(cR & kLeafCode);
          float4 qaL = make_float4(0.f, 0.f, 0.f, 0.f), qbL = qaL, qaR = qaL, qbR = qaL;
          if (qL) {
            qaL = __ldg(&b.nodeQ[2 * (size_t)cL]);
            qbL = __ldg(&b.nodeQ[2 * (size_t)cL + 1]);
          }
          if (qR) {
            qaR = __ldg(&b.nodeQ[2 * (size_t)cR]);
            qbR = __ldg(&b.nodeQ[2 * (size_t)cR + 1]);
          }
          if (qL) put_quad(Q.dqa, Q.dqb, Q.dqc, eAL, qaL, qbL);
          if (qR) put_quad(Q.dqa, Q.dqb, Q.dqc, eAR, qaR, qbR);
        }
        if (accL || accR) {
          // dense entries relative to the box centre: (c_hi - o) + c_lo
          const float2 rx = __fadd2_rn(__fadd2_rn(chx, L.no[0]), clx);
          const float2 ry = __fadd2_rn(__fadd2_rn(chy, L.no[1]), cly);
          const float2 rz = __fadd2_rn(__fadd2_rn(chz, L.no[2]), clz);
          if (accL) put_dense(eAL, rx.x, ry.x, rz.x, r1.z, M, cL);
          if (accR) put_dense(eAR, rx.y, ry.y, rz.y, r1.w, M, cR);
        }
        dl += __popc(bAL) + __popc(bAR);
        if (undL)
          put_und(eUL, chx.x, chy.x, chz.x, r1.z, clx.x, cly.x, clz.x, r3.z, r4.x, cL | (nearL ? kNearCode : 0u), M);
        if (undR)
          put_und(eUR, chx.y, chy.y, chz.y, r1.w, clx.y, cly.y, clz.y, r3.w, r4.y, cR | (nearR ? kNearCode : 0u), M);
        ul += __popc(bUL) + __popc(bUR);
        const int npush = __popc(bOL) + __popc(bOR);
        if (sp + npush > kWalkStack) {
          bad = true;
        } else {
          if (opnL) L.stk[sp + __popc(bOL & lt)] = make_uint2(cL, M);
          if (opnR) L.stk[sp + __popc(bOL) + __popc(bOR & lt)] = make_uint2(cR, M);
          sp += npush;
        }
        if (STATS) {
          n_vis += kk;
          n_open += (opnL ? __popc(M) : 0) + (opnR ? __popc(M) : 0);
        }
        __syncwarp();
      };
      // The dense terms of pair p (entries 2p, 2p + 1) for this lane's target.
      auto dense_pair = [&](int p) {
        const float4 A = L.da[p], B = L.db[p];
        const uint2 Mk = L.dm[p];
        const float2 dx = __fadd2_rn(f2(A.x, A.y), nxr);
        const float2 dy = __fadd2_rn(f2(A.z, A.w), nyr);
        const float2 dz = __fadd2_rn(f2(B.x, B.y), nzr);
        const bool t0 = (Mk.x & tbit) != 0u, t1 = (Mk.y & tbit) != 0u;
        float i0, i1;
        mono2(dx, dy, dz, f2(B.z, B.w), eps2, t0, t1, tx, ty, tz, i0, i1);
        if (QUAD || STATS) {
          const uint32_t c0 = L.dcode[2 * p], c1 = L.dcode[2 * p + 1];
          if (QUAD) {
            const float2 iq = f2(t0 && !(c0 & kLeafCode) ? i0 : 0.f, t1 && !(c1 & kLeafCode) ? i1 : 0.f);
            quad2(dx, dy, dz, iq, Q.dqa[p], Q.dqb[p], Q.dqc[p], tx, ty, tz);
          }
          if (STATS) {
            const uint32_t self = kLeafCode | k;
            n_leaf += (t0 && (c0 & kLeafCode) && c0 != self ? 1 : 0) + (t1 && (c1 & kLeafCode) && c1 != self ? 1 : 0);
            n_far += (t0 && !(c0 & kLeafCode) ? 1 : 0) + (t1 && !(c1 & kLeafCode) ? 1 : 0);
          }
        }
      };
      // Evaluate the dense list: every target adds the terms of the entries in its mask.
      // An iteration takes 4 R entries, the R lanes of a target two pairs each; the entries
      // short of a whole iteration move to the front of the list and wait for more, except
      // at the walk's end, when empty entries fill the iteration up.
      const int chunk = 4 * R;
      auto flush_dense = [&](bool last) {
        int full = dl & ~(chunk - 1);
        if (last && full < dl) {
          full += chunk;
          if (dl + lane < full) put_dense(dl + lane, 0.f, 0.f, 0.f, 0.f, 0u, kLeafCode);
          dl = full;
          __syncwarp();
        }
        for (int pa = 2 * sl; 2 * pa < full; pa += 2 * R) {
          dense_pair(pa);
          dense_pair(pa + 1);
          fold();
        }
        const int rest = dl - full;  // < chunk <= 32
        if (rest && full) {
          const int e = full + lane;
          const bool mv = lane < rest;
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          uint32_t mk = 0, code = 0;
          float4 qa = v, qb = v;
          if (mv) {
            const float* A = reinterpret_cast<const float*>(L.da + (e >> 1)) + (e & 1);
            const float* B = reinterpret_cast<const float*>(L.db + (e >> 1)) + (e & 1);
            v = make_float4(A[0], A[2], B[0], B[2]);
            mk = reinterpret_cast<const uint32_t*>(L.dm + (e >> 1))[e & 1];
            code = L.dcode[e];
            if (QUAD) {
              const float* qA = reinterpret_cast<const float*>(Q.dqa + (e >> 1)) + (e & 1);
              const float* qB = reinterpret_cast<const float*>(Q.dqb + (e >> 1)) + (e & 1);
              const float* qC = reinterpret_cast<const float*>(Q.dqc + (e >> 1)) + (e & 1);
              qa = make_float4(qA[0], qA[2], qB[0], qB[2]);
              qb = make_float4(qC[0], qC[2], 0.f, 0.f);
            }
          }
          __syncwarp();
          if (mv) {
            put_dense(lane, v.x, v.y, v.z, v.w, mk, code);
            if (QUAD) put_quad(Q.dqa, Q.dqb, Q.dqc, lane, qa, qb);
          }
        }
        dl = rest;
        __syncwarp();  // read before the next round overwrites the list
      };
      // Evaluate the near list as flush_dense does the dense one, on float-float coordinates.
      auto flush_near = [&](bool last) {
        int full = nl & ~(chunk - 1);
        if (last && full < nl) {
          full += chunk;
          if (nl + lane < full)
            put_und(kWalkPool - 1 - (nl + lane), 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, kLeafCode, 0u);
          nl = full;
          __syncwarp();
        }
        const float* TA = reinterpret_cast<const float*>(L.ta + (tg >> 1)) + (tg & 1);
        const float* TB = reinterpret_cast<const float*>(L.tb + (tg >> 1)) + (tg & 1);
        const float* TC = reinterpret_cast<const float*>(L.tc + (tg >> 1)) + (tg & 1);
        const float2 nxh = f2(TA[0], TA[0]), nyh = f2(TA[2], TA[2]), nzh = f2(TB[0], TB[0]);
        const float2 nxl = f2(TB[2], TB[2]), nyl = f2(TC[0], TC[0]), nzl = f2(TC[2], TC[2]);
        auto at = [](const float* a, int e) { return *reinterpret_cast<const float2*>(a + e); };
        for (int q = 2 * sl; 2 * q < full; q += 2 * R) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int e = kWalkPool - 2 - 2 * (q + h);
            const float2 dx = __fadd2_rn(__fadd2_rn(at(L.uxh, e), nxh), __fadd2_rn(at(L.uxl, e), nxl));
            const float2 dy = __fadd2_rn(__fadd2_rn(at(L.uyh, e), nyh), __fadd2_rn(at(L.uyl, e), nyl));
            const float2 dz = __fadd2_rn(__fadd2_rn(at(L.uzh, e), nzh), __fadd2_rn(at(L.uzl, e), nzl));
            const uint2 Mk = *reinterpret_cast<const uint2*>(L.umask + e);
            const bool t0 = (Mk.x & tbit) != 0u, t1 = (Mk.y & tbit) != 0u;
            float i0, i1;
            mono2(dx, dy, dz, at(L.um, e), eps2, t0, t1, tx, ty, tz, i0, i1);
            if (QUAD || STATS) {
              const uint2 cc = *reinterpret_cast<const uint2*>(L.ucode + e);
              const bool f0 = t0 && !(cc.x & kLeafCode), f1 = t1 && !(cc.y & kLeafCode);
              if (QUAD && (f0 || f1)) {
                const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 a0 = f0 ? __ldg(&b.nodeQ[2 * (size_t)cc.x]) : z4, c0 = f0 ? __ldg(&b.nodeQ[2 * (size_t)cc.x + 1]) : z4;
                const float4 a1 = f1 ? __ldg(&b.nodeQ[2 * (size_t)cc.y]) : z4, c1 = f1 ? __ldg(&b.nodeQ[2 * (size_t)cc.y + 1]) : z4;
                quad2(dx, dy, dz, f2(f0 ? i0 : 0.f, f1 ? i1 : 0.f), make_float4(a0.x, a1.x, a0.y, a1.y),
                      make_float4(a0.z, a1.z, a0.w, a1.w), make_float4(c0.x, c1.x, c0.y, c1.y), tx, ty, tz);
              }
              if (STATS) {
                const uint32_t self = kLeafCode | k;
                n_leaf += (t0 && (cc.x & kLeafCode) && cc.x != self ? 1 : 0) + (t1 && (cc.y & kLeafCode) && cc.y != self ? 1 : 0);
                n_far += (f0 ? 1 : 0) + (f1 ? 1 : 0);
              }
            }
          }
          fold();
        }
        const int rest = nl - full;  // < chunk <= 32
        if (rest && full) {
          const int e = kWalkPool - 1 - (full + min(lane, rest - 1)), d = kWalkPool - 1 - lane;
          const float v0 = L.uxh[e], v1 = L.uyh[e], v2 = L.uzh[e], v3 = L.um[e], v4 = L.uxl[e], v5 = L.uyl[e], v6 = L.uzl[e];
          const uint32_t code = L.ucode[e], mk = L.umask[e];
          __syncwarp();
          if (lane < rest) put_und(d, v0, v1, v2, v3, v4, v5, v6, 0.f, 0.f, code, mk);
        }
        nl = rest;
        __syncwarp();  // read before it is overwritten
      };
      // Decide the last cnt (<= 32) undecided entries, one a lane, for every target: bit t of
      // tm / om is set when target t takes / opens the entry. The comparisons are sign bits
      // (take - d2 < 0, d2 - open < 0) shifted into the masks, highest target first; NaN
      // thresholds become infinite ones, which neither comparison passes.
      auto und_batch = [&](int cnt) {
        ul -= cnt;
        const bool act = lane < cnt;
        const int e = ul + (act ? lane : 0);
        const float ex = L.uxh[e], ey = L.uyh[e], ez = L.uzh[e], exl = L.uxl[e], eyl = L.uyl[e], ezl = L.uzl[e];
        const float em = L.um[e], take = L.utake[e], open = L.uopen[e];
        const uint32_t fcode = L.ucode[e], code = fcode & ~kNearCode;
        const uint32_t M = act ? L.umask[e] : 0u;
        const float2 X = f2(ex, ex), Y = f2(ey, ey), Z = f2(ez, ez), XL = f2(exl, exl), YL = f2(eyl, eyl), ZL = f2(ezl, ezl);
        const float tk = take == take ? take : INFINITY, no_ = open == open ? -open : INFINITY;
        const float2 T = f2(tk, tk), N = f2(no_, no_), neg1 = f2(-1.f, -1.f);
        uint32_t tm = 0, om = 0;
#pragma unroll 4
        for (int p = static_cast<int>(G >> 1) - 1; p >= 0; --p) {
          const float4 A = L.ta[p], B = L.tb[p], C = L.tc[p];
          const float2 dx = __fadd2_rn(__fadd2_rn(X, f2(A.x, A.y)), __fadd2_rn(XL, f2(B.z, B.w)));
          const float2 dy = __fadd2_rn(__fadd2_rn(Y, f2(A.z, A.w)), __fadd2_rn(YL, f2(C.x, C.y)));
          const float2 dz = __fadd2_rn(__fadd2_rn(Z, f2(B.x, B.y)), __fadd2_rn(ZL, f2(C.z, C.w)));
          const float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
          const float2 dt = __ffma2_rn(d2, neg1, T);  // take - d2
          const float2 dn = __fadd2_rn(d2, N);        // d2 - open
          tm = __funnelshift_l(__float_as_uint(dt.y), tm, 1);
          om = __funnelshift_l(__float_as_uint(dn.y), om, 1);
          tm = __funnelshift_l(__float_as_uint(dt.x), tm, 1);
          om = __funnelshift_l(__float_as_uint(dn.x), om, 1);
        }
        tm &= M;
        om &= M & ~tm;
        uint32_t am = M & ~(tm | om);
        const auto target = [&](int t) { return LIST ? b.targets[it.begin + t] : it.begin + t; };
        if (inside_rule && !(code & kLeafCode)) {
          for (uint32_t w = tm; w; w &= w - 1u) {
            const int t = __ffs(w) - 1;
            const float* A = reinterpret_cast<const float*>(L.ta + (t >> 1)) + (t & 1);
            const float xt[3] = {-A[0], -A[2], -reinterpret_cast<const float*>(L.tb + (t >> 1))[t & 1]};
            bool tk1 = true, op1 = false, am1 = false;
            inside_test(b, xt, code, tk1, op1, am1);
            if (!tk1) tm &= ~(1u << t);
            if (op1) om |= 1u << t;
            if (am1) am |= 1u << t;
          }
        }
        if (__any_sync(0xffffffffu, am != 0u)) {
          if (STATS) n_re += __popc(am);
          for (uint32_t w = am; w; w &= w - 1u) {
            const int t = __ffs(w) - 1;
            bool tk1, op1;
            resolve(b, target(t), sd.theta, code, tk1, op1);
            if (tk1) tm |= 1u << t;
            if (op1) om |= 1u << t;
          }
          __syncwarp();
        }
        const bool nr = tm != 0u && (fcode & kNearCode), dn = tm != 0u && !nr;
        const uint32_t bo = __ballot_sync(0xffffffffu, om != 0u);
        const uint32_t bt = __ballot_sync(0xffffffffu, dn), bn = __ballot_sync(0xffffffffu, nr);
        if (sp + __popc(bo) > kWalkStack) {
          bad = true;
        } else {
          if (om) L.stk[sp + __popc(bo & lt)] = make_uint2(code, om);
          sp += __popc(bo);
        }
        __syncwarp();  // every lane has read its entry before a near one may take a slot of the batch
        if (nr) put_und(kWalkPool - 1 - (nl + __popc(bn & lt)), ex, ey, ez, em, exl, eyl, ezl, 0.f, 0.f, code, tm);
        nl += __popc(bn);
        if (dn) {
          const int d = dl + __popc(bt & lt);
          put_dense(d, (ex + L.no[0].x) + exl, (ey + L.no[1].x) + eyl, (ez + L.no[2].x) + ezl, em, tm, code);
          if (QUAD && !(code & kLeafCode))
            put_quad(Q.dqa, Q.dqb, Q.dqc, d, __ldg(&b.nodeQ[2 * (size_t)code]), __ldg(&b.nodeQ[2 * (size_t)code + 1]));
        }
        dl += __popc(bt);
        if (STATS) n_open += __popc(om);
        __syncwarp();  // pushes and entries visible; the batch read before it is overwritten
      };
      for (;;) {
        if (__any_sync(0xffffffffu, bad)) break;
        if (dl >= kWalkFlush) flush_dense(false);
        if (nl >= kWalkFlush) flush_near(false);
        if (sp == 0) {
          if (ul == 0) break;
          und_batch(min(32, ul));
          continue;
        }
        const int kk = max(1, min(min(32, sp), kWalkDeep - sp - ul));
        const bool deep = kk == 1;
        pairs_done += kk;
        if (pairs_done > max_pairs) {
          bad = true;
          break;
        }
        round(kk);
        while (ul >= kWalkFlush || (deep && ul > 0)) {
          if (dl >= kWalkFlush) flush_dense(false);
          if (nl >= kWalkFlush) flush_near(false);
          und_batch(min(32, ul));
        }
      }
      if (!__any_sync(0xffffffffu, bad)) {
        if (dl > 0) flush_dense(true);
        if (nl > 0) flush_near(true);
      }
      __syncwarp();  // the next item's stack writes must not race this item's last reads
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) raise_err(b.ctl, kErrBadIndex);
    // The sums leave FP32 here: the compensation is applied, and the R lanes of a target
    // (partial sums over disjoint entries) are added, in FP64.
    double ax = KAHAN ? static_cast<double>(sxy.x) - cxy.x : sxy.x;
    double ay = KAHAN ? static_cast<double>(sxy.y) - cxy.y : sxy.y;
    double az = KAHAN ? static_cast<double>(sz) - cz : sz;
    for (int o = G; o < 32; o <<= 1) {
      ax += __shfl_xor_sync(0xffffffffu, ax, o);
      ay += __shfl_xor_sync(0xffffffffu, ay, o);
      az += __shfl_xor_sync(0xffffffffu, az, o);
    }
    if (valid && sl == 0) {
      const uint32_t o = b.order[k];
      b.acc[3 * (size_t)o + 0] = dmul(ax, sd.g);
      b.acc[3 * (size_t)o + 1] = dmul(ay, sd.g);
      b.acc[3 * (size_t)o + 2] = dmul(az, sd.g);
    }
    if (STATS) {
      n_leaf = warp_sum64(n_leaf);
      n_far = warp_sum64(n_far);
      n_open = warp_sum64(n_open);
      n_re = warp_sum64(n_re);
      const uint32_t n_valid = __popc(vmask);  // the root, opened by all
      if (lane == 0) {
        atomicAdd(&b.ctl->stats[0], n_leaf);
        atomicAdd(&b.ctl->stats[1], n_far);
        atomicAdd(&b.ctl->stats[2], n_open + (sd.n > 1 ? n_valid : 0u));
        atomicAdd(&b.ctl->stats[3], n_re);
        atomicAdd(&b.ctl->stats[4], n_vis);
      }
    }
    if (persistent) {
      uint32_t nxt = 0;
      if (lane == 0) nxt = atomicAdd(&b.counters[kWalkItemCounter], 1u) + warps_total;
      item = __shfl_sync(0xffffffffu, nxt, 0);
    } else {
      item = b.nitems;
    }
  }
}

namespace {

template <class K>
void launch_k(K kern, const StepBufs& b, const WalkCfg& cfg, size_t smem, cudaStream_t st) {
  const int block = cfg.block > 0 ? cfg.block : kWalkThreads;
  const int wpb = block / 32;
  const int ctas = cfg.persistent_ctas > 0 ? cfg.persistent_ctas
                   : b.nitems > static_cast<uint32_t>(cfg.auto_ctas * wpb) ? cfg.auto_ctas : 0;
  if (ctas > 0) {
    kern<<<ctas, block, smem, st>>>(b, 1);
  } else {
    const uint32_t grid = (b.nitems + wpb - 1) / wpb;
    if (grid) kern<<<grid, block, smem, st>>>(b, 0);
  }
}

template <bool QUAD, bool KAHAN, bool LIST>
void dispatch_f32(const StepBufs& b, const WalkCfg& cfg, cudaStream_t st) {
  const size_t smem = walk_smem_bytes(cfg.block > 0 ? cfg.block : kWalkThreads, QUAD);
  if (cfg.stats) {
    if (cfg.inside_test)
      launch_k(k_walk_f32<QUAD, KAHAN, true, true, LIST>, b, cfg, smem, st);
    else
      launch_k(k_walk_f32<QUAD, KAHAN, true, false, LIST>, b, cfg, smem, st);
  } else {
    if (cfg.inside_test)
      launch_k(k_walk_f32<QUAD, KAHAN, false, true, LIST>, b, cfg, smem, st);
    else
      launch_k(k_walk_f32<QUAD, KAHAN, false, false, LIST>, b, cfg, smem, st);
  }
}

template <bool LIST>
void dispatch(const StepBufs& b, const WalkCfg& cfg, cudaStream_t st) {
  if (cfg.precision == 1) {
    // The FP64 walk has no quadrupole or compensation variants: it is the
    // reference's arithmetic.
    if (cfg.stats)
      launch_k(k_walk_f64<true, LIST>, b, cfg, 0, st);
    else
      launch_k(k_walk_f64<false, LIST>, b, cfg, 0, st);
  } else if (cfg.quad) {
    if (cfg.kahan)
      dispatch_f32<true, true, LIST>(b, cfg, st);
    else
      dispatch_f32<true, false, LIST>(b, cfg, st);
  } else {
    if (cfg.kahan)
      dispatch_f32<false, true, LIST>(b, cfg, st);
    else
      dispatch_f32<false, false, LIST>(b, cfg, st);
  }
}

template <class K>
int resident(K kern, int block, size_t smem) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, block, smem) != cudaSuccess) n = 1;
  return n > 0 ? n : 1;
}

// Quadrupole blocks take more than the default 48 KB of dynamic shared memory. (No
// carveout preference is set: the driver sizes the L1 / shared split per launch, which
// leaves the L1 of the kernels that follow the walk in a step as large as they need.)
template <class K>
void smem_attrs(K kern, bool quad) {
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       static_cast<int>(walk_smem_bytes(kWalkThreads, quad)));
}

template <bool QUAD, bool KAHAN, bool LIST>
void smem_f32() {
  smem_attrs(k_walk_f32<QUAD, KAHAN, false, false, LIST>, QUAD);
  smem_attrs(k_walk_f32<QUAD, KAHAN, false, true, LIST>, QUAD);
  smem_attrs(k_walk_f32<QUAD, KAHAN, true, false, LIST>, QUAD);
  smem_attrs(k_walk_f32<QUAD, KAHAN, true, true, LIST>, QUAD);
}

}  // namespace

void walk_prepare() {
  smem_f32<false, false, false>();
  smem_f32<false, true, false>();
  smem_f32<true, false, false>();
  smem_f32<true, true, false>();
  smem_f32<false, false, true>();
  smem_f32<false, true, true>();
  smem_f32<true, false, true>();
  smem_f32<true, true, true>();
}

int walk_resident_ctas(const WalkCfg& cfg) {
  const int block = cfg.block > 0 ? cfg.block : kWalkThreads;
  if (cfg.precision == 1) return resident(k_walk_f64<false, false>, block, 0);
  if (cfg.quad) return resident(k_walk_f32<true, true, false, false, false>, block, walk_smem_bytes(block, true));
  return resident(k_walk_f32<false, true, false, false, false>, block, walk_smem_bytes(block, false));
}

void launch_walk_records64(const StepBufs& b, cudaStream_t st) {
  const int split = stream_split(b.ntiles);
  if (b.ntiles) k_walk_records64<<<b.ntiles * split, kTileThreads, 0, st>>>(b, split);
}

void launch_walk(const StepBufs& b, const WalkCfg& cfg, cudaStream_t st) {
  // A target list (active-subset walk) has its own instantiations, so the full walk's
  // code is not burdened with it.
  if (b.targets)
    dispatch<true>(b, cfg, st);
  else
    dispatch<false>(b, cfg, st);
}

}  // namespace gx
