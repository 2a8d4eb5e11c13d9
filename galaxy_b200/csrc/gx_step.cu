// gx_step.cu -- the streaming stages of a step: leapfrog kick + drift fused with the
// per-system bounding-box reduction, and the Morton-code kernel fused with the
// radix sort's up-front digit histogram.
//
// Reference: core/src/integrator.rs:59-73 (half kicks and drift),
// solvers/src/lbvh.rs:105-129 (bbox, padded cube, lane quantisation, interleave).
// All f64 arithmetic uses round-to-nearest intrinsics, so no product is fused into
// an FMA and every value rounds as the reference's Rust f64 code.
#include "gx_kernels.h"

namespace gx {

namespace {

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// CTA-wide max of 6 values (x, y, z maxima and the maxima of -x, -y, -z), then one
// atomicMax per value into the system's encoded bounds.
__device__ __forceinline__ void block_bbox_commit(double v[6], unsigned long long* enc) {
  __shared__ double red[kTileThreads / 32][6];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < 6; ++c) v[c] = warp_max(v[c]);
  if (lane == 0) {
#pragma unroll
    for (int c = 0; c < 6; ++c) red[warp][c] = v[c];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double m = red[0][threadIdx.x];
    for (int w = 1; w < kTileThreads / 32; ++w) m = fmax(m, red[w][threadIdx.x]);
    if (m == m) atomicMax(&enc[threadIdx.x], enc_max(m));  // skip empty (-inf identity) lanes
  }
}

}  // namespace

// `split` CTAs per tile. kick: apply the (deferred closing +) opening half kick and the
// drift before reducing the bounding box of the new positions.
//   pending:  v += a*h   (closing half kick of the previous step, kept separate)
//   always:   v += a*h ; x += v*dt        with h = 0.5*dt     (integrator.rs:59-67)
__global__ void __launch_bounds__(kTileThreads) k_kick_drift_bbox(const TileDesc* __restrict__ tiles,
                                                                  const SysDesc* __restrict__ sys,
                                                                  double* __restrict__ pos, double* __restrict__ vel,
                                                                  const double* __restrict__ acc, int kick,
                                                                  int pending, unsigned long long* __restrict__ enc,
                                                                  unsigned long long* __restrict__ slots, int split) {
  const TileDesc t = tile_part(tiles, split);
  const SysDesc s = sys[t.sys];
  const double dt = s.dt;
  const double h = dmul(0.5, dt);
  const bool pend = pending || (s.flags & kSysPendingKick);
  double v6[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) v6[c] = -INFINITY;
  for (uint32_t i = t.begin + threadIdx.x; i < t.end; i += kTileThreads) {
    slots[i] = kEmptySlot;  // the build's exchange words, armed here instead of by a memset
    double p[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) p[c] = pos[3 * (size_t)i + c];
    if (kick) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double a = acc[3 * (size_t)i + c];
        double v = vel[3 * (size_t)i + c];
        if (pend) v = dadd(v, dmul(a, h));
        v = dadd(v, dmul(a, h));
        p[c] = dadd(p[c], dmul(v, dt));
        vel[3 * (size_t)i + c] = v;
        pos[3 * (size_t)i + c] = p[c];
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      v6[c] = fmax(v6[c], p[c]);
      v6[3 + c] = fmax(v6[3 + c], -p[c]);
    }
  }
  block_bbox_commit(v6, enc + 6 * (size_t)t.sys);
}

// Closing half kick only (applied before a snapshot when one is pending).
__global__ void __launch_bounds__(kTileThreads) k_kick_half(const TileDesc* __restrict__ tiles,
                                                            const SysDesc* __restrict__ sys, double* __restrict__ vel,
                                                            const double* __restrict__ acc, int split) {
  const TileDesc t = tile_part(tiles, split);
  const double h = dmul(0.5, sys[t.sys].dt);
  for (uint32_t i = t.begin + threadIdx.x; i < t.end; i += kTileThreads) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
      vel[3 * (size_t)i + c] = dadd(vel[3 * (size_t)i + c], dmul(acc[3 * (size_t)i + c], h));
  }
}

// Cube of solvers/src/lbvh.rs:116-120 from the reduced lo/hi.
__device__ __forceinline__ void make_bounds(const unsigned long long* e, Bounds& b) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    b.hi[c] = dec_max(e[c]);
    b.lo[c] = -dec_max(e[3 + c]);
  }
  double ext = fmax(dsub(b.hi[0], b.lo[0]), fmax(dsub(b.hi[1], b.lo[1]), dsub(b.hi[2], b.lo[2])));
  double half = dmul(fmax(dmul(0.5, ext), 1e-12), 1.0 + 1e-9);
  double amax = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double center = dmul(dadd(b.lo[c], b.hi[c]), 0.5);
    b.bmin[c] = dsub(center, half);
    amax = fmax(amax, fmax(fabs(b.lo[c]), fabs(b.hi[c])));
  }
  b.size = dmul(2.0, half);
  b.scale = ddiv(1024.0, b.size);
  b.scale63 = ddiv(2097152.0, b.size);
  // The float-float split keeps ~2^-48 of a coordinate; below that, distance
  // comparisons are re-done in FP64.
  double t = amax * 0x1p-40;
  b.tiny2 = static_cast<float>(t * t);
}

// `split` CTAs per tile: Morton code of every particle of the tile (original order) and
// the tile's contribution to the per-system digit histograms of all radix passes
// (4 for 30-bit keys, 8 for 63-bit). The tile's system cube is rebuilt from the
// reduced lo/hi by every CTA (a few flops), and the system's first tile publishes it.
template <bool K64, int BITS>
__global__ void __launch_bounds__(kTileThreads) k_morton_hist(const TileDesc* __restrict__ tiles,
                                                              const double* __restrict__ pos,
                                                              const unsigned long long* __restrict__ enc,
                                                              const SysDesc* __restrict__ sys,
                                                              Bounds* __restrict__ bounds, uint32_t* __restrict__ codes,
                                                              uint32_t* __restrict__ lanes_out,
                                                              uint32_t* __restrict__ hist, int split) {
  step_kernel_begin();
  constexpr int BINS = 1 << BITS;
  constexpr int P = K64 ? (63 + BITS - 1) / BITS : (30 + BITS - 1) / BITS;
  __shared__ uint32_t sh[P][BINS];
  __shared__ Bounds sb;
  const TileDesc t = tile_part(tiles, split);
  for (int i = threadIdx.x; i < P * BINS; i += kTileThreads) (&sh[0][0])[i] = 0;
  if (threadIdx.x == 0) {
    make_bounds(enc + 6 * (size_t)t.sys, sb);
    if (sys[t.sys].first_tile * split == blockIdx.x) bounds[t.sys] = sb;
  }
  __syncthreads();
  const double bx = sb.bmin[0], by = sb.bmin[1], bz = sb.bmin[2];
  const double scale = K64 ? sb.scale63 : sb.scale;
  for (uint32_t i = t.begin + threadIdx.x; i < t.end; i += kTileThreads) {
    const double vx = dmul(dsub(pos[3 * (size_t)i + 0], bx), scale);
    const double vy = dmul(dsub(pos[3 * (size_t)i + 1], by), scale);
    const double vz = dmul(dsub(pos[3 * (size_t)i + 2], bz), scale);
    if (K64) {
      const uint64_t code = morton3_63(quantize_lane21(vx), quantize_lane21(vy), quantize_lane21(vz));
      reinterpret_cast<uint64_t*>(codes)[i] = code;
#pragma unroll
      for (int p = 0; p < P; ++p) atomicAdd(&sh[p][(code >> (p * BITS)) & (BINS - 1)], 1u);
    } else {
      const uint32_t lx = quantize_lane(vx), ly = quantize_lane(vy), lz = quantize_lane(vz);
      const uint32_t code = morton3(lx, ly, lz);
      codes[i] = code;
      if (lanes_out) {
        lanes_out[3 * (size_t)i + 0] = lx;
        lanes_out[3 * (size_t)i + 1] = ly;
        lanes_out[3 * (size_t)i + 2] = lz;
      }
#pragma unroll
      for (int p = 0; p < P; ++p) atomicAdd(&sh[p][(code >> (p * BITS)) & (BINS - 1)], 1u);
    }
  }
  __syncthreads();
  uint32_t* hs = hist + (size_t)t.sys * kHistWords;
  for (int i = threadIdx.x; i < P * BINS; i += kTileThreads) {
    const uint32_t c = (&sh[0][0])[i];
    if (c) atomicAdd(&hs[i], c);
  }
}

namespace {

constexpr int kSmallThreads = 1024, kSmallWarps = kSmallThreads / 32;

// Shared memory of the one-block Morton sort.
template <typename K, int ITEMS>
struct SmallSmem {
  K key[kSmallThreads * ITEMS];
  uint16_t val[kSmallThreads * ITEMS];  // local particle index
  uint32_t cnt[kSmallWarps][kRadixBins];  // digit counts, then offsets, per warp
  uint32_t part[kSmallThreads / kRadixBins][kRadixBins];
  uint32_t start[kRadixBins];
  uint32_t wsum[kRadixBins / 32];
  Bounds bounds;
};

}  // namespace

// Morton codes and the whole stable sort of one small system in one block: every digit pass
// stays in registers and shared memory, in place of the code kernel and four (eight)
// launches whose look-back, histograms and scattered writes take 7 to 10 us each whatever
// N is. Keys are ranked as in k_onesweep (a warp owns 32 ITEMS consecutive keys, peers from
// __match_any_sync), so the permutation is the same. Bound by the ranking's chain of ITEMS
// steps a pass, so it stops at a tile: kick, codes and sort together 512 particles 45 -> 24
// us, 4,096 63 -> 41 (63-bit keys 107 -> 67); 8,192 would gain nothing (62 and 59, 113 and
// 110), 16,384 lose (57 and 81).
template <typename K, int ITEMS>
__global__ void __launch_bounds__(kSmallThreads) k_small_sort(uint32_t n, const double* __restrict__ pos,
                                                              const unsigned long long* __restrict__ enc,
                                                              Bounds* __restrict__ bounds, K* __restrict__ codes,
                                                              uint32_t* __restrict__ order) {
  step_kernel_begin();
  extern __shared__ __align__(16) unsigned char s_small_raw[];
  SmallSmem<K, ITEMS>& S = *reinterpret_cast<SmallSmem<K, ITEMS>*>(s_small_raw);
  constexpr int PASSES = sizeof(K) == 8 ? kRadixPasses63 : kRadixPasses;
  constexpr int PARTS = kSmallThreads / kRadixBins;  // threads a digit
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  if (tid == 0) {
    make_bounds(enc, S.bounds);
    bounds[0] = S.bounds;
  }
  __syncthreads();
  const double bx = S.bounds.bmin[0], by = S.bounds.bmin[1], bz = S.bounds.bmin[2];
  const double scale = sizeof(K) == 8 ? S.bounds.scale63 : S.bounds.scale;
  K key[ITEMS];
  uint32_t val[ITEMS], rank[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const uint32_t i = warp * (32 * ITEMS) + 32 * j + lane;
    val[j] = i;
    key[j] = ~K(0);  // past the end: the largest digits, and last among equals
    if (i < n) {
      const double vx = dmul(dsub(pos[3 * (size_t)i + 0], bx), scale);
      const double vy = dmul(dsub(pos[3 * (size_t)i + 1], by), scale);
      const double vz = dmul(dsub(pos[3 * (size_t)i + 2], bz), scale);
      if (sizeof(K) == 8)
        key[j] = static_cast<K>(morton3_63(quantize_lane21(vx), quantize_lane21(vy), quantize_lane21(vz)));
      else
        key[j] = static_cast<K>(morton3(quantize_lane(vx), quantize_lane(vy), quantize_lane(vz)));
    }
  }
  for (int pass = 0; pass < PASSES; ++pass) {
    const int shift = pass * kRadixBits;
    for (int i = tid; i < kSmallWarps * kRadixBins; i += kSmallThreads) (&S.cnt[0][0])[i] = 0u;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const uint32_t d = static_cast<uint32_t>(key[j] >> shift) & (kRadixBins - 1);
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
      const uint32_t before = S.cnt[warp][d];
      rank[j] = before + __popc(peers & lt);
      __syncwarp();
      if (lane == 31 - __clz(peers)) S.cnt[warp][d] = before + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    // digit totals and the warps' offsets within a digit, PARTS threads a digit
    const uint32_t d = tid & (kRadixBins - 1), part = tid / kRadixBins;
    constexpr int WP = kSmallWarps / PARTS;
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < WP; ++w) {
      const uint32_t c = S.cnt[part * WP + w][d];
      S.cnt[part * WP + w][d] = sum;
      sum += c;
    }
    S.part[part][d] = sum;
    __syncthreads();
    uint32_t below = 0, incl = 0, total = 0;
    if (tid < kRadixBins) {
#pragma unroll
      for (int p = 0; p < PARTS; ++p) {
        const uint32_t c = S.part[p][d];
        S.part[p][d] = total;
        total += c;
      }
      incl = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) S.wsum[warp] = incl;
    }
    __syncthreads();
    if (tid < kRadixBins) {
      for (int w = 0; w < warp; ++w) below += S.wsum[w];
      S.start[d] = below + incl - total;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const uint32_t dj = static_cast<uint32_t>(key[j] >> shift) & (kRadixBins - 1);
      const uint32_t at = S.start[dj] + S.part[warp / WP][dj] + S.cnt[warp][dj] + rank[j];
      S.key[at] = key[j];
      S.val[at] = static_cast<uint16_t>(val[j]);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const uint32_t i = warp * (32 * ITEMS) + 32 * j + lane;
      key[j] = S.key[i];
      val[j] = S.val[i];
    }
  }
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const uint32_t i = warp * (32 * ITEMS) + 32 * j + lane;
    if (i < n) {
      codes[i] = key[j];
      order[i] = val[j];
    }
  }
}

// ---- host launchers ---------------------------------------------------------------
namespace {

template <typename K, int ITEMS>
void run_small(const StepBufs& b, cudaStream_t st) {
  launch_after(b.ntiles, k_small_sort<K, ITEMS>, 1, kSmallThreads, sizeof(SmallSmem<K, ITEMS>), st, b.n, b.pos, b.bbox_enc,
               b.bounds, reinterpret_cast<K*>(b.codes), b.order);
}

// The histogram kernel pays one merge of its bins per CTA, so it splits less than stream_split.
int hist_split(uint32_t ntiles) { return ntiles <= 37 ? 8 : ntiles <= 148 ? 4 : 1; }

}  // namespace

void launch_kick_drift_bbox(const StepBufs& b, int kick, int pending, cudaStream_t st) {
  const int split = stream_split(b.ntiles);
  k_kick_drift_bbox<<<b.ntiles * split, kTileThreads, 0, st>>>(b.tiles, b.sys, b.pos, b.vel, b.acc, kick, pending,
                                                               b.bbox_enc, b.slots, split);
}

uint32_t small_sort_max() { return kTile; }

void small_sort_prepare() {
  auto set = [](auto kern, size_t bytes) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  };
  set(k_small_sort<uint32_t, 1>, sizeof(SmallSmem<uint32_t, 1>));
  set(k_small_sort<uint32_t, 4>, sizeof(SmallSmem<uint32_t, 4>));
  set(k_small_sort<uint64_t, 1>, sizeof(SmallSmem<uint64_t, 1>));
  set(k_small_sort<uint64_t, 4>, sizeof(SmallSmem<uint64_t, 4>));
}

void launch_small_sort(const StepBufs& b, cudaStream_t st) {
  const bool one = b.n <= kSmallThreads;  // a key a thread, else four
  if (b.key64)
    one ? run_small<uint64_t, 1>(b, st) : run_small<uint64_t, 4>(b, st);
  else
    one ? run_small<uint32_t, 1>(b, st) : run_small<uint32_t, 4>(b, st);
}

void launch_kick_half(const StepBufs& b, cudaStream_t st) {
  const int split = stream_split(b.ntiles);
  k_kick_half<<<b.ntiles * split, kTileThreads, 0, st>>>(b.tiles, b.sys, b.vel, b.acc, split);
}

void launch_morton_hist(const StepBufs& b, uint32_t* lanes_out, cudaStream_t st) {
  const int split = hist_split(b.ntiles);
  auto kern = b.key64 ? k_morton_hist<true, kRadixBits>
              : b.radix_bits == kRadixBitsWide ? k_morton_hist<false, kRadixBitsWide> : k_morton_hist<false, kRadixBits>;
  launch_after(b.ntiles, kern, b.ntiles * split, kTileThreads, 0, st, b.tiles, b.pos, b.bbox_enc, b.sys, b.bounds, b.codes,
               b.key64 ? nullptr : lanes_out, b.hist, split);
}

}  // namespace gx
