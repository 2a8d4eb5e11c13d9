// gx_diag.cu -- FP64 O(N^2) kernels for the force oracle and the energy diagnostics.
//
// Reference: solvers/src/direct_sum.rs:25-45 (Plummer-softened pairwise sum; here
// unpaired, one thread per target, so the summation order differs and results are
// compared with a tolerance), solvers/src/potential.rs:17-58 (softened potential,
// U = -sum_{i<j} G m_i m_j / sqrt(r^2 + eps^2)), core/src/diagnostics.rs:8-68 (kinetic energy, momentum, angular
// momentum). Per-block partials are summed on the host in block order, so every
// result is deterministic. Both O(N^2) sums use FMA and an FP64 reciprocal
// square root; they are checks, compared with tolerances.
#include "gx_kernels.h"

namespace gx {

namespace {
constexpr int kDiagThreads = 256;

__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kDiagThreads / 32; ++w) t += sh[w];
  return t;
}
}  // namespace

// acc[3t] for target t = targets ? targets[t] : t. Sources staged through shared
// memory in tiles of kDiagThreads.
__global__ void __launch_bounds__(kDiagThreads) k_direct_sum_f64(uint32_t n, const double* __restrict__ pos,
                                                                const double* __restrict__ mass, double g, double eps2,
                                                                uint32_t n_targets,
                                                                const uint32_t* __restrict__ targets,
                                                                double* __restrict__ acc) {
  __shared__ double4 src[kDiagThreads];
  const uint32_t t = blockIdx.x * kDiagThreads + threadIdx.x;
  const bool valid = t < n_targets;
  const uint32_t i = valid ? (targets ? targets[t] : t) : 0u;
  double xi[3] = {0, 0, 0};
  if (valid)
    for (int c = 0; c < 3; ++c) xi[c] = pos[3 * (size_t)i + c];
  double a[3] = {0, 0, 0};
  for (uint32_t base = 0; base < n; base += kDiagThreads) {
    const uint32_t j = base + threadIdx.x;
    __syncthreads();
    if (j < n)
      src[threadIdx.x] = make_double4(pos[3 * (size_t)j], pos[3 * (size_t)j + 1], pos[3 * (size_t)j + 2], mass[j]);
    else
      src[threadIdx.x] = make_double4(0, 0, 0, 0);
    __syncthreads();
    const uint32_t cnt = min((uint32_t)kDiagThreads, n - base);
    for (uint32_t q = 0; q < cnt; ++q) {
      // the pair with itself adds nothing (massless, at unit distance)
      const bool self = base + q == i;
      const double4 s = src[q];
      const double dx = s.x - xi[0], dy = s.y - xi[1], dz = s.z - xi[2];
      const double r2 = self ? 1.0 : fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
      const double inv = rsqrt(r2);
      const double f = (self ? 0.0 : s.w) * (inv * inv * inv);
      a[0] = fma(dx, f, a[0]);
      a[1] = fma(dy, f, a[1]);
      a[2] = fma(dz, f, a[2]);
    }
  }
  if (valid)
    for (int c = 0; c < 3; ++c) acc[3 * (size_t)t + c] = a[c] * g;
}

constexpr int kPotThreads = 128;
constexpr int kPotTile = 256;  // rows and columns of a unit: two rows a thread

// The softened potential, U = -G sum_{i<j} m_i m_j / sqrt(r^2 + eps^2): units of kPotTile
// rows by kPotTile columns on and above the diagonal (half of the double sum), taken by
// the blocks in turn, so that a few thousand units of equal work keep every SM busy
// whatever N is. FP64-bound: 12 FP64 operations a pair. partial[b] = block b's sum, in a
// fixed order; the host adds the up to 2,368 partials with compensation (potential_total).
// (A thread a row over all columns, half the pairs counted twice, one block a 256 rows: a
// call at 100 / 300 / 1,000 / 65,537 / 131,072 particles in 42 / 70 / 143 / 7,430 / 25,400 us; this
// way 41 / 62 / 81 / 2,250 / 8,340. Mean error against 80-bit sums over 64 to 20,011
// particles: 1.2e-16 and 5.7e-17; 2.8e-16 with a plain sum of the partials.)
__global__ void __launch_bounds__(kPotThreads) k_potential_f64(uint32_t n, const double* __restrict__ pos,
                                                               const double* __restrict__ mass, double g, double eps2,
                                                               double* __restrict__ partial) {
  __shared__ double4 src[kPotTile];
  __shared__ double sh[kPotThreads / 32];
  const int tid = threadIdx.x;
  const unsigned long long tiles = (n + kPotTile - 1u) / kPotTile, units = tiles * (tiles + 1ull) / 2ull;
  double total = 0.0;
  // The thread's rows of a tile. The second ones go to the warps in reverse, so that on the
  // diagonal, where later rows have fewer columns, every warp has as much to do.
  const uint32_t row[2] = {static_cast<uint32_t>(tid), static_cast<uint32_t>(kPotThreads + (tid ^ (kPotThreads - 32)))};
  for (unsigned long long u = blockIdx.x; u < units; u += gridDim.x) {
    // unit u is (row tile I, column tile J) with u = J (J + 1) / 2 + I, I <= J
    unsigned long long J = static_cast<unsigned long long>((sqrt(8.0 * static_cast<double>(u) + 1.0) - 1.0) * 0.5);
    while (J * (J + 1ull) / 2ull > u) --J;
    while ((J + 1ull) * (J + 2ull) / 2ull <= u) ++J;
    const unsigned long long I = u - J * (J + 1ull) / 2ull;
    const uint32_t r0 = static_cast<uint32_t>(I) * kPotTile, c0 = static_cast<uint32_t>(J) * kPotTile;
    const uint32_t cnt = min(static_cast<uint32_t>(kPotTile), n - c0);
    double x[2], y[2], z[2], m[2], s[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t i = r0 + row[k];
      x[k] = y[k] = z[k] = m[k] = 0.0;
      if (i < n) {
        x[k] = pos[3 * (size_t)i];
        y[k] = pos[3 * (size_t)i + 1];
        z[k] = pos[3 * (size_t)i + 2];
        m[k] = mass[i];
      }
    }
    __syncthreads();  // the last unit's columns are read
    for (uint32_t q = tid; q < cnt; q += kPotThreads) {
      const size_t j = c0 + q;
      src[q] = make_double4(pos[3 * j], pos[3 * j + 1], pos[3 * j + 2], mass[j]);
    }
    __syncthreads();
    if (I != J) {
#pragma unroll 4
      for (uint32_t q = 0; q < cnt; ++q) {
        const double4 c = src[q];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const double dx = c.x - x[k], dy = c.y - y[k], dz = c.z - z[k];
          s[k] = fma(c.w, rsqrt(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)))), s[k]);
        }
      }
    } else {
      // only columns right of a row's own; the warp's other rows add nothing there (massless,
      // at unit distance), and columns left of all of them are passed over
#pragma unroll
      for (int k = 0; k < 2; ++k) {
#pragma unroll 4
        for (uint32_t q = (row[k] & ~31u) + 1u; q < cnt; ++q) {
          const double4 c = src[q];
          const double dx = c.x - x[k], dy = c.y - y[k], dz = c.z - z[k];
          const bool on = q > row[k];
          const double r2 = on ? fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))) : 1.0;
          s[k] = fma(on ? c.w : 0.0, rsqrt(r2), s[k]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (r0 + row[k] < n) total = fma(-g * m[k], s[k], total);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  if ((tid & 31) == 0) sh[tid >> 5] = total;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < kPotThreads / 32; ++w) t += sh[w];
    partial[blockIdx.x] = t;
  }
}

// partial[7 b + c]: kinetic, px, py, pz, lx, ly, lz sums over the block's particles.
__global__ void __launch_bounds__(kDiagThreads) k_diag_sums(uint32_t n, const double* __restrict__ pos,
                                                           const double* __restrict__ vel,
                                                           const double* __restrict__ mass,
                                                           double* __restrict__ partial) {
  __shared__ double sh[kDiagThreads / 32];
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  for (uint32_t i = blockIdx.x * kDiagThreads + threadIdx.x; i < n; i += gridDim.x * kDiagThreads) {
    const double m = mass[i];
    const double rx = pos[3 * (size_t)i], ry = pos[3 * (size_t)i + 1], rz = pos[3 * (size_t)i + 2];
    const double vx = vel[3 * (size_t)i], vy = vel[3 * (size_t)i + 1], vz = vel[3 * (size_t)i + 2];
    v[0] += dmul(dmul(0.5, m), dlen2(vx, vy, vz));
    v[1] += dmul(vx, m);
    v[2] += dmul(vy, m);
    v[3] += dmul(vz, m);
    v[4] += dmul(dsub(dmul(ry, vz), dmul(rz, vy)), m);
    v[5] += dmul(dsub(dmul(rz, vx), dmul(rx, vz)), m);
    v[6] += dmul(dsub(dmul(rx, vy), dmul(ry, vx)), m);
  }
  for (int c = 0; c < 7; ++c) {
    const double t = block_sum(v[c], sh);
    if (threadIdx.x == 0) partial[7 * blockIdx.x + c] = t;
  }
}

// Failure-detection self-test: lane 0 waits, through the sort look-back's bounded wait,
// for a word nothing sets; the wait runs out, raises the error word and returns.
__global__ void k_selftest_wait(const uint32_t* word, uint32_t spins, DevCtl* ctl) {
  if (threadIdx.x == 0) (void)wait_flagged(word, spins, ctl);
}

void launch_selftest_wait(const uint32_t* word, uint32_t spins, DevCtl* ctl, cudaStream_t st) {
  k_selftest_wait<<<1, 32, 0, st>>>(word, spins, ctl);
}

void launch_direct_sum_f64(uint32_t n, const double* pos, const double* mass, double g, double eps,
                           uint32_t n_targets, const uint32_t* targets, double* acc, cudaStream_t st) {
  const uint32_t grid = (n_targets + kDiagThreads - 1) / kDiagThreads;
  if (grid) k_direct_sum_f64<<<grid, kDiagThreads, 0, st>>>(n, pos, mass, g, eps * eps, n_targets, targets, acc);
}

// At most 8 partials a 256 particles (the diagnostics' buffer) and two waves of 148 SMs x 8.
uint32_t potential_partials(uint32_t n) {
  const unsigned long long t = (n + kPotTile - 1u) / kPotTile;
  const unsigned long long cap = 8ull * (n / 256u + 1u), units = t * (t + 1ull) / 2ull;
  return static_cast<uint32_t>(units < cap ? (units < 2368ull ? units : 2368ull) : (cap < 2368ull ? cap : 2368ull));
}

void launch_potential_f64(uint32_t n, const double* pos, const double* mass, double g, double eps, double* partial,
                          uint32_t n_partial, cudaStream_t st) {
  if (n_partial) k_potential_f64<<<n_partial, kPotThreads, 0, st>>>(n, pos, mass, g, eps * eps, partial);
}

void launch_diag_sums(uint32_t n, const double* pos, const double* vel, const double* mass, double* partial,
                      uint32_t n_partial, cudaStream_t st) {
  if (n_partial) k_diag_sums<<<n_partial, kDiagThreads, 0, st>>>(n, pos, vel, mass, partial);
}

}  // namespace gx
