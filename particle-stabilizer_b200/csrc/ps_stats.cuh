// ps_stats.cuh — per-scene statistics on the grid.
//
// Same quantities as ParticleStatisticsCUDA::calculateStatistics
// (src/ParticleStabilizerCUDA/ParticleStatisticsCUDA.cpp:11-62), whose host
// loop is O(N^2): kinetic energy sum 0.5 m |v|^2 and extents in FP64, the
// number of particles overlapping a higher-indexed particle and the largest
// overlap.  Overlapping pairs are found through the 27 neighbour cells of the
// current grid (exact, since cells are at least 2 r_max wide).  Each block
// adds its own in a fixed order, and the last one to finish adds the blocks'
// partials in a fixed order, so the result is deterministic.
//
// What bounds it: the neighbour walk's chain of loads, as in k_contacts, so
// the 18 range bounds are loaded together, and the square root and the index
// are left to pairs that may overlap.  30,011 spheres, with the rebuild of
// the grid before it: 260 us as a walk with its bounds column by column and
// one thread adding 592 partials, 95 us like this.
#pragma once

#include "ps_step_kernels.cuh"

namespace psb {

constexpr int kStatsBlocks = 592;  // 4 x 148 SMs
constexpr int kStatsThreads = 256;

struct StatsPartial {
  double ke;
  double mn[3];
  double mx[3];
  double max_overlap;
  unsigned long long collided;
  unsigned long long pad_;
};

__device__ __forceinline__ void stats_add(StatsPartial& x, const StatsPartial& y) {
  x.ke = __dadd_rn(x.ke, y.ke);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    x.mn[k] = fmin(x.mn[k], y.mn[k]);
    x.mx[k] = fmax(x.mx[k], y.mx[k]);
  }
  x.max_overlap = fmax(x.max_overlap, y.max_overlap);
  x.collided += y.collided;
}

__device__ __forceinline__ StatsPartial stats_empty() {
  StatsPartial a;
  a.ke = 0.0;
  for (int k = 0; k < 3; ++k) {
    a.mn[k] = INFINITY;
    a.mx[k] = -INFINITY;
  }
  a.max_overlap = 0.0;
  a.collided = 0;
  a.pad_ = 0;
  return a;
}

// The block's sum in its thread 0, in a fixed order.
__device__ __forceinline__ void stats_reduce(StatsPartial& a, StatsPartial (&red)[kStatsThreads / 32]) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    StatsPartial o;
    o.ke = __shfl_down_sync(0xffffffffu, a.ke, d);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      o.mn[k] = __shfl_down_sync(0xffffffffu, a.mn[k], d);
      o.mx[k] = __shfl_down_sync(0xffffffffu, a.mx[k], d);
    }
    o.max_overlap = __shfl_down_sync(0xffffffffu, a.max_overlap, d);
    o.collided = __shfl_down_sync(0xffffffffu, a.collided, d);
    stats_add(a, o);
  }
  if ((threadIdx.x & 31u) == 0u) red[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kStatsThreads / 32; ++w) stats_add(a, red[w]);
}

template <class T>
__global__ void __launch_bounds__(kStatsThreads) k_stats(StepBufs<T> b, SceneParams<T> sp, uint32_t first, uint32_t n,
                                                         StatsPartial* part, StatsPartial* out, uint32_t* ticket) {
  __shared__ StatsPartial red[kStatsThreads / 32];
  __shared__ bool s_last;
  pdl_wait();
  StatsPartial a = stats_empty();
  for (uint32_t t = blockIdx.x * kStatsThreads + threadIdx.x; t < n; t += gridDim.x * kStatsThreads) {
    const uint32_t i = first + t;
    const vec4_t<T> P = b.P0[i];
    const vec4_t<T> V = b.V1[i];
    const uint32_t oi = b.orig[i];
    int32_t cx, cy, cz;
    (void)cell_of<T>(P.x, P.y, P.z, sp, cx, cy, cz);
    const int32_t nx = sp.nb[0], ny = sp.nb[1], nz = sp.nb[2];
    const uint32_t z0 = (uint32_t)(cz > 0 ? cz - 1 : 0), z1 = (uint32_t)(cz + 1 < nz ? cz + 1 : nz - 1) + 1u;
    uint32_t lo[9], hi[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const int32_t bx = cx - 1 + q / 3, by = cy - 1 + q % 3;
      const bool ok = bx >= 0 && bx < nx && by >= 0 && by < ny;
      const uint32_t col = ok ? sp.cbase + ((uint32_t)bx * (uint32_t)ny + (uint32_t)by) * (uint32_t)nz : sp.cbase;
      lo[q] = ok ? __ldg(b.offset + col + z0) : 0u;
      hi[q] = ok ? __ldg(b.offset + col + z1) : 0u;
    }
    const double vx = (double)V.x, vy = (double)V.y, vz = (double)V.z, m = (double)V.w;
    // 0.5 * m * (vx*vx + vy*vy + vz*vz)
    const double v2 = __dadd_rn(__dadd_rn(__dmul_rn(vx, vx), __dmul_rn(vy, vy)), __dmul_rn(vz, vz));
    a.ke = __dadd_rn(a.ke, __dmul_rn(__dmul_rn(0.5, m), v2));
    const double x[3] = {(double)P.x, (double)P.y, (double)P.z}, r = (double)P.w;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      a.mn[k] = fmin(a.mn[k], __dsub_rn(x[k], r));
      a.mx[k] = fmax(a.mx[k], __dadd_rn(x[k], r));
    }
    bool hit = false;
#pragma unroll
    for (int q = 0; q < 9; ++q)
      for (uint32_t j = lo[q]; j < hi[q]; ++j) {
        const vec4_t<T> Q = ld4<T>(b.P0 + j);
        const double dx = __dsub_rn(x[0], (double)Q.x), dy = __dsub_rn(x[1], (double)Q.y),
                     dz = __dsub_rn(x[2], (double)Q.z);
        const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        const double s = __dadd_rn(r, (double)Q.w);
        // no overlap without the square root: d2 above s * s by more than its rounding
        if (d2 >= __dmul_rn(__dmul_rn(s, s), 1.0 + 1e-12)) continue;
        if (__ldg(b.orig + j) <= oi) continue;
        const double ov = __dsub_rn(s, __dsqrt_rn(d2));
        if (ov > 0.0) {
          hit = true;
          a.max_overlap = fmax(a.max_overlap, ov);
        }
      }
    a.collided += hit ? 1ull : 0ull;
  }
  stats_reduce(a, red);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = a;
    __threadfence();
    s_last = atomicAdd(ticket, 1u) == gridDim.x - 1u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  a = stats_empty();
  for (uint32_t k = threadIdx.x; k < gridDim.x; k += kStatsThreads) stats_add(a, part[k]);
  __syncthreads();  // the reduction's shared words are used again
  stats_reduce(a, red);
  if (threadIdx.x == 0) {
    *out = a;
    *ticket = 0u;
  }
}

}  // namespace psb
