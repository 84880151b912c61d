// ps_run.cuh — many steps in one launch: the default path of calls of
// RUN_MIN_STEPS steps and more.
//
// The step kernels rebuild the grid from nothing in every step, although a
// sphere moves about a ten-thousandth of a cell per step.  k_run is one
// cooperative kernel, one wave of CTAs, that advances the scenes by a whole
// block of steps and rebuilds only when the motion since the last rebuild
// requires it.  Between rebuilds the state stays in the order of the last
// one, in two alternating buffers, and each sphere walks a short list of
// neighbours; a step is then one phase and one grid barrier.
//
// Exactness.  The states are those of the step kernels bit for bit.
//   * Lists hold every pair closer than r_i + r_j + skin at the build.  D
//     adds up, step by step, the largest displacement of any sphere (in
//     cells of its scene); while D <= 0.49 skin no pair outside a list can
//     overlap.  Past that the grid and the lists are rebuilt before the step.
//   * A sphere's overlapping pairs are applied in ascending (cell at this
//     step, original index) order, the order of the 27-cell walk.  A list is
//     in that order at the build and stays so until a sphere leaves the cell
//     it was in then.  A sphere that has left carries the sign bit of its
//     radius word, so its neighbours see it with its position; a pair with
//     such a sphere, or whose cells were not adjacent at the build, sends
//     the receiving sphere to run_slow, which forms every key from the
//     positions and also tests that the cells are adjacent, as the walk does.
//   * Only a sphere that was within skin / 2 of one of its cell's faces at
//     the build can leave it; a bit of its count word says so, and the other
//     spheres do not compute a cell at all.
//   * A sphere with more than the list's capacity of neighbours walks the
//     cells of the last build instead (run_slow); where such spheres are too
//     many for that, the launch goes on without lists (RUN_CROWD).
//   * In a triangle container a build also lists the triangles that a sphere
//     may come to touch; one that moves a good part of the skin at once walks
//     its bin.
//
// When the fastest sphere moves more than RUN_CALM_MAX cells in a step, or
// did within the last RUN_CALM_STEPS steps, no list would last two steps,
// below which it does not pay: such a step rebuilds the grid and walks the 27
// cells, like the step kernels.  The skin of a build follows from the speed,
// so that a build lasts about RUN_STEPS_PER_BUILD steps.
//
// ps_set_neighbor_lists sets the skin and the lists' capacity of the same
// kernel, for every build.
//
// What bounds it: a list step moves 66 B per sphere in FP32 (position and
// velocity in and out, one 2-byte count), mostly through L2 up to a million
// spheres; what remains is the chain count -> list entry -> position ->
// velocity of the touching pairs and the barrier (about 1.5 us).
#pragma once

#include "ps_step_kernels.cuh"

namespace psb {

constexpr int RUN_MIN_STEPS = 8;
constexpr uint32_t RUN_LIST_CAP = 32;
constexpr float RUN_CALM_MAX = 0.05f;
constexpr uint32_t RUN_CALM_STEPS = 2;
constexpr float RUN_STEPS_PER_BUILD = 64.0f;
constexpr float RUN_SKIN_MIN = 0.02f, RUN_SKIN_MAX = 0.25f, RUN_SKIN_FIRST = 0.06f;

// count word of a sphere: list length and what its step needs besides
enum : uint32_t {
  RUN_COUNT = 0xffu,
  RUN_NEAR_FACE = 1u << 8,  // may leave its cell before the next build
  RUN_OVERFLOW = 1u << 9,   // more neighbours than the list holds
  RUN_TRIS = 10,            // shift: triangles that may come within reach, RUN_TRI_MANY if not all are listed
};
constexpr int RUN_TRI_CAP = 16;
constexpr uint32_t RUN_TRI_MANY = RUN_TRI_CAP + 1;
constexpr uint32_t RUN_FAR_CELL = 0x80000000u;  // list entry: cells not adjacent at the build
constexpr uint32_t RUN_LIST_CAP_MAX = RUN_COUNT;  // list capacity that a program may ask for

// control words
enum : int {
  RUN_BAR = 0,      // grid barrier of even launches: arrivals so far (64 bits)
  RUN_MAXD = 2,     // largest squared displacement of a step, in cells (3 words, by step)
  RUN_STREAK = 5,   // calm steps up to now
  RUN_RMAX = 6,     // largest radius, in cells of its scene
  RUN_BEFORE = 7,   // largest displacement of the last step, in cells (0: none yet)
  RUN_FULL = 8,     // a sphere had more neighbours than a list holds
  RUN_BUILDS = 9,   // builds after a run's first
  RUN_REPORT = 10,  // (2 words) the report of runs that choose no path: recorded ones, and those with a set skin
  RUN_BAR_ODD = 12, // grid barrier of odd launches
  RUN_LEFT = 14,    // CTAs that left because a barrier gave up
  RUN_CROWD = 16,   // spheres beyond their lists at the last build: 0 none, 1 some, 2 too many of some CTA
};

template <class T>
struct RunBufs {
  vec4_t<T>* P[2];
  vec4_t<T>* V[2];
  uint32_t* list;       // [k][slot]
  uint16_t* cnt;
  uint32_t* tris;       // [k][slot]: triangles within reach (triangle containers)
  uint32_t* later;      // per CTA: the slots of its RunLate beyond what fits in shared memory
  uint32_t* ctl;
  uint32_t *bar, *bar_next;  // grid barrier of this launch, and of the next one on these control words
  // recording for the backward pass (null otherwise): rows of the tape, one
  // list and count array per build (max_builds of them), the build of every
  // step, and after them 1 when the run is complete
  char* tape;
  size_t tape_row_bytes;
  uint32_t* tape_build;
  uint32_t max_builds;
  uint32_t* report;     // number of the last run, and whether it rebuilt too often
  uint32_t cap;
  float skin;           // skin of every build, as a fraction of the cell edge; 0: from the speed
  uint32_t later_stride;  // entries of `later` per CTA
  __device__ __forceinline__ vec4_t<T>* p(int k) const { return k ? P[1] : P[0]; }
  __device__ __forceinline__ vec4_t<T>* v(int k) const { return k ? V[1] : V[0]; }
  // list and count words of build `build` (one only unless recording)
  template <bool TAPE>
  __device__ __forceinline__ uint32_t* lists(uint32_t build, uint32_t n) const {
    return TAPE ? list + (size_t)build * cap * n : list;
  }
  template <bool TAPE>
  __device__ __forceinline__ uint16_t* counts(uint32_t build, uint32_t n) const {
    return TAPE ? cnt + (size_t)build * n : cnt;
  }
};

// One phase's end for the whole grid.  Arrivals only ever count up, by
// gridDim per barrier, so nothing is reset between the barriers of a launch.
// A launch's count starts at zero whatever the grid of the one before it and
// however that ended: two words take turns, and a launch clears the other one.
// Every wait is bounded: a CTA that gives up records PS_DEVERR_LIST_BARRIER
// and leaves the kernel, and no later barrier can then complete.  The limit
// is about a minute, because one phase of a diverged scene (spheres crowded
// into one cell) may take long.  What was queued behind such a launch stays
// inside its arrays: later runs see the bit and return at once, and the last
// CTA to leave clears the counts that the step kernels start from (run_leave).
// The host clears the bit and the control words with its report.
constexpr uint32_t RUN_BARRIER_SPIN_LIMIT = 1u << 26;

__device__ __forceinline__ bool run_barrier(uint32_t* word, uint32_t* err) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(word);
    unsigned long long seen;
    asm volatile("fence.acq_rel.gpu;" ::: "memory");  // the CTA's writes, gathered by the barrier above
    asm volatile("atom.add.release.gpu.global.u64 %0, [%1], 1;" : "=l"(seen) : "l"(bar) : "memory");
    const unsigned long long target = (seen / gridDim.x + 1ull) * gridDim.x;
    ++seen;
    for (uint32_t spins = 0; seen < target; ++spins) {
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(bar) : "memory");
      if (spins == RUN_BARRIER_SPIN_LIMIT) {
        atomicOr(err, PS_DEVERR_LIST_BARRIER);
        ok = 0;
        break;
      }
      if (spins >= 64u) __nanosleep(64);
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

template <class T>
__device__ __noinline__ void run_leave(const StepBufs<T>& b, uint32_t* ctl) {
  __shared__ bool s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(ctl + RUN_LEFT, 1u) + 1u == gridDim.x;
  }
  __syncthreads();
  if (!s_last) return;  // (a CTA that passed the last barrier has no counts to clear)
  __threadfence();
  for (uint32_t c = threadIdx.x; c < b.n_scan; c += STEP_THREADS) b.count[c] = 0u;
  for (uint32_t t = threadIdx.x; t < b.n_tiles; t += STEP_THREADS) b.tile_sum[t] = 0u;
}

template <class T>
__device__ __forceinline__ bool marked(T w) {
  return signbit(w);
}

// Squared displacement of a sphere in cells of its scene; infinite when it
// is finite now and the distance is not, zero when it is not finite now (it
// then touches nothing).
template <class T>
__device__ __forceinline__ float moved2(const vec4_t<T>& P, const vec4_t<T>& old, T inv2) {
  const T ex = P.x - old.x, ey = P.y - old.y, ez = P.z - old.z;
  const float m = (float)((ex * ex + ey * ey + ez * ez) * inv2);
  if (m <= 3.0e38f) return m;
  return isfinite(P.x) && isfinite(P.y) && isfinite(P.z) ? INFINITY : 0.0f;
}

// cell_of without its divisions where the cell is beyond doubt: a point more
// than a thousandth of a cell from every cell face, which covers the rounding
// of both up to 4,096 cells on an axis.
template <class T>
__device__ __forceinline__ uint32_t run_cell_of(const vec4_t<T>& P, const SceneParams<T>& sp) {
  const T qx = (P.x - sp.grid_lo[0]) * sp.inv_interval, qy = (P.y - sp.grid_lo[1]) * sp.inv_interval,
          qz = (P.z - sp.grid_lo[2]) * sp.inv_interval;
  const T fx = floor(qx), fy = floor(qy), fz = floor(qz);
  const T lo = T(1e-3), hi = T(1) - T(1e-3), far = T(4096);
  const T rx = qx - fx, ry = qy - fy, rz = qz - fz;
  if (rx > lo && rx < hi && ry > lo && ry < hi && rz > lo && rz < hi && fabs(qx) < far && fabs(qy) < far &&
      fabs(qz) < far) {
    const int32_t cx = min(max((int32_t)fx, 0), sp.nb[0] - 1), cy = min(max((int32_t)fy, 0), sp.nb[1] - 1),
                  cz = min(max((int32_t)fz, 0), sp.nb[2] - 1);
    return sp.cbase + ((uint32_t)cx * (uint32_t)sp.nb[1] + (uint32_t)cy) * (uint32_t)sp.nb[2] + (uint32_t)cz;
  }
  int32_t cx, cy, cz;
  return cell_of<T>(P.x, P.y, P.z, sp, cx, cy, cz);
}

// Largest displacement of the CTA's spheres into the step's word (squares
// are not negative, so their bit patterns order like the values).
__device__ __forceinline__ void publish_max(float m, uint32_t* word) {
  __shared__ uint32_t s_max[STEP_THREADS / 32];
  const uint32_t w = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  if ((threadIdx.x & 31u) == 0u) s_max[threadIdx.x >> 5] = w;
  __syncthreads();
  if (threadIdx.x < 32u) {
    const uint32_t v = __reduce_max_sync(0xffffffffu, threadIdx.x < STEP_THREADS / 32 ? s_max[threadIdx.x] : 0u);
    if (threadIdx.x == 0u && v != 0u) atomicMax(word, v);
  }
}

// Slot ranges of the 27-cell walk around cell (cx, cy, cz), read coherently.
template <class T>
__device__ __forceinline__ void cell_ranges(const StepBufs<T>& b, const SceneParams<T>& sp, bool live, int32_t cx,
                                            int32_t cy, int32_t cz, uint32_t (&lo)[9], uint32_t (&hi)[9]) {
  const int32_t nx = sp.nb[0], ny = sp.nb[1], nz = sp.nb[2];
  const uint32_t z0 = (uint32_t)(cz > 0 ? cz - 1 : 0);
  const uint32_t z1 = (uint32_t)(cz + 1 < nz ? cz + 1 : nz - 1) + 1u;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    const int32_t bx = cx - 1 + q / 3, by = cy - 1 + q % 3;
    const bool ok = live && bx >= 0 && bx < nx && by >= 0 && by < ny;
    const uint32_t col = ok ? sp.cbase + ((uint32_t)bx * (uint32_t)ny + (uint32_t)by) * (uint32_t)nz : sp.cbase;
    const bool inb = ok && in_bounds(col + z1, b.n_scan, b.err);
    lo[q] = inb ? b.offset[col + z0] : 0u;
    hi[q] = inb ? b.offset[col + z1] : 0u;
    if (!in_bounds(hi[q], b.n + 1u, b.err)) hi[q] = lo[q] = 0u;
  }
}

// Cells [c0, c1] of one axis that can hold a point within `reach` of x.
// The hash is monotonic in x, so the cells of x - reach and x + reach bound
// them; the pad covers the rounding of x +- reach, by eight units of the last
// place (far from the origin a pad of FP32's size took FP64 scenes into cells
// whose spheres are out of reach: 60,000 spheres 1e6 from it, 2.1 ms a step
// instead of 0.13).
template <class T>
__device__ __forceinline__ void axis_span(T x, T reach, T lo, T iv, int32_t nb, int32_t& c0, int32_t& c1) {
  constexpr T ULPS = sizeof(T) == 4 ? T(1.0 / 1048576.0) : T(1.0 / 562949953421312.0);  // 2^-20, 2^-49
  const T pad = reach + (fabs(x) + fabs(lo)) * ULPS;
  c0 = axis_cell<T>(x - pad, lo, iv, nb);
  c1 = axis_cell<T>(x + pad, lo, iv, nb);
}

// Cells that can hold, at the last build, a partner of a sphere now at P.
template <class T>
struct Span {
  int32_t x0, x1, y0, y1, z0, z1;
};
template <class T>
__device__ __forceinline__ Span<T> reach_span(const vec4_t<T>& P, T reach, const SceneParams<T>& sp) {
  Span<T> s;
  axis_span<T>(P.x, reach, sp.grid_lo[0], sp.interval, sp.nb[0], s.x0, s.x1);
  axis_span<T>(P.y, reach, sp.grid_lo[1], sp.interval, sp.nb[1], s.y0, s.y1);
  axis_span<T>(P.z, reach, sp.grid_lo[2], sp.interval, sp.nb[2], s.z0, s.z1);
  return s;
}

// Row s + 1 of the tape: sphere i's state after step s's contacts.
template <class T>
__device__ __forceinline__ void run_record(const RunBufs<T>& R, const StepBufs<T>& b, uint32_t s, uint32_t i,
                                           const vec4_t<T>& P, const vec4_t<T>& V, const vec4_t<T>& Vi) {
  const TapeRow<T> row = tape_row<T>(R.tape, R.tape_row_bytes, b.n, (int64_t)s + 1);
  row.p[i] = P;
  row.v[i] = V;
  row.vpre[i] = Vi;
  row.o[i] = b.orig[i];
}

// Candidates whose positions are fetched together.
template <class T>
__host__ __device__ constexpr int run_batch() {
  return sizeof(T) == 4 ? 4 : 2;
}

// What the CTA's spheres beyond their lists cost at a build (run_tell_crowd).
struct RunCrowd {
  float sum;      // of run_slow's trips
  uint32_t most;  // the most of one sphere (the bits of a float that is not negative order like it)
  uint32_t cand;  // the most candidates of one
};

// Sphere i, beyond its list, into `c` (shared): passes of run_slow over the
// columns of `s`, 32 candidates a trip, and the keys that a pass keeps.
template <class T>
__device__ __noinline__ void run_cost(uint32_t i, const StepBufs<T>& b, const SceneParams<T>& sp, const vec4_t<T>* Ps,
                                      const Span<T>& s, RunCrowd& c) {
  const vec4_t<T> P = Ps[i];
  uint32_t touch = 0, trips = 0, cand = 0;
  for (int32_t bx = s.x0; bx <= s.x1; ++bx)
    for (int32_t by = s.y0; by <= s.y1; ++by) {
      const uint32_t col = sp.cbase + ((uint32_t)bx * (uint32_t)sp.nb[1] + (uint32_t)by) * (uint32_t)sp.nb[2];
      const uint32_t j0 = b.offset[col + (uint32_t)s.z0], j1 = b.offset[col + (uint32_t)s.z1 + 1u];
      if (!in_bounds(j1, (uint64_t)b.n + 1u, b.err)) continue;
      cand += j1 - j0;
      trips += (j1 - j0 + 31u) / 32u;
      for (uint32_t j = j0; j < j1; ++j) {
        const vec4_t<T> Q = Ps[j];
        const T dx = P.x - Q.x, dy = P.y - Q.y, dz = P.z - Q.z, r = P.w + Q.w;
        touch += dx * dx + dy * dy + dz * dz < r * r ? 1u : 0u;
      }
    }
  const float cost = (1.0f + (float)(touch / 32u)) * (float)(trips + min(touch, 96u)) + 30.0f;
  atomicAdd(&c.sum, cost);
  atomicMax(&c.most, __float_as_uint(cost));
  atomicMax(&c.cand, cand);
}

// List and count word of slot i of the sorted state (positions P, sorted
// cell ids scell); columns are visited in ascending cell id, so a list is in
// ascending (cell, original index).
template <class T, bool MULTI, bool MESH, bool TAPE>
__device__ __forceinline__ void run_build_one(uint32_t i, const StepBufs<T>& b, const SceneParams<T>& sp,
                                              const MeshView* mv, const RunBufs<T>& R, const vec4_t<T>* Ps, T frac,
                                              T rmax, uint32_t build, RunCrowd& crowd) {
  uint32_t* const list = R.template lists<TAPE>(build, b.n);
  const vec4_t<T> P = Ps[i];
  const T skin = frac * sp.interval;
  uint32_t k = 0, word = 0;
  if (isfinite(P.x) && isfinite(P.y) && isfinite(P.z)) {
    int32_t cx, cy, cz;
    cell_coords<T>(b.scell[i], sp, cx, cy, cz);
    const Span<T> s = reach_span<T>(P, (P.w + rmax * sp.interval + skin) * T(1.001), sp);
    const uint32_t ny = (uint32_t)sp.nb[1], nz = (uint32_t)sp.nb[2];
    // cells more than one away are in reach: their spheres are marked
    const bool wide = s.x0 < cx - 1 || s.x1 > cx + 1 || s.y0 < cy - 1 || s.y1 > cy + 1 || s.z0 < cz - 1 || s.z1 > cz + 1;
    auto take = [&](uint32_t j, const vec4_t<T>& Q) {
      const T dx = P.x - Q.x, dy = P.y - Q.y, dz = P.z - Q.z;
      const T cut = (P.w + Q.w + skin) * T(1.0001);
      if (dx * dx + dy * dy + dz * dz < cut * cut && j != i) {
        if (k < R.cap) {
          uint32_t entry = j;
          if (wide) {
            int32_t jx, jy, jz;
            cell_coords<T>(b.scell[j], sp, jx, jy, jz);
            if (abs(jx - cx) > 1 || abs(jy - cy) > 1 || abs(jz - cz) > 1) entry |= RUN_FAR_CELL;
          }
          list[(size_t)k * b.n + i] = entry;
        }
        ++k;
      }
    };
    // a row of columns at a time, their range bounds loaded together, and
    // candidates a few at a time, all ahead of the list's stores
    constexpr int COLS = 4, NB = run_batch<T>();
    for (int32_t bx = s.x0; bx <= s.x1; ++bx)
      for (int32_t y0 = s.y0; y0 <= s.y1; y0 += COLS) {
        uint32_t lo[COLS], hi[COLS];
#pragma unroll
        for (int q = 0; q < COLS; ++q) {
          const bool ok = y0 + q <= s.y1;
          const uint32_t col = sp.cbase + ((uint32_t)bx * ny + (uint32_t)(ok ? y0 + q : y0)) * nz;
          lo[q] = ok ? b.offset[col + (uint32_t)s.z0] : 0u;
          hi[q] = ok ? b.offset[col + (uint32_t)s.z1 + 1u] : 0u;
          if (!in_bounds(hi[q], (uint64_t)b.n + 1u, b.err)) hi[q] = lo[q] = 0u;
        }
#pragma unroll
        for (int q = 0; q < COLS; ++q)
          for (uint32_t j = lo[q]; j < hi[q]; j += NB) {
            vec4_t<T> Q[NB];
#pragma unroll
            for (int u = 0; u < NB; ++u) Q[u] = Ps[j + u < hi[q] ? j + u : j];
#pragma unroll
            for (int u = 0; u < NB; ++u)
              if (j + u < hi[q]) take(j + u, Q[u]);
          }
      }
    {
      const T pad = T(0.5) * skin;
      const T *bx = b.bounds + sp.bnd_base[0] + cx, *by = b.bounds + sp.bnd_base[1] + cy,
              *bz = b.bounds + sp.bnd_base[2] + cz;
      const bool inner = P.x - __ldg(bx) > pad && __ldg(bx + 1) - P.x > pad && P.y - __ldg(by) > pad &&
                         __ldg(by + 1) - P.y > pad && P.z - __ldg(bz) > pad && __ldg(bz + 1) - P.z > pad;
      if (!inner) word |= RUN_NEAR_FACE;
    }
    if constexpr (MESH) {
      if (sp.mesh_tris > 0) {
        uint32_t ids[RUN_TRI_CAP];
        const uint32_t nt = min(mesh_candidates<T, RUN_TRI_CAP>(P, skin, sp, *mv, b.err, ids), RUN_TRI_MANY);
        for (uint32_t q = 0; q < nt && nt <= RUN_TRI_CAP; ++q) R.tris[(size_t)q * b.n + i] = ids[q];
        word |= nt << RUN_TRIS;
      }
    }
  }
  if (k > R.cap) {
    run_cost<T>(i, b, sp, Ps, reach_span<T>(P, (P.w + rmax * sp.interval + skin) * T(1.001), sp), crowd);
    word |= RUN_OVERFLOW, k = 0;
    R.ctl[RUN_FULL] = 1u;
  }
  R.template counts<TAPE>(build, b.n)[i] = (uint16_t)(word | k);
}

// A CTA's verdict on its spheres beyond their lists: too many when they would
// take longer than steps without lists.  It takes them a warp each, 0.25 us a
// trip for the warp with the most to do, against the rebuild and 0.2 us for
// every candidate of a thread's spheres.  Both are good to a factor of two (us
// a step with lists / without, and which the rule takes, FP32: 100 spheres in a
// heap among 8,000, 543 / 72, without; 400 among 200,000, 14,430 / 341,
// without; 600,000-sphere pile, lists of 1, 247 / 109, without; of 3, 68 / 103,
// with; 79,420 spheres, 3 % of them four times as large, lists of 16, 37 / 189,
// with; 20 of 83,474 ten times as large, lists of 48, 321 / 5,210, with; 3,000
// in one cell, 440 / 587, without).
__device__ __noinline__ void run_tell_crowd(const RunCrowd& c, uint32_t n, uint32_t* ctl) {
  const float cost = fmaxf(c.sum / (float)(STEP_THREADS / 32), __uint_as_float(c.most));
  const float share = (float)((n + gridDim.x * STEP_THREADS - 1u) / (gridDim.x * STEP_THREADS));
  const bool many = 0.25f * cost > 20.0f + (float)n / 12000.0f + 0.2f * (float)c.cand * share;
  atomicMax(ctl + RUN_CROWD, many ? 2u : 1u);
}

// Whether some CTA found too many; the launch then goes on without lists.  (A
// recorded run has to keep all its lists.)  It is asked before a build, when
// the word is complete.  The first step on lists does not depend on it
// (run_fresh); a CTA that sees the verdict there reports an infinite motion,
// so that the next step asks.
template <bool TAPE, class T>
__device__ __forceinline__ bool run_crowded(const RunBufs<T>& R) {
  return *reinterpret_cast<volatile uint32_t*>(R.ctl + RUN_CROWD) >= (TAPE ? 1u : 2u);
}

// Contacts of slot i in the exact order whatever has moved: the overlapping
// partners whose cell is adjacent now, by ascending (cell now, original
// index).  Every lane of the warp calls it with the same sphere.
//
// The lanes take the list's entries side by side (`mine`), each forms its
// pair's key and force, and the forces are added in the order of the keys.
// A list of more than an entry per lane, and the cells of the last build in
// place of a list that overflowed, are gone through once for every 32 pairs in
// contact: a pass keeps the 32 smallest keys above the last one, ordered by
// lane.  (A pass for every pair, as this was at first, takes the cube of the
// spheres that touch one another: 400 on top of one another among 4,000 took
// 3.8 ms a step, now 47 us; twenty spheres ten times as large as the 83,474
// others 1.89 ms, now 0.28 ms.)
template <class T>
__device__ __forceinline__ vec4_t<T> run_slow(uint32_t i, uint32_t word, uint32_t mine, const uint32_t* list,
                                              const StepBufs<T>& b, const SceneParams<T>& sp, const vec4_t<T>* Ps,
                                              const vec4_t<T>* Vs, T frac, const vec4_t<T>& P, const vec4_t<T>& Vi) {
  using A = Ar<T>;
  const unsigned lane = threadIdx.x & 31u;
  vec4_t<T> V = Vi;
  int32_t cx, cy, cz;
  cell_of<T>(P.x, P.y, P.z, sp, cx, cy, cz);
  constexpr uint64_t NONE = ~0ull;
  // key of the pair (i, j), NONE if it is not in contact; f and d of the force
  T f = T(0), dx = T(0), dy = T(0), dz = T(0);
  auto key_of = [&](uint32_t j) -> uint64_t {
    if (j == i) return NONE;
    const vec4_t<T> Q = Ps[j], W = Vs[j];  // (all three loads before the test)
    const uint32_t oj = b.orig[j];
    const T margin = T(1) + T(1.0 / 1048576.0);
    dx = A::sub(P.x, Q.x), dy = A::sub(P.y, Q.y), dz = A::sub(P.z, Q.z);
    const T d2 = A::fma(dz, dz, A::fma(dy, dy, A::mul(dx, dx)));
    const T s = A::add(fabs(P.w), fabs(Q.w));
    if (d2 >= A::mul(A::mul(s, s), margin)) return NONE;
    const T dist = A::sqrt(d2);
    const T overlap = A::sub(s, dist);
    if (!(overlap > T(0))) return NONE;
    int32_t jx, jy, jz;
    const uint32_t cj = cell_of<T>(Q.x, Q.y, Q.z, sp, jx, jy, jz);
    if (abs(jx - cx) > 1 || abs(jy - cy) > 1 || abs(jz - cz) > 1) return NONE;
    f = contact_force<T>(Vi, W, dx, dy, dz, d2, dist, overlap, sp.k_spring, sp.e_sphere);
    return ((uint64_t)cj << 32) | (uint64_t)oj;
  };
  auto smallest = [&](uint64_t key) -> uint64_t {
    const uint32_t cell = (uint32_t)(key >> 32);
    const uint32_t c = __reduce_min_sync(0xffffffffu, cell);
    const uint32_t o = __reduce_min_sync(0xffffffffu, cell == c ? (uint32_t)key : 0xffffffffu);
    return ((uint64_t)c << 32) | (uint64_t)o;
  };
  auto apply = [&](int from) {
    const T g = __shfl_sync(0xffffffffu, f, from);
    V.x = A::fma(g, __shfl_sync(0xffffffffu, dx, from), V.x);
    V.y = A::fma(g, __shfl_sync(0xffffffffu, dy, from), V.y);
    V.z = A::fma(g, __shfl_sync(0xffffffffu, dz, from), V.z);
  };
  const uint32_t nl = word & RUN_COUNT;
  if (!(word & RUN_OVERFLOW) && nl <= 32u) {
    uint64_t key = lane < nl ? key_of(mine) : NONE;
    for (uint64_t best = smallest(key); best != NONE; best = smallest(key)) {
      apply(__ffs(__ballot_sync(0xffffffffu, key == best)) - 1);
      if (key == best) key = NONE;
    }
    return V;
  }
  const T skin = frac * sp.interval;
  const Span<T> s = reach_span<T>(P, (fabs(P.w) + T(0.5) * sp.interval + T(2) * skin) * T(1.001), sp);
  for (uint64_t from = 0;;) {
    uint64_t kept = NONE;  // ascending by lane
    uint32_t kept_j = i;
    auto offer = [&](uint64_t key, uint32_t j) {
      const uint64_t most = __shfl_sync(0xffffffffu, kept, 31);
      for (uint32_t who = __ballot_sync(0xffffffffu, key >= from && key < most); who != 0u; who &= who - 1u) {
        const int l = __ffs(who) - 1;
        const uint64_t k = __shfl_sync(0xffffffffu, key, l), below = __shfl_up_sync(0xffffffffu, kept, 1);
        const uint32_t kj = __shfl_sync(0xffffffffu, j, l), below_j = __shfl_up_sync(0xffffffffu, kept_j, 1);
        if (kept > k) {
          const bool here = lane == 0u || below < k;
          kept = here ? k : below;
          kept_j = here ? kj : below_j;
        }
      }
    };
    if (word & RUN_OVERFLOW) {
      for (int32_t bx = s.x0; bx <= s.x1; ++bx)
        for (int32_t by = s.y0; by <= s.y1; ++by) {
          const uint32_t col = sp.cbase + ((uint32_t)bx * (uint32_t)sp.nb[1] + (uint32_t)by) * (uint32_t)sp.nb[2];
          const uint32_t j1 = b.offset[col + (uint32_t)s.z1 + 1u];
          if (!in_bounds(j1, (uint64_t)b.n + 1u, b.err)) continue;
          for (uint32_t j0 = b.offset[col + (uint32_t)s.z0]; j0 < j1; j0 += 32u) {
            const uint32_t j = j0 + lane;
            offer(j < j1 ? key_of(j) : NONE, j);
          }
        }
    } else {
      for (uint32_t k0 = 0; k0 < nl; k0 += 32u) {
        const uint32_t j = k0 + lane < nl ? list[(size_t)(k0 + lane) * b.n + i] & ~RUN_FAR_CELL : i;
        offer(in_bounds(j, b.n, b.err) ? key_of(j) : NONE, j);
      }
    }
    if (kept != NONE) (void)key_of(kept_j);  // the force of the lane's pair
    const int pairs = __popc(__ballot_sync(0xffffffffu, kept != NONE));
    for (int l = 0; l < pairs; ++l) apply(l);
    if (pairs < 32) return V;
    from = __shfl_sync(0xffffffffu, kept, 31) + 1u;
  }
}

// The phases that few steps take are functions of their own, so that the
// registers of the list step are its own.

// The first integration, from the at-rest state (P0, V1) into buffer 1; the
// cells are counted on the way.
template <class T, bool MULTI, bool MESH>
__device__ __noinline__ void run_begin(const StepBufs<T>& b, const SceneParams<T>& sp0, const MeshView* mv,
                                       const RunBufs<T>& R) {
  float m = 0.0f, rmax = 0.0f;
  for (uint32_t base = blockIdx.x * STEP_THREADS; base < b.n; base += gridDim.x * STEP_THREADS) {
    const uint32_t i = base + threadIdx.x;
    const bool valid = i < b.n;
    uint32_t c = 0;
    if (valid) {
      const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
      vec4_t<T> P = R.P[0][i], V = R.V[1][i];
      P.w = fabs(P.w);
      rmax = fmaxf(rmax, (float)(P.w / sp.interval));
      const vec4_t<T> old = P;
      integrate<T>(P, V, sp);
      finish_integrated<T, MESH>(P, V, sp, mv, b.err, c);
      m = fmaxf(m, moved2<T>(P, old, sp.inv_interval2));
      R.P[1][i] = P;
      R.V[1][i] = V;
      b.cell[i] = c;
    }
    count_cell(b.count, b.tile_sum, c, valid && in_bounds(c, b.n_scan - 1u, b.err), b.tile_shift);
  }
  publish_max(m, R.ctl + RUN_MAXD);
  __syncthreads();  // the reduction's shared words are used again
  publish_max(rmax, R.ctl + RUN_RMAX);
}

// Grid of the state in buffer `cur`, sorted into the other one, and with
// frac > 0 its lists.  False: a barrier gave up.
template <class T, bool MULTI, bool MESH, bool TAPE>
__device__ __noinline__ bool run_rebuild(const StepBufs<T>& b, const SceneParams<T>& sp0, const MeshView* mv,
                                         const RunBufs<T>& R, int cur, bool counted, float frac, uint32_t build,
                                         int64_t n_cells, uint32_t scatter_blocks, uint32_t move_blocks) {
  const uint32_t stride = gridDim.x * STEP_THREADS;
  if (!counted) {
    vec4_t<T>* Ps = R.p(cur);
    for (uint32_t base = blockIdx.x * STEP_THREADS; base < b.n; base += stride) {
      const uint32_t i = base + threadIdx.x;
      const bool valid = i < b.n;
      uint32_t c = 0;
      if (valid) {
        const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
        const vec4_t<T> P = Ps[i];
        int32_t cx, cy, cz;
        c = cell_of<T>(P.x, P.y, P.z, sp, cx, cy, cz);
        if (marked<T>(P.w)) Ps[i].w = fabs(P.w);
        b.cell[i] = c;
      }
      count_cell(b.count, b.tile_sum, c, valid && in_bounds(c, b.n_scan - 1u, b.err), b.tile_shift);
    }
    if (!run_barrier(R.bar, b.err)) return false;
  }
  for (uint32_t t = blockIdx.x; t < b.n_tiles; t += gridDim.x) {
    __syncthreads();  // the tile scan reuses its shared arrays
    if (b.tile_shift == 13u)
      scan_tile_with_sums<true, STEP_SCAN_ITEMS_LARGE>(t, b.count, b.offset, n_cells, b.tile_sum);
    else
      scan_tile_with_sums<true, STEP_SCAN_ITEMS_SMALL>(t, b.count, b.offset, n_cells, b.tile_sum);
  }
  if (!run_barrier(R.bar, b.err)) return false;
  // (behind a barrier that every CTA came to after it read the word)
  if (frac > 0.0f && blockIdx.x == 0 && threadIdx.x == 0) R.ctl[RUN_CROWD] = 0u;
  for (uint32_t blk = blockIdx.x; blk < scatter_blocks; blk += gridDim.x)
    scatter_block<true>(blk, b.cell, b.slot, b.orig, b.offset, b.tmp, b.count, b.n, b.tile_sum, b.n_tiles, b.err);
  if (!run_barrier(R.bar, b.err)) return false;
  StepBufs<T> mb = b;
  mb.P1 = R.p(cur);
  mb.V1 = R.v(cur);
  mb.P0 = R.p(1 - cur);
  mb.V0 = R.v(1 - cur);
  for (uint32_t blk = blockIdx.x; blk < move_blocks; blk += gridDim.x) rank_move_block<T, true>(blk, mb);
  if (!run_barrier(R.bar, b.err)) return false;
  if (frac > 0.0f) {
    const vec4_t<T>* Ps = R.p(1 - cur);
    const T rmax = (T)__uint_as_float(R.ctl[RUN_RMAX]) * T(1.0001);
    __shared__ RunCrowd crowd;
    if (threadIdx.x == 0) crowd = {0.0f, 0u, 0u};
    __syncthreads();
    for (uint32_t i = blockIdx.x * STEP_THREADS + threadIdx.x; i < b.n; i += stride)
      run_build_one<T, MULTI, MESH, TAPE>(i, b, scene_of<T, MULTI>(i, sp0, b), mv, R, Ps, (T)frac, rmax, build, crowd);
    __syncthreads();
    if (threadIdx.x == 0 && crowd.cand != 0u) run_tell_crowd(crowd, b.n, R.ctl);
  }
  return true;
}

// One step without lists on a grid built for it; the next step's cells are
// counted on the way.  Returns the thread's largest squared displacement.
template <class T, bool MULTI, bool MESH>
__device__ __noinline__ float run_grid_step(const StepBufs<T>& b, const SceneParams<T>& sp0, const MeshView* mv,
                                            const RunBufs<T>& R, int cur, bool last) {
  const vec4_t<T>* Ps = R.p(cur);
  const vec4_t<T>* Vs = R.v(cur);
  vec4_t<T>* Pd = R.p(1 - cur);
  vec4_t<T>* Vd = R.v(1 - cur);
  float m = 0.0f;
  for (uint32_t base = blockIdx.x * STEP_THREADS; base < b.n; base += gridDim.x * STEP_THREADS) {
    const uint32_t i = base + threadIdx.x;
    const bool valid = i < b.n;
    uint32_t c = 0;
    if (valid) {
      const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
      vec4_t<T> P = Ps[i];
      const vec4_t<T> Vi = Vs[i];
      vec4_t<T> V = Vi;
      const bool live = isfinite(P.x) && isfinite(P.y) && isfinite(P.z);
      int32_t cx, cy, cz;
      cell_coords<T>(b.scell[i], sp, cx, cy, cz);
      uint32_t lo[9], hi[9];
      cell_ranges<T>(b, sp, live, cx, cy, cz, lo, hi);
#pragma unroll
      for (int q = 0; q < 9; ++q)
        for (uint32_t j = lo[q]; j < hi[q]; ++j) {
          if (q == 4 && j == i) continue;
          contact_one<T, true>(Vs, j, P, Vi, Ps[j], sp.k_spring, sp.e_sphere, V.x, V.y, V.z);
        }
      if (!last) {
        const vec4_t<T> old = P;
        integrate<T>(P, V, sp);
        if constexpr (MESH) {
          if (sp.mesh_tris > 0)
            mesh_contacts<T>(P, V, sp, *mv, b.err);
          else
            walls<T>(P, V, sp);
        } else {
          walls<T>(P, V, sp);
        }
        m = fmaxf(m, moved2<T>(P, old, sp.inv_interval2));
        c = cell_near<T>(P.x, P.y, P.z, sp, b.bounds, cx, cy, cz);
        b.cell[i] = c;
      }
      Pd[i] = P;
      Vd[i] = V;
    }
    if (!last) count_cell(b.count, b.tile_sum, c, valid && in_bounds(c, b.n_scan - 1u, b.err), b.tile_shift);
  }
  return m;
}

// The end of a sphere's step after the container: its displacement from
// `old`, and the mark of a sphere outside its cell of the build, which
// cell_then() gives (few spheres ask).  DIVIDE: by cell_of, whose chain of
// instructions is the shorter one where nothing else hides it (4,096 spheres:
// 3.8 against 4.2 us a step); else by run_cell_of, which takes fewer (1M
// pile, FP32: 42.0 against 43.6 us).
template <class T, bool DIVIDE, class F>
__device__ __forceinline__ void run_finish(vec4_t<T>& P, F cell_then, uint32_t word, const SceneParams<T>& sp,
                                           const vec4_t<T>& old, float& m) {
  m = fmaxf(m, moved2<T>(P, old, sp.inv_interval2));
  if (word & RUN_NEAR_FACE) {
    uint32_t now;
    if constexpr (DIVIDE) {
      int32_t cx, cy, cz;
      now = cell_of<T>(P.x, P.y, P.z, sp, cx, cy, cz);
    } else {
      now = run_cell_of<T>(P, sp);
    }
    if (now != cell_then()) P.w = -P.w;
  }
}

// Whether an integrated sphere has to test triangles: some may be within
// reach since the build, or it moves a good part of the skin at once.
template <class T>
__device__ __forceinline__ bool run_near_mesh(const vec4_t<T>& P, const vec4_t<T>& old, uint32_t word, T skin) {
  const T lim = T(0.25) * skin;
  const T ex = P.x - old.x, ey = P.y - old.y, ez = P.z - old.z;
  return (word >> RUN_TRIS) != 0u || !(ex * ex + ey * ey + ez * ez <= lim * lim);
}

// Spheres that a CTA's list step puts aside, their chains of loads being
// long: taken inline by their own thread, a handful of them held the whole
// step up (30,011-sphere pile: 7.2 us a step without any, 14.5 us with forty).
constexpr uint32_t RUN_LATE_HERE = 256;
struct RunLate {
  uint32_t n_slow, n_near;
  uint32_t slow[RUN_LATE_HERE];  // need run_slow's order
  uint32_t near[RUN_LATE_HERE];  // need their triangles (contacts and integration done)
};

template <class T>
__device__ __forceinline__ void run_put_aside(RunLate& l, const RunBufs<T>& R, uint32_t i, bool slow) {
  const uint32_t k = atomicAdd(slow ? &l.n_slow : &l.n_near, 1u);
  uint32_t* const here = slow ? l.slow : l.near;
  uint32_t* const there = R.later + (size_t)blockIdx.x * R.later_stride;
  if (k < RUN_LATE_HERE)
    here[k] = i;
  else  // one kind from the front, the other from the back
    there[slow ? k : R.later_stride - 1u - k] = i;
}
template <class T>
__device__ __forceinline__ uint32_t run_put(const RunLate& l, const RunBufs<T>& R, uint32_t k, bool slow) {
  const uint32_t* there = R.later + (size_t)blockIdx.x * R.later_stride;
  return k < RUN_LATE_HERE ? (slow ? l.slow[k] : l.near[k]) : there[slow ? k : R.later_stride - 1u - k];
}

// Triangle container of a sphere from the triangles listed at the build, by
// half a warp: the lanes test a triangle each, and the hits, which come in
// ascending index, are added in turn.  The other half may have another
// sphere (or none: nt = 0).
template <class T>
__device__ __forceinline__ void run_mesh_half(vec4_t<T>& P, vec4_t<T>& V, uint32_t nt, uint32_t t, const StepBufs<T>& b,
                                              const SceneParams<T>& sp, const MeshView& mv) {
  using A = Ar<T>;
  static_assert(RUN_TRI_CAP == 16, "a triangle per lane of half a warp");
  const unsigned sub = threadIdx.x & 15u;
  const T r = P.w;
  const V3<T> c = {P.x, P.y, P.z};
  const V3<T> lo = {A::sub(c.x, r), A::sub(c.y, r), A::sub(c.z, r)};
  const V3<T> hi = {A::add(c.x, r), A::add(c.y, r), A::add(c.z, r)};
  bool hit = sub < nt && in_bounds(t, mv.n_tri, b.err);
  Triangle<T> g = {};
  if (hit) {
    g = triangle<T>(mv, t);  // (with the box, not after it)
    hit = in_box<T>(mv, t, lo, hi) && mesh_hit<T>(g, c, r, sp);
  }
  // what the hit adds (mesh_add's operations)
  const V3<T> n = g.n;
  const T vn2 = A::mul(T(2), dot3<T>(V.x, V.y, V.z, n.x, n.y, n.z));
  const V3<T> refl = {A::fma(-vn2, n.x, V.x), A::fma(-vn2, n.y, V.y), A::fma(-vn2, n.z, V.z)};
  const T sc = A::sub(r, dot3<T>(-n.x, -n.y, -n.z, A::sub(c.x, g.a.x), A::sub(c.y, g.a.y), A::sub(c.z, g.a.z)));
  const uint32_t who = __ballot_sync(0xffffffffu, hit);
  const uint32_t ours = (threadIdx.x & 16u) ? who >> 16 : who & 0xffffu;
  MeshSums<T> m = {};
  for (uint32_t left = (who | (who >> 16)) & 0xffffu; left != 0u; left &= left - 1u) {
    const int k = __ffs(left) - 1;
    const V3<T> rk = {__shfl_sync(0xffffffffu, refl.x, k, 16), __shfl_sync(0xffffffffu, refl.y, k, 16),
                      __shfl_sync(0xffffffffu, refl.z, k, 16)};
    const V3<T> nk = {__shfl_sync(0xffffffffu, n.x, k, 16), __shfl_sync(0xffffffffu, n.y, k, 16),
                      __shfl_sync(0xffffffffu, n.z, k, 16)};
    const T sk = __shfl_sync(0xffffffffu, sc, k, 16);
    if ((ours >> k) & 1u) {
      m.v = {A::fma(sp.e_poly, rk.x, m.v.x), A::fma(sp.e_poly, rk.y, m.v.y), A::fma(sp.e_poly, rk.z, m.v.z)};
      m.x = {A::fma(-sk, nk.x, m.x.x), A::fma(-sk, nk.y, m.x.y), A::fma(-sk, nk.z, m.x.z)};
      ++m.hits;
    }
  }
  mesh_apply<T>(m, c, P, V);
}

// The spheres that need run_slow's order, in the step right after a build and
// where they are many: the grid is that of the present positions, so the
// 27-cell walk of a grid step gives the order, a lane to each sphere, and the
// step takes no longer than one of those however many contacts they have.
// run_list_step calls it: a call inside run_late, whose registers it takes,
// cost every step (4,000-sphere funnel, steps 42 to 328, each against the
// kernel without this function in turn: 2,447 -> 2,628 us; now 2,600 -> 2,495).
constexpr uint32_t RUN_FRESH_MIN = STEP_THREADS / 32;  // more than a warp each
template <class T, bool MULTI, bool MESH, bool TAPE>
__device__ __noinline__ float run_fresh(const StepBufs<T>& b, const SceneParams<T>& sp0, const MeshView* mv,
                                        const RunBufs<T>& R, const RunLate& l, int cur, uint32_t build, uint32_t s,
                                        bool last) {
  const vec4_t<T>* Ps = R.p(cur);
  const vec4_t<T>* Vs = R.v(cur);
  float m = 0.0f;
  for (uint32_t k = threadIdx.x; k < l.n_slow; k += STEP_THREADS) {
    const uint32_t i = run_put<T>(l, R, k, true);
    const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
    vec4_t<T> P = Ps[i];
    const vec4_t<T> Vi = Vs[i];
    vec4_t<T> V = Vi;
    const bool live = isfinite(P.x) && isfinite(P.y) && isfinite(P.z);
    int32_t cx, cy, cz;
    cell_coords<T>(b.scell[i], sp, cx, cy, cz);
    uint32_t lo[9], hi[9];
    cell_ranges<T>(b, sp, live, cx, cy, cz, lo, hi);
#pragma unroll
    for (int q = 0; q < 9; ++q)
      for (uint32_t j = lo[q]; j < hi[q]; ++j) {
        if (q == 4 && j == i) continue;
        contact_one<T, true>(Vs, j, P, Vi, Ps[j], sp.k_spring, sp.e_sphere, V.x, V.y, V.z);
      }
    if (TAPE) run_record<T>(R, b, s, i, P, V, Vi);
    if (!last) {
      const vec4_t<T> old = P;
      integrate<T>(P, V, sp);
      if constexpr (MESH) {
        if (sp.mesh_tris > 0)
          mesh_contacts<T>(P, V, sp, *mv, b.err);
        else
          walls<T>(P, V, sp);
      } else {
        walls<T>(P, V, sp);
      }
      run_finish<T, false>(P, [&] { return b.scell[i]; }, R.template counts<TAPE>(build, b.n)[i], sp, old, m);
    }
    (cur ? R.P[0] : R.P[1])[i] = P;
    (cur ? R.V[0] : R.V[1])[i] = V;
  }
  return m;
}

// The step of the spheres put aside: a warp to each of the n_slow that need
// run_slow's order (none where run_fresh has taken them), half a warp to each
// near a triangle.  (A function for each of the two kinds: 30,011-sphere pile,
// 328 steps, 2,750 -> 2,804 us.  The part of run_slow for more than 32 pairs as
// a function of its own: 2,717 -> 2,778.)
template <class T, bool MULTI, bool MESH, bool TAPE>
__device__ __noinline__ float run_late(const StepBufs<T>& b, const SceneParams<T>& sp0, const MeshView* mv,
                                       const RunBufs<T>& R, const RunLate& l, int cur, float frac, uint32_t build,
                                       uint32_t s, bool last, uint32_t n_slow) {
  const vec4_t<T>* Ps = R.p(cur);
  const vec4_t<T>* Vs = R.v(cur);
  vec4_t<T>* Pd = R.p(1 - cur);
  vec4_t<T>* Vd = R.v(1 - cur);
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t n_near = MESH ? l.n_near : 0u;
  float m = 0.0f;
  for (uint32_t k = threadIdx.x >> 5; k < n_slow; k += STEP_THREADS / 32) {
    const uint32_t i = run_put<T>(l, R, k, true);
    const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
    const uint32_t word = R.template counts<TAPE>(build, b.n)[i];
    const uint32_t* list = R.template lists<TAPE>(build, b.n);
    uint32_t mine = lane < R.cap ? list[(size_t)lane * b.n + i] & ~RUN_FAR_CELL : i;
    vec4_t<T> old = Ps[i];
    const vec4_t<T> Vi = Vs[i];
    if (lane >= (word & RUN_COUNT) || !in_bounds(mine, b.n, b.err)) mine = i;
    vec4_t<T> V = run_slow<T>(i, word, mine, list, b, sp, Ps, Vs, (T)frac, old, Vi);
    old.w = fabs(old.w);
    vec4_t<T> P = old;
    if (TAPE && lane == 0u) run_record<T>(R, b, s, i, P, V, Vi);
    if (!last) {
      integrate<T>(P, V, sp);
      if constexpr (MESH) {
        if (sp.mesh_tris > 0)
          mesh_contacts<T>(P, V, sp, *mv, b.err);
        else
          walls<T>(P, V, sp);
      } else {
        walls<T>(P, V, sp);
      }
      run_finish<T, false>(P, [&] { return b.scell[i]; }, word, sp, old, m);
    }
    __syncwarp();
    if (lane == 0u) {
      Pd[i] = P;
      Vd[i] = V;
    }
  }
  if constexpr (MESH) {
    for (uint32_t k0 = (threadIdx.x >> 5) * 2u; k0 < n_near; k0 += STEP_THREADS / 16) {
      const uint32_t k = k0 + ((threadIdx.x >> 4) & 1u);
      const bool on = k < n_near;
      const uint32_t i = run_put<T>(l, R, on ? k : k0, false);
      const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
      const uint32_t word = R.template counts<TAPE>(build, b.n)[i], nt = word >> RUN_TRIS;
      const uint32_t t = R.tris[(size_t)(lane & 15u) * b.n + i];
      const vec4_t<T> old = Ps[i];
      vec4_t<T> P = Pd[i], V = Vd[i];
      // a sphere beyond its list walks its bin instead
      const bool walk = on && (nt > RUN_TRI_CAP || run_near_mesh<T>(P, old, 0u, (T)frac * sp.interval));
      vec4_t<T> Pw = P, Vw = V;
      if (walk) mesh_contacts<T>(Pw, Vw, sp, *mv, b.err);
      __syncwarp();
      run_mesh_half<T>(P, V, on && !walk ? nt : 0u, t, b, sp, *mv);
      if (walk) P = Pw, V = Vw;
      run_finish<T, false>(P, [&] { return b.scell[i]; }, word, sp, old, m);
      __syncwarp();
      if (on && (lane & 15u) == 0u) {
        Pd[i] = P;
        Vd[i] = V;
      }
    }
  }
  return m;
}

// A thread's own sphere, kept in registers from step to step when the grid
// has a thread for every sphere.
template <class T>
struct RunOwn {
  vec4_t<T> P, V;
  uint32_t word, cell;
  uint32_t head[run_batch<T>()];  // first entries of its list
};

template <class T, bool OWN>
__device__ __forceinline__ void run_load_own(RunOwn<T>& o, uint32_t i, const StepBufs<T>& b, const vec4_t<T>* Ps,
                                             const vec4_t<T>* Vs, const uint32_t* list, const uint16_t* cnt) {
  o.P = Ps[i];
  o.V = Vs[i];
  o.word = cnt[i];
  if constexpr (!OWN) return;
  o.cell = b.scell[i];
#pragma unroll
  for (int u = 0; u < run_batch<T>(); ++u)
    o.head[u] = (uint32_t)u < (o.word & RUN_COUNT) ? list[(size_t)u * b.n + i] : i;
}

// One step on the lists: contacts of the state in buffer `cur`, then, unless
// it is the call's last step, the next step's integration and container.
// OWN: each thread has one sphere at most, and `own` holds it (loaded when
// `fresh`), so that a step waits for its neighbours' positions alone.
template <class T, bool MULTI, bool MESH, bool OWN, bool TAPE>
__device__ __forceinline__ float run_list_step(const StepBufs<T>& b, const SceneParams<T>& sp0, const MeshView* mv,
                                               const RunBufs<T>& R, int cur, float frac, uint32_t build, uint32_t s,
                                               bool last, RunOwn<T>& own, bool fresh) {
  const uint32_t* list = R.template lists<TAPE>(build, b.n);
  const uint16_t* cnt = R.template counts<TAPE>(build, b.n);
  const vec4_t<T>* Ps = R.p(cur);
  const vec4_t<T>* Vs = R.v(cur);
  vec4_t<T>* Pd = R.p(1 - cur);
  vec4_t<T>* Vd = R.v(1 - cur);
  constexpr int NB = run_batch<T>();
  __shared__ RunLate late;
  if (threadIdx.x == 0) late.n_slow = late.n_near = 0u;
  __syncthreads();
  float m = 0.0f;
  bool odd = false, near = false;
  for (uint32_t i = blockIdx.x * STEP_THREADS + threadIdx.x; i < b.n; i += gridDim.x * STEP_THREADS) {
    odd = near = false;
    {
      const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
      if (!OWN || fresh) run_load_own<T, OWN>(own, i, b, Ps, Vs, list, cnt);
      const vec4_t<T> Vi = own.V;
      const uint32_t nl = own.word & RUN_COUNT;
      // Partners that have left their cell of the build may change the order,
      // if there are two; a pair as wide as a cell may be of cells that are
      // not adjacent, by the rounding of the hash (below a thousandth of a
      // cell up to 4,096 cells on an axis), and is marked or was so at the build.
      uint32_t touching = 0;
      bool moved = false, wide = (own.word & RUN_OVERFLOW) != 0u;
      uint32_t next[NB];
      if constexpr (OWN) {
#pragma unroll
        for (int u = 0; u < NB; ++u) next[u] = own.head[u];
      }
      for (uint32_t k0 = 0; k0 < nl; k0 += NB) {
        uint32_t jj[NB];
        vec4_t<T> Q[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          jj[u] = OWN ? next[u] : (k0 + u < nl ? list[(size_t)(k0 + u) * b.n + i] : i);
          if (!in_bounds(jj[u] & ~RUN_FAR_CELL, b.n, b.err)) jj[u] = i;
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) Q[u] = Ps[jj[u] & ~RUN_FAR_CELL];
        if constexpr (OWN) {  // (64 registers, of the other form, do not hold them)
#pragma unroll
          for (int u = 0; u < NB; ++u) next[u] = k0 + NB + u < nl ? list[(size_t)(k0 + NB + u) * b.n + i] : i;
        }
#pragma unroll
        for (int u = 0; u < NB; ++u)
          if (k0 + u < nl && contact_one<T, true>(Vs, jj[u] & ~RUN_FAR_CELL, own.P, Vi, Q[u], sp.k_spring, sp.e_sphere,
                                                  own.V.x, own.V.y, own.V.z)) {
            ++touching;
            moved |= marked<T>(Q[u].w);
            wide |= (jj[u] & RUN_FAR_CELL) != 0u ||
                    ((marked<T>(Q[u].w) || marked<T>(own.P.w)) &&
                     (fabs(own.P.w) + fabs(Q[u].w) > T(0.999) * sp.interval ||
                      max(sp.nb[0], max(sp.nb[1], sp.nb[2])) > 4096));
          }
      }
      odd = wide || (moved && touching > 1u);
      own.P.w = fabs(own.P.w);
      if (TAPE && !odd) run_record<T>(R, b, s, i, own.P, own.V, Vi);
      if (!last && !odd) {
        const vec4_t<T> old = own.P;
        integrate<T>(own.P, own.V, sp);
        bool box = true;
        if constexpr (MESH) {
          if (sp.mesh_tris > 0) {
            box = false;
            near = run_near_mesh<T>(own.P, old, own.word, (T)frac * sp.interval);
            if (!near) {  // the container adds a zero correction
              own.P.x = Ar<T>::add(own.P.x, T(0));
              own.P.y = Ar<T>::add(own.P.y, T(0));
              own.P.z = Ar<T>::add(own.P.z, T(0));
            }
          }
        }
        if (box) walls<T>(own.P, own.V, sp);
        if (!near) run_finish<T, OWN>(own.P, [&] { return OWN ? own.cell : b.scell[i]; }, own.word, sp, old, m);
      }
      Pd[i] = own.P;
      Vd[i] = own.V;
    }
    if (odd || near) run_put_aside<T>(late, R, i, odd);
  }
  __syncthreads();
  if (late.n_slow + late.n_near > 0u) {
    const bool walk = fresh && late.n_slow > RUN_FRESH_MIN;
    if (walk) m = fmaxf(m, run_fresh<T, MULTI, MESH, TAPE>(b, sp0, mv, R, late, cur, build, s, last));
    m = fmaxf(m, run_late<T, MULTI, MESH, TAPE>(b, sp0, mv, R, late, cur, frac, build, s, last, walk ? 0u : late.n_slow));
    if (fresh && run_crowded<TAPE>(R)) m = INFINITY;
    if constexpr (OWN) {
      __syncthreads();
      if (odd || near) {
        const uint32_t i = blockIdx.x * STEP_THREADS + threadIdx.x;
        own.P = Pd[i];
        own.V = Vd[i];
      }
    }
  }
  return m;
}

// `steps` steps from the at-rest state (P0, V1, orig), which is also where
// the state ends.
// OWN: the grid has a thread for every sphere.  TAPE: recording for the
// backward pass.
//
// CTAs per SM: with more spheres than threads the warps in flight hide the
// latency, and four CTAs leave 64 registers (FP32); with a thread for every
// sphere there are no more warps to have, and half the CTAs leave room for
// the sphere's state.
template <class T, bool OWN>
__host__ __device__ constexpr int run_ctas() {
  return (sizeof(T) == 4 ? 4 : 2) / (OWN ? 2 : 1);
}

template <class T, bool MULTI, bool MESH, bool OWN, bool TAPE>
__global__ void __launch_bounds__(STEP_THREADS, run_ctas<T, OWN>())
    k_run(const __grid_constant__ StepBufs<T> b, const __grid_constant__ SceneParams<T> sp0, const MeshView* mv,
          const __grid_constant__ RunBufs<T> R, uint32_t steps, int64_t n_cells, uint32_t scatter_blocks,
          uint32_t move_blocks, uint32_t run_id) {
  uint32_t* maxd = R.ctl + RUN_MAXD;
  if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<unsigned long long*>(R.bar_next) = 0ull;
  const uint32_t failed = *reinterpret_cast<volatile uint32_t*>(b.err) & PS_DEVERR_LIST_BARRIER;
  uint32_t streak = *reinterpret_cast<volatile uint32_t*>(R.ctl + RUN_STREAK);
  // the last step's m, of an earlier run if need be
  float before = __uint_as_float(*reinterpret_cast<volatile uint32_t*>(R.ctl + RUN_BEFORE));
  if (!(before > 0.0f) || TAPE) before = INFINITY;
  if (failed) return;  // (an earlier launch: of this one, no CTA gives up before the others have read the word)
  run_begin<T, MULTI, MESH>(b, sp0, mv, R);
  int cur = 1;           // buffer with the state before the step's contacts
  bool lists = false;    // the lists are those of a build that still covers the motion
  bool counted = true;   // the state's cells are counted already
  if (blockIdx.x == 0 && threadIdx.x == 0) R.ctl[RUN_CROWD] = 0u;
  float D = 0.0f;        // motion since the last build, in cells
  float frac = 0.0f;     // skin of the last build, in cells
  uint32_t rebuilds = 0, build = 0;
  RunOwn<T> own;
  for (uint32_t s = 0; s < steps; ++s) {
    if (!run_barrier(R.bar, b.err)) return run_leave(b, R.ctl);
    const float m = sqrtf(__uint_as_float(*reinterpret_cast<volatile uint32_t*>(maxd + s % 3u)));
    if (blockIdx.x == 0 && threadIdx.x == 0) maxd[(s + 2u) % 3u] = 0u;
    streak = m <= RUN_CALM_MAX ? (streak < RUN_CALM_STEPS ? streak + 1u : streak) : 0u;
    D = D * 1.000001f + m;
    bool fresh = false;  // the state's grid was built before this step
    if (!lists || !(D <= 0.49f * frac)) {
      if (TAPE) {  // a recorded run has lists in every step, or gives up
        if (m > RUN_CALM_MAX || rebuilds == R.max_builds) return;
        build = rebuilds;
        streak = RUN_CALM_STEPS;
      }
      lists = !run_crowded<TAPE>(R) && (streak >= RUN_CALM_STEPS || R.skin > 0.0f);
      // (a single fast step, a sphere pushed out of a wall, is no measure)
      // (A recorded run depends on its starting state alone, for the backward
      // pass to give the same sums every time; its builds have to last for
      // the block, and the first, of unknown speed, is kept thin.)
      const float last_for = TAPE ? fmaxf(RUN_STEPS_PER_BUILD, 0.7f * (float)steps) : RUN_STEPS_PER_BUILD;
      const float widest = TAPE && s == 0u ? RUN_SKIN_FIRST : RUN_SKIN_MAX;
      frac = fminf(fmaxf(fminf(m, before) * (last_for / 0.49f), RUN_SKIN_MIN), widest);
      frac = !lists ? 0.0f : (R.skin > 0.0f ? R.skin : frac);
      if (!run_rebuild<T, MULTI, MESH, TAPE>(b, sp0, mv, R, cur, counted, frac, build, n_cells, scatter_blocks, move_blocks))
        return run_leave(b, R.ctl);
      cur = 1 - cur;
      D = 0.0f;
      fresh = true;
      ++rebuilds;
    }
    before = m;
    if (TAPE && blockIdx.x == 0 && threadIdx.x == 0) R.tape_build[s] = build;
    const bool last = s + 1u == steps;
    float mm;
    if (lists)
      mm = run_list_step<T, MULTI, MESH, OWN, TAPE>(b, sp0, mv, R, cur, frac, build, s, last, own, fresh);
    else
      mm = run_grid_step<T, MULTI, MESH>(b, sp0, mv, R, cur, last);
    if (!last) publish_max(mm, maxd + (s + 1u) % 3u);
    counted = !lists;
    cur = 1 - cur;
  }
  // the state is in buffer `cur`; at rest the positions are in P0 and the velocities in V1
  if (!run_barrier(R.bar, b.err)) return run_leave(b, R.ctl);
  for (uint32_t i = blockIdx.x * STEP_THREADS + threadIdx.x; i < b.n; i += gridDim.x * STEP_THREADS) {
    if (cur == 1)
      R.P[0][i] = R.P[1][i];
    else
      R.V[1][i] = R.V[0][i];
  }
  if (blockIdx.x == 0 && threadIdx.x < 3u) maxd[threadIdx.x] = 0u;
  if (blockIdx.x == 0 && threadIdx.x == 3u) R.ctl[RUN_RMAX] = 0u;
  if (blockIdx.x == 0 && threadIdx.x == 0u) {
    if (TAPE) R.tape_build[steps] = R.ctl[RUN_FULL] == 0u ? 1u : 0u;
    R.ctl[RUN_BUILDS] += rebuilds - 1u;
    R.ctl[RUN_STREAK] = streak;
    R.report[0] = run_id;
    R.ctl[RUN_BEFORE] = __float_as_uint(before);
    R.report[1] = (steps >= 64u ? 4u : 2u) * rebuilds > steps ? 1u : 0u;
  }
}

}  // namespace psb
