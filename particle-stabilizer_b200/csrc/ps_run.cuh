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
//     cells of the last build instead (run_slow).
//
// When the fastest sphere moves more than RUN_CALM_MAX cells in a step, or
// did within the last RUN_CALM_STEPS steps, no list would last: such a step
// rebuilds the grid and walks the 27 cells, like the step kernels.  The skin
// of a build follows from the speed, so that a build lasts about
// RUN_STEPS_PER_BUILD steps.
//
// What bounds it: a list step moves 66 B per sphere in FP32 (position and
// velocity in and out, one 2-byte count), mostly through L2 up to a million
// spheres; what remains is the chain count -> list entry -> position ->
// velocity of the touching pairs and the barrier (about 1.5 us).
#pragma once

#include "ps_lists.cuh"

namespace psb {

constexpr int RUN_MIN_STEPS = 8;
constexpr uint32_t RUN_LIST_CAP = 32;
constexpr float RUN_CALM_MAX = 0.02f;
constexpr uint32_t RUN_CALM_STEPS = 2;
constexpr float RUN_STEPS_PER_BUILD = 64.0f;
constexpr float RUN_SKIN_MIN = 0.02f, RUN_SKIN_MAX = 0.25f;

// count word of a sphere: list length and what its step needs besides
enum : uint32_t {
  RUN_COUNT = 0x1fffu,
  RUN_NEAR_MESH = 1u << 13,  // a triangle may come within reach before the next build
  RUN_OVERFLOW = 1u << 14,   // more neighbours than the list holds
  RUN_NEAR_FACE = 1u << 15,  // may leave its cell before the next build
};
constexpr uint32_t RUN_FAR_CELL = 0x80000000u;  // list entry: cells not adjacent at the build
static_assert(RUN_LIST_CAP <= RUN_COUNT, "list length fits the count word");

// control words
enum : int {
  RUN_BAR = 0,      // grid barrier: arrivals so far (64 bits)
  RUN_MAXD = 2,     // largest squared displacement of a step, in cells (3 words, by step)
  RUN_STREAK = 5,   // calm steps up to now
  RUN_RMAX = 6,     // largest radius, in cells of its scene
};

template <class T>
struct RunBufs {
  vec4_t<T>* P[2];
  vec4_t<T>* V[2];
  uint32_t* list;       // [k][slot]
  uint16_t* cnt;
  uint32_t* later;      // per CTA: slots that the step takes after the others (run_late)
  uint32_t* ctl;
  uint32_t* report;     // number of the last run, and whether most of its steps rebuilt the grid
  uint32_t cap;
  uint32_t later_stride;  // entries of `later` per CTA
  __device__ __forceinline__ vec4_t<T>* p(int k) const { return k ? P[1] : P[0]; }
  __device__ __forceinline__ vec4_t<T>* v(int k) const { return k ? V[1] : V[0]; }
};

// One phase's end for the whole grid.  Arrivals only ever count up, by
// gridDim per barrier, so nothing is reset between barriers or launches.
// Bounded like grid_barrier; the limit is longer because one phase of a
// diverged scene (spheres crowded into one cell) may take long.
constexpr uint32_t RUN_BARRIER_SPIN_LIMIT = 1u << 26;

__device__ __forceinline__ bool run_barrier(uint32_t* ctl, uint32_t* err) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(ctl + RUN_BAR);
    __threadfence();
    const unsigned long long ticket = atomicAdd(bar, 1ull);
    const unsigned long long target = (ticket / gridDim.x + 1ull) * gridDim.x;
    uint32_t spins = 0;
    unsigned long long seen = ticket + 1ull;
    while (seen < target) {
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(bar) : "memory");
      if (seen >= target) break;
      if (++spins == RUN_BARRIER_SPIN_LIMIT) {
        atomicOr(err, PS_DEVERR_LIST_BARRIER);
        ok = 0;
        break;
      }
      __nanosleep(20);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
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
  const bool fin = isfinite(P.x) && isfinite(P.y) && isfinite(P.z);
  return !fin ? 0.0f : (m <= 3.0e38f ? m : INFINITY);
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

// Candidates whose positions are fetched together.
template <class T>
__host__ __device__ constexpr int run_batch() {
  return sizeof(T) == 4 ? 4 : 2;
}

// List and count word of slot i of the sorted state (positions P, sorted
// cell ids scell); columns are visited in ascending cell id, so a list is in
// ascending (cell, original index).
template <class T, bool MULTI, bool MESH>
__device__ __forceinline__ void run_build_one(uint32_t i, const StepBufs<T>& b, const SceneParams<T>& sp,
                                              const MeshView* mv, const RunBufs<T>& R, const vec4_t<T>* Ps, T frac,
                                              T rmax) {
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
          R.list[(size_t)k * b.n + i] = entry;
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
      if (sp.mesh_tris > 0 && mesh_within<T>(P, skin, sp, *mv, b.err)) word |= RUN_NEAR_MESH;
    }
  }
  if (k > R.cap) word |= RUN_OVERFLOW, k = 0;
  R.cnt[i] = (uint16_t)(word | k);
}

// Contacts of slot i in the exact order whatever has moved: the overlapping
// partners whose cell is adjacent now, by ascending (cell now, original
// index).  Every lane of the warp calls it with the same sphere.
//
// The lanes take the list's entries side by side, each forms its pair's key
// and force, and the forces are added in the order of the keys.  With the
// list overflowed the candidates are those of the cells of the last build,
// and the smallest key above the last one is looked for in turn.
template <class T>
__device__ __forceinline__ vec4_t<T> run_slow(uint32_t i, uint32_t word, const StepBufs<T>& b,
                                              const SceneParams<T>& sp, const RunBufs<T>& R, const vec4_t<T>* Ps,
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
    const vec4_t<T> Q = Ps[j];
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
    f = contact_force<T>(Vi, Vs[j], dx, dy, dz, d2, dist, overlap, sp.k_spring, sp.e_sphere);
    return ((uint64_t)cj << 32) | (uint64_t)b.orig[j];
  };
  auto smallest = [&](uint64_t key) -> uint64_t {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const uint64_t t = __shfl_xor_sync(0xffffffffu, key, d);
      key = t < key ? t : key;
    }
    return key;
  };
  auto apply = [&](int from) {
    const T g = __shfl_sync(0xffffffffu, f, from);
    V.x = A::fma(g, __shfl_sync(0xffffffffu, dx, from), V.x);
    V.y = A::fma(g, __shfl_sync(0xffffffffu, dy, from), V.y);
    V.z = A::fma(g, __shfl_sync(0xffffffffu, dz, from), V.z);
  };
  if (!(word & RUN_OVERFLOW)) {
    static_assert(RUN_LIST_CAP <= 32, "a list is one entry per lane");
    uint64_t key = NONE;
    if (lane < (word & RUN_COUNT)) {
      const uint32_t j = R.list[(size_t)lane * b.n + i] & ~RUN_FAR_CELL;
      if (in_bounds(j, b.n, b.err)) key = key_of(j);
    }
    for (uint64_t best = smallest(key); best != NONE; best = smallest(key)) {
      apply(__ffs(__ballot_sync(0xffffffffu, key == best)) - 1);
      if (key == best) key = NONE;
    }
    return V;
  }
  const T skin = frac * sp.interval;
  const Span<T> s = reach_span<T>(P, (fabs(P.w) + T(0.5) * sp.interval + T(2) * skin) * T(1.001), sp);
  for (uint64_t from = 0;;) {
    uint64_t best = NONE;
    T bf = T(0), bdx = T(0), bdy = T(0), bdz = T(0);
    for (int32_t bx = s.x0; bx <= s.x1; ++bx)
      for (int32_t by = s.y0; by <= s.y1; ++by) {
        const uint32_t col = sp.cbase + ((uint32_t)bx * (uint32_t)sp.nb[1] + (uint32_t)by) * (uint32_t)sp.nb[2];
        const uint32_t j1 = b.offset[col + (uint32_t)s.z1 + 1u];
        if (!in_bounds(j1, (uint64_t)b.n + 1u, b.err)) continue;
        for (uint32_t j = b.offset[col + (uint32_t)s.z0] + lane; j < j1; j += 32u) {
          const uint64_t key = key_of(j);
          if (key >= from && key < best) {
            best = key;
            bf = f, bdx = dx, bdy = dy, bdz = dz;
          }
        }
      }
    __syncwarp();
    f = bf, dx = bdx, dy = bdy, dz = bdz;
    const uint64_t next = smallest(best);
    if (next == NONE) return V;
    apply(__ffs(__ballot_sync(0xffffffffu, best == next)) - 1);
    from = next + 1u;
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
      m = fmaxf(m, moved2<T>(P, old, T(1) / (sp.interval * sp.interval)));
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
template <class T, bool MULTI, bool MESH>
__device__ __noinline__ bool run_rebuild(const StepBufs<T>& b, const SceneParams<T>& sp0, const MeshView* mv,
                                         const RunBufs<T>& R, int cur, bool counted, float frac, int64_t n_cells,
                                         uint32_t scatter_blocks, uint32_t move_blocks) {
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
    if (!run_barrier(R.ctl, b.err)) return false;
  }
  for (uint32_t t = blockIdx.x; t < b.n_tiles; t += gridDim.x) {
    __syncthreads();  // the tile scan reuses its shared arrays
    if (b.tile_shift == 13u)
      scan_tile_with_sums<true, STEP_SCAN_ITEMS_LARGE>(t, b.count, b.offset, n_cells, b.tile_sum);
    else
      scan_tile_with_sums<true, STEP_SCAN_ITEMS_SMALL>(t, b.count, b.offset, n_cells, b.tile_sum);
  }
  if (!run_barrier(R.ctl, b.err)) return false;
  for (uint32_t blk = blockIdx.x; blk < scatter_blocks; blk += gridDim.x)
    scatter_block<true>(blk, b.cell, b.slot, b.orig, b.offset, b.tmp, b.count, b.n, b.tile_sum, b.n_tiles, b.err);
  if (!run_barrier(R.ctl, b.err)) return false;
  StepBufs<T> mb = b;
  mb.P1 = R.p(cur);
  mb.V1 = R.v(cur);
  mb.P0 = R.p(1 - cur);
  mb.V0 = R.v(1 - cur);
  for (uint32_t blk = blockIdx.x; blk < move_blocks; blk += gridDim.x) rank_move_block<T, true>(blk, mb);
  if (!run_barrier(R.ctl, b.err)) return false;
  if (frac > 0.0f) {
    const vec4_t<T>* Ps = R.p(1 - cur);
    const T rmax = (T)__uint_as_float(R.ctl[RUN_RMAX]) * T(1.0001);
    for (uint32_t i = blockIdx.x * STEP_THREADS + threadIdx.x; i < b.n; i += stride)
      run_build_one<T, MULTI, MESH>(i, b, scene_of<T, MULTI>(i, sp0, b), mv, R, Ps, (T)frac, rmax);
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
        m = fmaxf(m, moved2<T>(P, old, T(1) / (sp.interval * sp.interval)));
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

// The end of sphere i's step, after its integration: the container, the
// displacement from `old`, and the mark of a sphere outside its cell of the
// build.  TEST: triangles are tested; else none is within reach and a
// triangle container adds zero.
template <class T, bool MESH, bool TEST>
__device__ __forceinline__ void run_advance(vec4_t<T>& P, vec4_t<T>& V, uint32_t i, uint32_t word,
                                            const StepBufs<T>& b, const SceneParams<T>& sp, const MeshView* mv,
                                            const vec4_t<T>& old, float& m) {
  if constexpr (MESH) {
    if (sp.mesh_tris > 0) {
      if constexpr (TEST) {
        mesh_contacts<T>(P, V, sp, *mv, b.err);
      } else {
        P.x = Ar<T>::add(P.x, T(0));
        P.y = Ar<T>::add(P.y, T(0));
        P.z = Ar<T>::add(P.z, T(0));
      }
    } else {
      walls<T>(P, V, sp);
    }
  } else {
    walls<T>(P, V, sp);
  }
  m = fmaxf(m, moved2<T>(P, old, T(1) / (sp.interval * sp.interval)));
  if (word & RUN_NEAR_FACE) {
    int32_t cx, cy, cz;
    if (cell_of<T>(P.x, P.y, P.z, sp, cx, cy, cz) != b.scell[i]) P.w = -P.w;
  }
}

// The list step of the spheres it put aside, whose chains of loads are long:
// taken inline by their own thread, a handful of them held the whole step up
// (30,011-sphere pile: 7.2 us a step without any, 14.5 us with forty).  A
// warp takes each sphere that needs run_slow's order (the first n_slow
// entries); a thread each near a triangle (the last n_mesh entries, contacts
// and integration done), which gathers them into full warps.
template <class T, bool MULTI, bool MESH>
__device__ __noinline__ float run_late(const StepBufs<T>& b, const SceneParams<T>& sp0, const MeshView* mv,
                                       const RunBufs<T>& R, int cur, float frac, bool last, uint32_t n_slow,
                                       uint32_t n_mesh) {
  const vec4_t<T>* Ps = R.p(cur);
  const vec4_t<T>* Vs = R.v(cur);
  vec4_t<T>* Pd = R.p(1 - cur);
  vec4_t<T>* Vd = R.v(1 - cur);
  const uint32_t* later = R.later + (size_t)blockIdx.x * R.later_stride;
  float m = 0.0f;
  for (uint32_t k = threadIdx.x >> 5; k < n_slow; k += STEP_THREADS / 32) {
    const uint32_t i = later[k];
    const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
    const uint32_t word = R.cnt[i];
    vec4_t<T> old = Ps[i];
    vec4_t<T> V = run_slow<T>(i, word, b, sp, R, Ps, Vs, (T)frac, old, Vs[i]);
    old.w = fabs(old.w);
    vec4_t<T> P = old;
    if (!last) {
      integrate<T>(P, V, sp);
      run_advance<T, MESH, true>(P, V, i, word, b, sp, mv, old, m);
    }
    __syncwarp();
    if ((threadIdx.x & 31u) == 0u) {
      Pd[i] = P;
      Vd[i] = V;
    }
  }
  if constexpr (MESH) {
    for (uint32_t k = threadIdx.x; k < n_mesh; k += STEP_THREADS) {
      const uint32_t i = later[R.later_stride - 1u - k];
      vec4_t<T> P = Pd[i], V = Vd[i];
      run_advance<T, MESH, true>(P, V, i, R.cnt[i], b, scene_of<T, MULTI>(i, sp0, b), mv, Ps[i], m);
      Pd[i] = P;
      Vd[i] = V;
    }
  }
  return m;
}

// One step on the lists: contacts of the state in buffer `cur`, then, unless
// it is the call's last step, the next step's integration and container.
template <class T, bool MULTI, bool MESH>
__device__ __forceinline__ float run_list_step(const StepBufs<T>& b, const SceneParams<T>& sp0, const MeshView* mv,
                                               const RunBufs<T>& R, int cur, float frac, bool last) {
  __shared__ uint32_t s_slow, s_mesh;
  if (threadIdx.x == 0) s_slow = s_mesh = 0u;
  __syncthreads();
  const vec4_t<T>* Ps = R.p(cur);
  const vec4_t<T>* Vs = R.v(cur);
  vec4_t<T>* Pd = R.p(1 - cur);
  vec4_t<T>* Vd = R.v(1 - cur);
  float m = 0.0f;
  for (uint32_t i = blockIdx.x * STEP_THREADS + threadIdx.x; i < b.n; i += gridDim.x * STEP_THREADS) {
    const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
    vec4_t<T> P = Ps[i];
    const vec4_t<T> Vi = Vs[i];
    const uint32_t word = R.cnt[i];
    vec4_t<T> V = Vi;
    const uint32_t nl = word & RUN_COUNT;
    bool odd = (word & RUN_OVERFLOW) != 0u;
    constexpr int NB = run_batch<T>();
    for (uint32_t k0 = 0; k0 < nl; k0 += NB) {
      uint32_t jj[NB];
      vec4_t<T> Q[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        jj[u] = k0 + u < nl ? R.list[(size_t)(k0 + u) * b.n + i] : i;
        if (!in_bounds(jj[u] & ~RUN_FAR_CELL, b.n, b.err)) jj[u] = i;
      }
#pragma unroll
      for (int u = 0; u < NB; ++u) Q[u] = Ps[jj[u] & ~RUN_FAR_CELL];
#pragma unroll
      for (int u = 0; u < NB; ++u)
        if (k0 + u < nl &&
            contact_one<T, true>(Vs, jj[u] & ~RUN_FAR_CELL, P, Vi, Q[u], sp.k_spring, sp.e_sphere, V.x, V.y, V.z))
          odd |= (jj[u] & RUN_FAR_CELL) != 0u || marked<T>(Q[u].w) || marked<T>(P.w);
    }
    P.w = fabs(P.w);
    bool mesh = false;
    if (!last && !odd) {
      const vec4_t<T> old = P;
      integrate<T>(P, V, sp);
      if constexpr (MESH) {
        // near a triangle at the build, or moving a good part of the skin now
        const T lim = T(0.25) * (T)frac * sp.interval;
        const T ex = P.x - old.x, ey = P.y - old.y, ez = P.z - old.z;
        mesh = sp.mesh_tris > 0 && ((word & RUN_NEAR_MESH) || !(ex * ex + ey * ey + ez * ez <= lim * lim));
      }
      if (!mesh) run_advance<T, MESH, false>(P, V, i, word, b, sp, mv, old, m);
    }
    if (odd || mesh) {
      uint32_t* later = R.later + (size_t)blockIdx.x * R.later_stride;
      later[odd ? atomicAdd(&s_slow, 1u) : R.later_stride - 1u - atomicAdd(&s_mesh, 1u)] = i;
    }
    Pd[i] = P;
    Vd[i] = V;
  }
  __syncthreads();
  const uint32_t n_slow = s_slow, n_mesh = s_mesh;
  if (n_slow + n_mesh > 0u) m = fmaxf(m, run_late<T, MULTI, MESH>(b, sp0, mv, R, cur, frac, last, n_slow, n_mesh));
  return m;
}

// `steps` steps from the at-rest state (P0, V1, orig), which is also where
// the state ends.
template <class T, bool MULTI, bool MESH>
__global__ void __launch_bounds__(STEP_THREADS, sizeof(T) == 4 ? 4 : 2)
    k_run(const __grid_constant__ StepBufs<T> b, const __grid_constant__ SceneParams<T> sp0, const MeshView* mv,
          const __grid_constant__ RunBufs<T> R, uint32_t steps, int64_t n_cells, uint32_t scatter_blocks,
          uint32_t move_blocks, uint32_t run_id) {
  uint32_t* maxd = R.ctl + RUN_MAXD;
  uint32_t streak = *reinterpret_cast<volatile uint32_t*>(R.ctl + RUN_STREAK);
  run_begin<T, MULTI, MESH>(b, sp0, mv, R);
  int cur = 1;           // buffer with the state before the step's contacts
  bool lists = false;    // the lists are those of a build that still covers the motion
  bool counted = true;   // the state's cells are counted already
  float D = 0.0f;        // motion since the last build, in cells
  float frac = 0.0f;     // skin of the last build, in cells
  uint32_t unsettled = 0;
  float before = INFINITY;  // the last step's m
  for (uint32_t s = 0; s < steps; ++s) {
    if (!run_barrier(R.ctl, b.err)) return;
    const float m = sqrtf(__uint_as_float(*reinterpret_cast<volatile uint32_t*>(maxd + s % 3u)));
    if (blockIdx.x == 0 && threadIdx.x == 0) maxd[(s + 2u) % 3u] = 0u;
    streak = m <= RUN_CALM_MAX ? (streak < RUN_CALM_STEPS ? streak + 1u : streak) : 0u;
    D = D * 1.000001f + m;
    if (!lists || !(D <= 0.49f * frac)) {
      lists = streak >= RUN_CALM_STEPS;
      // (a single fast step, a sphere pushed out of a wall, is no measure)
      frac = lists ? fminf(fmaxf(fminf(m, before) * (RUN_STEPS_PER_BUILD / 0.49f), RUN_SKIN_MIN), RUN_SKIN_MAX) : 0.0f;
      if (!run_rebuild<T, MULTI, MESH>(b, sp0, mv, R, cur, counted, frac, n_cells, scatter_blocks, move_blocks)) return;
      cur = 1 - cur;
      D = 0.0f;
      unsettled += lists ? 0u : 1u;
    }
    before = m;
    const bool last = s + 1u == steps;
    float mm;
    if (lists)
      mm = run_list_step<T, MULTI, MESH>(b, sp0, mv, R, cur, frac, last);
    else
      mm = run_grid_step<T, MULTI, MESH>(b, sp0, mv, R, cur, last);
    if (!last) publish_max(mm, maxd + (s + 1u) % 3u);
    counted = !lists;
    cur = 1 - cur;
  }
  // the state is in buffer `cur`; at rest the positions are in P0 and the velocities in V1
  if (!run_barrier(R.ctl, b.err)) return;
  for (uint32_t i = blockIdx.x * STEP_THREADS + threadIdx.x; i < b.n; i += gridDim.x * STEP_THREADS) {
    if (cur == 1)
      R.P[0][i] = R.P[1][i];
    else
      R.V[1][i] = R.V[0][i];
  }
  if (blockIdx.x == 0 && threadIdx.x < 3u) maxd[threadIdx.x] = 0u;
  if (blockIdx.x == 0 && threadIdx.x == 3u) R.ctl[RUN_RMAX] = 0u;
  if (blockIdx.x == 0 && threadIdx.x == 0u) {
    R.ctl[RUN_STREAK] = streak;
    R.report[0] = run_id;
    R.report[1] = 2u * unsettled > steps ? 1u : 0u;
  }
}

}  // namespace psb
