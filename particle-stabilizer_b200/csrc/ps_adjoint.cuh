// ps_adjoint.cuh — reverse-mode adjoint of the DEM step (box container).
//
// Forward step (per particle i, the CUDA scheme of PhysicsEngineCUDA.cpp:38-42):
//   x' = x + v dt,  v' = v + g dt                       (integrate)
//   per axis: clamp to the walls, v <- -v e              (walls, events)
//   v''' = v'' + sum_j f_ij d_ij,  x''' = x''            (Jacobi contacts)
//   d = x_i - x_j, L = |d|, ov = r_i + r_j - L > 0,
//   f = k ov / (L m_i) - B (u.d) / L^2,  B = 2 m_j e / (m_i + m_j),  u = v_i - v_j
//
// A block of steps is recomputed from its checkpoint and recorded, one row of
// the tape per step: row t + 1 holds the state after step t as the step's
// contacts left it (positions, velocities, original ids) and the velocities
// before the contacts, in slot order; row t is the step's input.  There are
// two forms:
//   * on lists, by a recorded run (k_run with TAPE): slots keep the order of
//     the run's last build, and the lists and counts of each build are kept;
//   * on the grid, by the step kernels, where a block moves too fast for lists
//     or would need more builds than are kept: slots are in the canonical sort
//     of their step, and the row also has the sorted cell ids and a copy of
//     the step's cell offsets.
// Either way row t + 1 is exactly the state after the walls that step t's
// contacts read, so the reverse sweep needs no rebuild.
//
// Reverse sweep of one step, given the adjoints (xbar, vbar) of its output:
//   k_adj_list       (slots of the build, gather over the slot's list) or
//   k_adj_contacts   (sorted order, gather over the 27 cells): for each
//                    particle, the terms of the pairs where it receives and
//                    the pairs where it is the source (pairs are symmetric),
//                    so no atomics; partials of dL/dk and dL/de_sphere
//                    accumulated per slot (a scene owns a fixed slot range,
//                    so per-scene sums are unchanged and the order is fixed
//                    by that of the slots).
//   walls and integrate: through the walls (clamp events recomputed from the
//                    recorded step input) and the integrate, with the partials
//                    of dL/de_wall.  In k_adj_list where the step before has
//                    the same slots, by k_adj_walls_integrate (slots of row t,
//                    found through `inv`) where it has not.
// Wall clamps and contact activation are piecewise events taken from the
// forward values; radii and masses are constants.
#pragma once

#include "ps_run.cuh"

namespace psb {

enum : int { ADJ_K = 0, ADJ_E = 1, ADJ_WALL = 2 };  // acc rows: k, e_sphere, e_wall[6] (zMin..yMax)
constexpr int ADJ_NACC = 8;

template <class T>
struct AdjBufs {
  TapeRow<T> tape;        // input of the step being reversed
  // Adjoints of positions and velocities (w unused), one 16/32-B record per
  // particle, kept in the sorted order of the at-rest state they belong to:
  // before step t's reverse they follow the order after step t (its grid's
  // order), after it the order of step t's input (the previous grid's), so
  // every kernel reads and writes them by slot.
  vec4_t<T>* ax;
  vec4_t<T>* av;
  vec4_t<T>* ax2;         // output of k_adj_contacts, in the order of step t's grid
  vec4_t<T>* av2;
  uint32_t* inv;          // slot in step t's grid of each original id (written by k_adj_contacts)
  double* acc;            // ADJ_NACC rows of n, accumulated over steps: rows k, e by the slot of
                          // step t's order, wall rows by that of its input
  uint32_t n;             // row length of acc
};

// Geometry of one active pair, shared by its two directions: d = x_i - x_j,
// u = v_i - v_j, L = |d|, ov = R - L, ud = u.d, and the reciprocals.
template <class T>
struct PairGeom {
  T dx, dy, dz, ux, uy, uz, L, iL, iL2, ov, ud, R;
};

// Terms of one direction of an active pair for the receiver r and the
// source s: c_r = f d with f = k ov / (L m_r) - B ud / L^2,
// B = 2 m_s e / (m_r + m_s); g = adjoint of v_r's output; sgn = +1 when r is
// the pair's first sphere (d as stored) and -1 when it is the second (d and
// u negated, ud and L unchanged).  Returns the adjoint of d and of u with
// respect to the pair's stored d and u, and adds the parameter partials.
template <class T>
__device__ __forceinline__ void pair_adjoint(const PairGeom<T>& q, T sgn, T mr, T ms, T inv_msum, T k, T e, T gx,
                                             T gy, T gz, T& ddx, T& ddy, T& ddz, T& dux, T& duy, T& duz,
                                             double& dk, double& de) {
  const T imr = T(1) / mr;
  const T Bc = T(2) * ms * e * inv_msum;
  const T f = k * q.ov * q.iL * imr - Bc * q.ud * q.iL2;
  const T fbar = sgn * (gx * q.dx + gy * q.dy + gz * q.dz);
  dk += (double)(fbar * q.ov * q.iL * imr);
  de += (double)(fbar * (-(T(2) * ms * q.ud) * inv_msum * q.iL2));
  const T fL = -k * q.R * q.iL2 * imr + T(2) * Bc * q.ud * q.iL2 * q.iL;
  const T Lb = fbar * fL * q.iL;
  const T udb = -fbar * Bc * q.iL2;
  // adjoint of the direction's own d (= sgn d) and u (= sgn u), mapped back
  ddx = sgn * (f * gx) + Lb * q.dx + udb * q.ux;
  ddy = sgn * (f * gy) + Lb * q.dy + udb * q.uy;
  ddz = sgn * (f * gz) + Lb * q.dz + udb * q.uz;
  dux = udb * q.dx;
  duy = udb * q.dy;
  duz = udb * q.dz;
}

// Same activation test as the forward contact kernel (contact_one).
template <class T>
__device__ __forceinline__ bool pair_active(const vec4_t<T>& P, const vec4_t<T>& Pj) {
  using A = Ar<T>;
  const T margin = T(1) + T(1.0 / 1048576.0);
  const T dx = A::sub(P.x, Pj.x), dy = A::sub(P.y, Pj.y), dz = A::sub(P.z, Pj.z);
  const T d2 = A::fma(dz, dz, A::fma(dy, dy, A::mul(dx, dx)));
  const T s = A::add(P.w, Pj.w);
  if (d2 >= A::mul(A::mul(s, s), margin)) return false;
  return A::sub(s, A::sqrt(d2)) > T(0);
}

// Both directions of the active pair (i, j): what j's part in the pair adds
// to the adjoints (xo, vo) of i's position and velocity, G and H being the
// adjoints of the two output velocities; the parameter partials of the
// direction in which i receives (those of the other belong to j's thread).
template <class T>
__device__ __forceinline__ void adj_pair(const vec4_t<T>& P, const vec4_t<T>& V, const vec4_t<T>& G,
                                         const vec4_t<T>& Pj, const vec4_t<T>& Vj, const vec4_t<T>& H, T k, T e,
                                         vec4_t<T>& xo, vec4_t<T>& vo, double& dk, double& de) {
  PairGeom<T> g;
  g.dx = P.x - Pj.x;
  g.dy = P.y - Pj.y;
  g.dz = P.z - Pj.z;
  g.ux = V.x - Vj.x;
  g.uy = V.y - Vj.y;
  g.uz = V.z - Vj.z;
  g.R = P.w + Pj.w;
  const T L2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz;
  g.L = sqrt(L2);
  g.iL = T(1) / g.L;
  g.iL2 = T(1) / L2;
  g.ov = g.R - g.L;
  g.ud = g.ux * g.dx + g.uy * g.dy + g.uz * g.dz;
  const T inv_msum = T(1) / (V.w + Vj.w);
  T ddx, ddy, ddz, dux, duy, duz;
  // i receives from j
  pair_adjoint<T>(g, T(1), V.w, Vj.w, inv_msum, k, e, G.x, G.y, G.z, ddx, ddy, ddz, dux, duy, duz, dk, de);
  xo.x += ddx;
  xo.y += ddy;
  xo.z += ddz;
  vo.x += dux;
  vo.y += duy;
  vo.z += duz;
  // j receives from i: that direction's d and u are -d and -u, so its
  // adjoints with respect to the stored d and u come back sign-mapped
  double dk2 = 0.0, de2 = 0.0;
  pair_adjoint<T>(g, T(-1), Vj.w, V.w, inv_msum, k, e, H.x, H.y, H.z, ddx, ddy, ddz, dux, duy, duz, dk2, de2);
  xo.x += ddx;
  xo.y += ddy;
  xo.z += ddz;
  vo.x += dux;
  vo.y += duy;
  vo.z += duz;
}

template <class T, bool MULTI>
__global__ void __launch_bounds__(STEP_THREADS) k_adj_contacts(StepBufs<T> b, AdjBufs<T> a, SceneParams<T> sp0) {
  // one wave of CTAs (occupancy x SMs, the host's choice) loops over the particles
  for (uint32_t i = blockIdx.x * STEP_THREADS + threadIdx.x; i < b.n; i += gridDim.x * STEP_THREADS) {
    const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
    const vec4_t<T> P = b.P0[i];
    const vec4_t<T> V = b.V0[i];
    const uint32_t oi = b.orig[i];
    a.inv[oi] = i;
    const vec4_t<T> G = a.av[i], X = a.ax[i];
    vec4_t<T> xo = X, vo = G;
    double dk = 0.0, de = 0.0;
    int32_t cx, cy, cz;
    cell_coords<T>(b.scell[i], sp, cx, cy, cz);
    const int32_t nx = sp.nb[0], ny = sp.nb[1], nz = sp.nb[2];
    const uint32_t z0 = (uint32_t)(cz > 0 ? cz - 1 : 0);
    const uint32_t z1 = (uint32_t)(cz + 1 < nz ? cz + 1 : nz - 1) + 1u;
    const T k = sp.k_spring, e = sp.e_sphere;
    const bool live = isfinite(P.x) && isfinite(P.y) && isfinite(P.z);  // no active pair otherwise
    uint32_t lo[9], hi[9];
  #pragma unroll
    for (int q = 0; q < 9; ++q) {  // the 18 range bounds, loaded together
      const int32_t bx = cx - 1 + q / 3, by = cy - 1 + q % 3;
      const bool ok = live && bx >= 0 && bx < nx && by >= 0 && by < ny;
      const uint32_t col = ok ? sp.cbase + ((uint32_t)bx * (uint32_t)ny + (uint32_t)by) * (uint32_t)nz : sp.cbase;
      lo[q] = ok ? __ldg(b.offset + col + z0) : 0u;
      hi[q] = ok ? __ldg(b.offset + col + z1) : 0u;
    }
  #pragma unroll
    for (int q = 0; q < 9; ++q)
      for (uint32_t j = lo[q]; j < hi[q]; ++j) {
        if (q == 4 && j == i) continue;  // only the own column holds the sphere itself
        const vec4_t<T> Pj = ld4<T>(b.P0 + j);
        if (!pair_active<T>(P, Pj)) continue;
        adj_pair<T>(P, V, G, Pj, b.V0[j], a.av[j], k, e, xo, vo, dk, de);
      }
    a.ax2[i] = xo;
    a.av2[i] = vo;
    a.acc[(size_t)ADJ_K * a.n + i] += dk;
    a.acc[(size_t)ADJ_E * a.n + i] += de;
  }
}

// Walls + integrate adjoint of slot p of the tape row: (x, v) come in as the
// adjoints of the post-wall state and leave as those of the step's input.
// The input comes from the tape; x' and v' and the clamp events are
// recomputed from it with the forward's operations.
template <class T>
__device__ __forceinline__ void adj_walls_integrate(const AdjBufs<T>& a, const SceneParams<T>& sp, uint32_t p,
                                                    vec4_t<T>& x, vec4_t<T>& v) {
  vec4_t<T> P = a.tape.p[p];
  vec4_t<T> V = a.tape.v[p];
  integrate<T>(P, V, sp);  // x', v'
  using A = Ar<T>;
  const T r = P.w;
  const T xs[3] = {P.x, P.y, P.z}, vs[3] = {V.x, V.y, V.z};
  const int lo_idx[3] = {PS_XMIN, PS_YMIN, PS_ZMIN}, hi_idx[3] = {PS_XMAX, PS_YMAX, PS_ZMAX};
  double* acc = a.acc + p;  // row c at acc[c * n]
  const T xb2[3] = {x.x, x.y, x.z}, vb2[3] = {v.x, v.y, v.z};
  T xo[3], vo[3];
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const bool lo_hit = A::sub(xs[ax], r) < sp.box_lo[ax];
    const bool hi_hit = A::add(xs[ax], r) > sp.box_hi[ax];
    T xb = xb2[ax], vb = vb2[ax];
    const T v1 = lo_hit ? A::mul(-vs[ax], sp.e_lo[ax]) : vs[ax];  // velocity after the min clamp
    if (hi_hit) {
      acc[(size_t)(ADJ_WALL + hi_idx[ax]) * a.n] += (double)(-v1 * vb);
      vb = -sp.e_hi[ax] * vb;
      xb = T(0);
    }
    if (lo_hit) {
      acc[(size_t)(ADJ_WALL + lo_idx[ax]) * a.n] += (double)(-vs[ax] * vb);
      vb = -sp.e_lo[ax] * vb;
      xb = T(0);
    }
    // integrate: x' = x + v dt, v' = v + g dt
    xo[ax] = xb;
    vo[ax] = vb + sp.dt * xb;
  }
  x.x = xo[0];
  x.y = xo[1];
  x.z = xo[2];
  v.x = vo[0];
  v.y = vo[1];
  v.z = vo[2];
}

// The same over all of the tape row's slots, from the order of step t's grid.
template <class T, bool MULTI>
__global__ void __launch_bounds__(STEP_THREADS) k_adj_walls_integrate(StepBufs<T> b, AdjBufs<T> a,
                                                                      SceneParams<T> sp0) {
  pdl_wait();
  const uint32_t p = blockIdx.x * STEP_THREADS + threadIdx.x;
  if (p >= b.n) return;
  const uint32_t i = a.inv[a.tape.o[p]];  // this particle's slot in step t's grid
  vec4_t<T> x = a.ax2[i], v = a.av2[i];
  adj_walls_integrate<T>(a, scene_of<T, MULTI>(p, sp0, b), p, x, v);
  a.ax[p] = x;
  a.av[p] = v;
}

// The reverse of a step that a recorded run took on lists (ps_run.cuh): row
// t + 1 holds what its contacts read, in the order of the build `list`
// belongs to, and the list's pairs take the place of the 27-cell walk (65,536
// spheres in contact, FP32: 19.1 us as a walk).  FUSED: row t is in the same order, so
// the walls and the integration follow at once and (ax, av) goes to
// (ax2, av2); else (ax2, av2) and inv are for k_adj_walls_integrate.
template <class T, bool MULTI, bool FUSED>
__global__ void __launch_bounds__(STEP_THREADS) k_adj_list(StepBufs<T> b, AdjBufs<T> a, SceneParams<T> sp0,
                                                           const uint32_t* __restrict__ list,
                                                           const uint16_t* __restrict__ cnt) {
  pdl_wait();
  const uint32_t i = blockIdx.x * STEP_THREADS + threadIdx.x;
  if (i >= b.n) return;
  const SceneParams<T>& sp = scene_of<T, MULTI>(i, sp0, b);
  const vec4_t<T> P = b.P0[i], V = b.V0[i], G = a.av[i], X = a.ax[i];
  const uint32_t nl = cnt[i] & RUN_COUNT;
  if (!FUSED) a.inv[b.orig[i]] = i;
  vec4_t<T> xo = X, vo = G;
  double dk = 0.0, de = 0.0;
  constexpr int NB = 4;  // pairs whose loads go together
  for (uint32_t k0 = 0; k0 < nl; k0 += NB) {
    uint32_t jj[NB];
    vec4_t<T> Q[NB];
    bool act[NB];
#pragma unroll
    for (int u = 0; u < NB; ++u) jj[u] = k0 + u < nl ? list[(size_t)(k0 + u) * b.n + i] : i;
#pragma unroll
    for (int u = 0; u < NB; ++u) Q[u] = ld4<T>(b.P0 + (jj[u] & ~RUN_FAR_CELL));
#pragma unroll
    for (int u = 0; u < NB; ++u) {
      act[u] = k0 + u < nl && pair_active<T>(P, Q[u]);
      if (act[u] && (jj[u] & RUN_FAR_CELL)) {  // the walk's own condition, which rounding can make stricter
        int32_t cx, cy, cz, jx, jy, jz;
        cell_of<T>(P.x, P.y, P.z, sp, cx, cy, cz);
        cell_of<T>(Q[u].x, Q[u].y, Q[u].z, sp, jx, jy, jz);
        act[u] = abs(jx - cx) <= 1 && abs(jy - cy) <= 1 && abs(jz - cz) <= 1;
      }
    }
#pragma unroll
    for (int u = 0; u < NB; ++u)
      if (act[u]) {
        const uint32_t j = jj[u] & ~RUN_FAR_CELL;
        adj_pair<T>(P, V, G, Q[u], ld4<T>(b.V0 + j), ld4<T>(a.av + j), sp.k_spring, sp.e_sphere, xo, vo, dk, de);
      }
  }
  a.acc[(size_t)ADJ_K * a.n + i] += dk;
  a.acc[(size_t)ADJ_E * a.n + i] += de;
  if constexpr (FUSED) adj_walls_integrate<T>(a, sp, i, xo, vo);
  a.ax2[i] = xo;
  a.av2[i] = vo;
}

// Adjoints from the order of one state (inverse permutation `inv` of its
// original ids) to that of another (`o`).
template <class T>
__global__ void k_adj_reorder(const vec4_t<T>* __restrict__ ax, const vec4_t<T>* __restrict__ av,
                              const uint32_t* __restrict__ inv, const uint32_t* __restrict__ o, vec4_t<T>* ax2,
                              vec4_t<T>* av2, uint32_t n) {
  const uint32_t p = blockIdx.x * STEP_THREADS + threadIdx.x;
  if (p >= n) return;
  const uint32_t i = inv[o[p]];
  ax2[p] = ax[i];
  av2[p] = av[i];
}

__global__ void k_adj_invert(const uint32_t* __restrict__ o, uint32_t* inv, uint32_t n) {
  const uint32_t p = blockIdx.x * STEP_THREADS + threadIdx.x;
  if (p < n) inv[o[p]] = p;
}

// Copy the at-rest state (P0, V1, orig) into a tape row.
template <class T>
__global__ void k_tape_write(StepBufs<T> b, TapeRow<T> row) {
  const uint32_t p = blockIdx.x * STEP_THREADS + threadIdx.x;
  if (p >= b.n) return;
  row.p[p] = b.P0[p];
  row.v[p] = b.V1[p];
  row.o[p] = b.orig[p];
}


// Per-scene sums of the parameter partials (acc: ADJ_NACC rows of n), in a
// fixed order: block (q, c) of a scene adds row c's q-th share, and
// k_adj_reduce_shares the shares.  One block per scene, as this was at first,
// left the GPU idle: 65,536 spheres of one scene took 1.64 ms.
constexpr int ADJ_REDUCE_THREADS = 256;

__device__ __forceinline__ double adj_block_sum(double v, double (&red)[ADJ_REDUCE_THREADS / 32]) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  if ((threadIdx.x & 31u) == 0u) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < ADJ_REDUCE_THREADS / 32; ++w) v += red[w];
  return v;
}

// grid (shares, ADJ_NACC, scenes up to 65,535 at a time, the first being s0)
__global__ void __launch_bounds__(ADJ_REDUCE_THREADS) k_adj_reduce(const double* __restrict__ acc,
                                                                  const uint32_t* __restrict__ pbase, int s0,
                                                                  int n_scenes, uint32_t n, double* part) {
  __shared__ double red[ADJ_REDUCE_THREADS / 32];
  const int s = s0 + (int)blockIdx.z, c = blockIdx.y;
  const uint32_t p0 = pbase[s], p1 = s + 1 < n_scenes ? pbase[s + 1] : n;
  double v = 0.0;
  for (uint64_t p = p0 + blockIdx.x * ADJ_REDUCE_THREADS + threadIdx.x; p < p1;
       p += (uint64_t)gridDim.x * ADJ_REDUCE_THREADS)
    v += acc[(size_t)c * n + p];
  v = adj_block_sum(v, red);
  if (threadIdx.x == 0) part[((size_t)s * ADJ_NACC + c) * gridDim.x + blockIdx.x] = v;
}

__global__ void k_adj_reduce_shares(const double* __restrict__ part, int shares, int n_sums, double* out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_sums) return;
  double v = 0.0;
  for (int q = 0; q < shares; ++q) v += part[(size_t)k * shares + q];
  out[k] = v;
}

}  // namespace psb
