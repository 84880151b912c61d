// ps_mesh.cuh — triangle container on a binned mesh.
//
// Replaces the reference's dense N x P container
// (src/ParticleStabilizerCUDA/PolygonContainerCUDA.cpp:130-226 and
// PolygonContainerCUDA_kernels.cu:155-294: a bool[N*P] intersection matrix
// and five launches per step).  Triangles are binned once, at set-up: a bin
// lists, in ascending index, every triangle that a sphere whose centre lies
// in the bin can touch, its radius being at most sp.mesh_reach.  A sphere
// therefore walks the one list of its centre's bin and adds its hits as it
// meets them, in ascending triangle index (the order of the oracle), with
// the same operations as the reference:
//   v <- mean over hits of e * (v - 2 (v.n) n)
//   x <- x + sum over hits of -(r - dot(-n, x - v0)) n
// all evaluated on the pre-container state, for any number of hits.
//
// What bounds it: the chain bin -> index -> box -> triangle of the few
// spheres near the wall.  262,144 spheres filling the 20,200-triangle funnel,
// FP32 contact launch: 84.5 us with bins by the triangles' boxes alone (up to
// eight bins per sphere, each triangle in several of them, hits sorted
// afterwards), 45.9 us with these lists.
#pragma once

#include "ps_device.cuh"

namespace psb {

// Every scene's binned triangles.
struct MeshView {
  const void* tri;     // three vec4 per triangle: v0, v1, v2, unit normal
  const void* aabb;    // two vec4 per triangle: min xyz, max xyz and (w) how far its vertices may be off its plane
  const uint32_t* bin_offset;  // CSR offsets per bin (+1)
  const uint32_t* bin_tri;     // triangle ids (global)
  uint32_t n_tri;      // triangles over all scenes
  uint32_t n_bins;     // bins over all scenes (bin_offset holds n_bins + 1)
  uint32_t n_bin_tri;  // entries of bin_tri
};

template <class T>
__device__ __forceinline__ T dot3(T ax, T ay, T az, T bx, T by, T bz) {
  using A = Ar<T>;
  return A::fma(az, bz, A::fma(ay, by, A::mul(ax, bx)));
}

template <class T>
struct V3 {
  T x, y, z;
};

template <class T>
__device__ __forceinline__ V3<T> v3sub(V3<T> a, V3<T> b) {
  using A = Ar<T>;
  return {A::sub(a.x, b.x), A::sub(a.y, b.y), A::sub(a.z, b.z)};
}
template <class T>
__device__ __forceinline__ T v3dot(V3<T> a, V3<T> b) {
  return dot3<T>(a.x, a.y, a.z, b.x, b.y, b.z);
}

// closest point on segment ab (PolygonContainerCUDA_kernels.cu:101-112)
template <class T>
__device__ __forceinline__ V3<T> seg_closest(V3<T> p, V3<T> a, V3<T> b) {
  using A = Ar<T>;
  const V3<T> ab = v3sub(b, a), ap = v3sub(p, a);
  T t = A::div(v3dot(ap, ab), v3dot(ab, ab));
  t = t < T(1) ? t : T(1);
  t = t > T(0) ? t : T(0);
  return {A::fma(ab.x, t, a.x), A::fma(ab.y, t, a.y), A::fma(ab.z, t, a.z)};
}

// getClosestPointOnPolygonKernelFunc (PolygonContainerCUDA_kernels.cu:114-153)
template <class T>
__device__ __forceinline__ V3<T> tri_closest(V3<T> a, V3<T> b, V3<T> c, V3<T> n, V3<T> p, int edge_quirk) {
  using A = Ar<T>;
  const T ip = v3dot(v3sub(p, a), n);
  const V3<T> q = {A::fma(-n.x, ip, p.x), A::fma(-n.y, ip, p.y), A::fma(-n.z, ip, p.z)};
  {
    const V3<T> v0 = v3sub(c, a), v1 = v3sub(b, a), v2 = v3sub(q, a);
    const T d00 = v3dot(v0, v0), d01 = v3dot(v0, v1), d02 = v3dot(v0, v2);
    const T d11 = v3dot(v1, v1), d12 = v3dot(v1, v2);
    const T inv = A::div(T(1), A::fma(d00, d11, -A::mul(d01, d01)));
    const T u = A::mul(A::fma(d11, d02, -A::mul(d01, d12)), inv);
    const T v = A::mul(A::fma(d00, d12, -A::mul(d01, d02)), inv);
    if ((u >= T(0)) && (v >= T(0)) && (A::add(u, v) <= T(1))) return q;
  }
  const V3<T> e0 = seg_closest(p, a, b), e1 = seg_closest(p, b, c), e2 = seg_closest(p, c, a);
  T s0, s1, s2;
  if (edge_quirk) {
    s0 = v3dot(p, e0);
    s1 = v3dot(p, e1);
    s2 = v3dot(p, e2);
  } else {
    const V3<T> d0 = v3sub(p, e0), d1 = v3sub(p, e1), d2 = v3sub(p, e2);
    s0 = v3dot(d0, d0);
    s1 = v3dot(d1, d1);
    s2 = v3dot(d2, d2);
  }
  V3<T> r = e0;
  T best = s0;
  if (s1 < best) { best = s1; r = e1; }
  if (s2 < best) { best = s2; r = e2; }
  return r;
}

template <class T>
__device__ __forceinline__ int32_t mesh_axis(T x, T lo, T iv, int32_t nb) {
  using A = Ar<T>;
  const T q = A::div(A::sub(x, lo), iv);
  if (!(q > T(0))) return 0;
  if (q >= (T)nb) return nb - 1;
  return (int32_t)q;
}

template <class T>
struct Triangle {
  V3<T> a, b, c, n;
};
template <class T>
__device__ __forceinline__ Triangle<T> triangle(const MeshView& mv, uint32_t t) {
  const vec4_t<T>* q = static_cast<const vec4_t<T>*>(mv.tri) + 3 * (size_t)t;
  const vec4_t<T> u = ld4<T>(q), v = ld4<T>(q + 1), w = ld4<T>(q + 2);
  return {{u.x, u.y, u.z}, {u.w, v.x, v.y}, {v.z, v.w, w.x}, {w.y, w.z, w.w}};
}

// Closed test of triangle t's AABB against [lo, hi] (isIntersectedKernel :191-197).
template <class T>
__device__ __forceinline__ bool in_box(const MeshView& mv, uint32_t t, const V3<T>& lo, const V3<T>& hi,
                                       T* off_plane = nullptr) {
  const vec4_t<T>* q = static_cast<const vec4_t<T>*>(mv.aabb) + 2 * (size_t)t;
  const vec4_t<T> mn = ld4<T>(q), mx = ld4<T>(q + 1);
  if (off_plane != nullptr) *off_plane = mx.w;
  return lo.x <= mx.x && hi.x >= mn.x && lo.y <= mx.y && hi.y >= mn.y && lo.z <= mx.z && hi.z >= mn.z;
}

// Sums over the hits of one sphere, from its pre-container state.
template <class T>
struct MeshSums {
  V3<T> v, x;
  uint32_t hits;
};

// Whether the sphere touches the triangle, and what a hit adds: the reflected
// velocity (calcModifiedVelocitySumKernel :235) and the position correction
// (calcPosModificationAmountKernel :276-281).
template <class T>
__device__ __forceinline__ bool mesh_hit(const Triangle<T>& g, const V3<T>& c, T r, const SceneParams<T>& sp) {
  const V3<T> rel = v3sub(tri_closest<T>(g.a, g.b, g.c, g.n, c, sp.edge_quirk), c);
  return v3dot(rel, rel) < Ar<T>::mul(r, r);
}
template <class T>
__device__ __forceinline__ void mesh_add(const Triangle<T>& g, const V3<T>& c, T r, const vec4_t<T>& V, T e,
                                         MeshSums<T>& m) {
  using A = Ar<T>;
  const V3<T> n = g.n;
  const T vn2 = A::mul(T(2), dot3<T>(V.x, V.y, V.z, n.x, n.y, n.z));
  m.v.x = A::fma(e, A::fma(-vn2, n.x, V.x), m.v.x);
  m.v.y = A::fma(e, A::fma(-vn2, n.y, V.y), m.v.y);
  m.v.z = A::fma(e, A::fma(-vn2, n.z, V.z), m.v.z);
  const T dtp = dot3<T>(-n.x, -n.y, -n.z, A::sub(c.x, g.a.x), A::sub(c.y, g.a.y), A::sub(c.z, g.a.z));
  const T sc = A::sub(r, dtp);
  m.x.x = A::fma(-sc, n.x, m.x.x);
  m.x.y = A::fma(-sc, n.y, m.x.y);
  m.x.z = A::fma(-sc, n.z, m.x.z);
  ++m.hits;
}

// f(triangle id) for the lists of every bin that [lo, hi] touches, bin by bin.
template <class T, class F>
__device__ __forceinline__ void mesh_bins(const V3<T>& lo, const V3<T>& hi, const SceneParams<T>& sp,
                                          const MeshView& mv, uint32_t* err, F f) {
  // outside the bins on some axis (or not a number): no triangle is in reach
  if (!(hi.x >= sp.mesh_lo[0] && lo.x <= sp.mesh_hi[0] && hi.y >= sp.mesh_lo[1] && lo.y <= sp.mesh_hi[1] &&
        hi.z >= sp.mesh_lo[2] && lo.z <= sp.mesh_hi[2]))
    return;
  const int32_t x0 = mesh_axis<T>(lo.x, sp.mesh_lo[0], sp.mesh_iv, sp.mesh_nb[0]);
  const int32_t y0 = mesh_axis<T>(lo.y, sp.mesh_lo[1], sp.mesh_iv, sp.mesh_nb[1]);
  const int32_t z0 = mesh_axis<T>(lo.z, sp.mesh_lo[2], sp.mesh_iv, sp.mesh_nb[2]);
  const int32_t x1 = mesh_axis<T>(hi.x, sp.mesh_lo[0], sp.mesh_iv, sp.mesh_nb[0]);
  const int32_t y1 = mesh_axis<T>(hi.y, sp.mesh_lo[1], sp.mesh_iv, sp.mesh_nb[1]);
  const int32_t z1 = mesh_axis<T>(hi.z, sp.mesh_lo[2], sp.mesh_iv, sp.mesh_nb[2]);
  for (int32_t x = x0; x <= x1; ++x)
    for (int32_t y = y0; y <= y1; ++y) {
      // the bins of a column are consecutive, and so are their lists
      const uint32_t col = sp.mesh_bin_base + ((uint32_t)x * (uint32_t)sp.mesh_nb[1] + (uint32_t)y) * (uint32_t)sp.mesh_nb[2];
      if (!in_bounds(col + (uint32_t)z1, mv.n_bins, err)) continue;
      const uint32_t s1 = __ldg(mv.bin_offset + col + (uint32_t)z1 + 1u);
      if (!in_bounds(s1, (uint64_t)mv.n_bin_tri + 1u, err)) continue;
      for (uint32_t s = __ldg(mv.bin_offset + col + (uint32_t)z0); s < s1; ++s) {
        const uint32_t t = __ldg(mv.bin_tri + s);
        if (in_bounds(t, mv.n_tri, err)) f(t);
      }
    }
}

// Hits of a sphere larger than the bins were made for (uploaded after them):
// the smallest id above the last one over all the bins around it, in turn.
template <class T>
__device__ __noinline__ void mesh_large(V3<T> c, T r, vec4_t<T> V, const SceneParams<T>& sp, const MeshView& mv,
                                        uint32_t* err, MeshSums<T>* m) {
  using A = Ar<T>;
  const V3<T> lo = {A::sub(c.x, r), A::sub(c.y, r), A::sub(c.z, r)};
  const V3<T> hi = {A::add(c.x, r), A::add(c.y, r), A::add(c.z, r)};
  uint32_t from = 0;
  while (true) {
    uint32_t next = 0xffffffffu;
    mesh_bins<T>(lo, hi, sp, mv, err, [&](uint32_t t) {
      if (t >= from && t < next && in_box<T>(mv, t, lo, hi) && mesh_hit<T>(triangle<T>(mv, t), c, r, sp)) next = t;
    });
    if (next == 0xffffffffu) return;
    mesh_add<T>(triangle<T>(mv, next), c, r, V, sp.e_poly, *m);
    from = next + 1u;
  }
}

// The container's effect on a sphere at c, once its hits are summed.
template <class T>
__device__ __forceinline__ void mesh_apply(const MeshSums<T>& m, const V3<T>& c, vec4_t<T>& P, vec4_t<T>& V) {
  using A = Ar<T>;
  if (m.hits > 0) {  // calcAveragedVelocityKernel: only particles with a hit
    const T hc = (T)m.hits;
    V.x = A::div(m.v.x, hc);
    V.y = A::div(m.v.y, hc);
    V.z = A::div(m.v.z, hc);
  }
  // modifyPositionKernel adds the (possibly zero) correction to every particle
  P.x = A::add(c.x, m.x.x);
  P.y = A::add(c.y, m.x.y);
  P.z = A::add(c.z, m.x.z);
}

// Triangle container of one particle, CUDA semantics
// (PolygonContainerCUDA.cpp:130-226): every hit triangle in ascending index.
template <class T>
__device__ __forceinline__ void mesh_contacts(vec4_t<T>& P, vec4_t<T>& V, const SceneParams<T>& sp,
                                              const MeshView& mv, uint32_t* err) {
  using A = Ar<T>;
  const T r = P.w;
  const V3<T> c = {P.x, P.y, P.z};
  MeshSums<T> m = {};
  if (r <= sp.mesh_reach) {
    const V3<T> lo = {A::sub(c.x, r), A::sub(c.y, r), A::sub(c.z, r)};
    const V3<T> hi = {A::add(c.x, r), A::add(c.y, r), A::add(c.z, r)};
    mesh_bins<T>(c, c, sp, mv, err, [&](uint32_t t) {
      if (!in_box<T>(mv, t, lo, hi)) return;
      const Triangle<T> g = triangle<T>(mv, t);
      if (mesh_hit<T>(g, c, r, sp)) mesh_add<T>(g, c, r, V, sp.e_poly, m);
    });
  } else {
    mesh_large<T>(c, r, V, sp, mv, err, &m);
  }
  mesh_apply<T>(m, c, P, V);
}

// Ascending ids of the triangles that a sphere at P may touch once each of
// its coordinates has moved by up to `skin` (plane and box within reach), at
// most CAP of them; the count, or more than CAP when they are not all there.
template <class T, int CAP>
__device__ __forceinline__ uint32_t mesh_candidates(const vec4_t<T>& P, T skin, const SceneParams<T>& sp,
                                                    const MeshView& mv, uint32_t* err, uint32_t (&ids)[CAP]) {
  if (!(P.w <= sp.mesh_reach)) return CAP + 1;
  const T reach = P.w + skin, along = (P.w + T(1.75) * skin) * T(1.001);  // sqrt(3) skin along a normal
  const V3<T> lo = {P.x - reach, P.y - reach, P.z - reach}, hi = {P.x + reach, P.y + reach, P.z + reach};
  uint32_t n = 0;
  mesh_bins<T>({P.x - skin, P.y - skin, P.z - skin}, {P.x + skin, P.y + skin, P.z + skin}, sp, mv, err,
               [&](uint32_t t) {
                 T off;  // (with the box: from the vertices here, funnels took 0.4 % longer)
                 if (n > CAP || !in_box<T>(mv, t, lo, hi, &off)) return;
                 const Triangle<T> g = triangle<T>(mv, t);
                 const T h = (P.x - g.a.x) * g.n.x + (P.y - g.a.y) * g.n.y + (P.z - g.a.z) * g.n.z;
                 if (fabs(h) > along + off) return;  // (a triangle without a normal stays)
                 uint32_t k = n;  // several bins: not in order, and not once
                 while (k > 0u && ids[k - 1] > t) --k;
                 if (k > 0u && ids[k - 1] == t) return;
                 if (n < CAP)
                   for (uint32_t q = n; q > k; --q) ids[q] = ids[q - 1];
                 if (n < CAP) ids[k] = t;
                 ++n;
               });
  return n;
}

}  // namespace psb
