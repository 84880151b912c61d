"""Performance cases of the DEM library: what programs that use it have it do.

Every case goes through the package's public entry points (psb200, the ctypes
binding of the C ABI).  The sizes are those of the repository's own scenes
(psb200/scenes.py) and benchmark, and odd ones between them.  A pass over a
prepared simulation starts from a saved state (the first checkpoint slot), so
that every pass does the same steps, and ends with the state in the program's
own host buffer, which is where a user of the library gets results.

The listed cases:

  whole_small_f64   one runSimulateCUDA-style call on host arrays (create, upload, steps, download, destroy) of
                    4,096 spheres in double precision: what a program that calls the library once does
  steps_small_f32   the same lattice kept on the GPU, 500 steps a call: small scenes, where launches and latency count
  settle_mid_f32    the settling loop: 4 times 50 steps and the statistics that decide whether the pile is at rest
  bench_1m_f32      the 1M-sphere box exactly as the benchmark runs it (spring 5e4, blocks of 100 steps)
  box_1m_f64        the 1M-sphere box with a spring that the scheme integrates stably, in double precision
  pile_1m_f32       a million spheres packed in contact, single precision: the state that long runs end in
  lists_400k_f32    neighbour-list mode on a sparse box scene
  funnel_262k_f32   spheres filling the 20,200-triangle funnel, outer ones against its wall
  batch_256_f32     256 independent scenes of 1,024 to 65,536 spheres in one simulation
  grad_65k_f32      forward with checkpoints and the backward pass of a settling loss, 65,536 spheres in contact
  e2e_262k_f32      upload of a new state, 20 steps, download: a host program that owns the state
  scan_8m           the exclusive prefix sum on its own, at the cell count of the 1M-sphere box
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "particle-stabilizer_b200", "python"))
import psb200  # noqa: E402
from psb200 import scenes  # noqa: E402


def listed():
    return [
        {"name": "whole_small_f64", "kind": "whole", "scene": "lattice", "n": 4096, "steps": 200, "precision": "f64"},
        {"name": "steps_small_f32", "kind": "steps", "scene": "lattice", "n": 4096, "steps": 500, "precision": "f32"},
        {"name": "settle_mid_f32", "kind": "settle", "scene": "pile", "n": 30011, "steps": 200, "precision": "f32"},
        {"name": "bench_1m_f32", "kind": "steps", "scene": "box_hard", "n": 1 << 20, "steps": 100, "precision": "f32"},
        {"name": "box_1m_f64", "kind": "steps", "scene": "box", "n": 1 << 20, "steps": 50, "precision": "f64"},
        {"name": "pile_1m_f32", "kind": "steps", "scene": "pile", "n": 1000003, "steps": 100, "precision": "f32"},
        {"name": "lists_400k_f32", "kind": "lists", "scene": "box", "n": 400009, "steps": 200, "precision": "f32"},
        {"name": "funnel_262k_f32", "kind": "steps", "scene": "funnel", "n": 262144, "steps": 100, "precision": "f32"},
        {"name": "batch_256_f32", "kind": "steps", "scene": "batch", "n": 256, "steps": 100, "precision": "f32"},
        {"name": "grad_65k_f32", "kind": "grad", "scene": "pile", "n": 65536, "steps": 100, "precision": "f32"},
        {"name": "e2e_262k_f32", "kind": "e2e", "scene": "box", "n": 262147, "steps": 20, "precision": "f32"},
        {"name": "scan_8m", "kind": "scan", "scene": "", "n": 7953877, "steps": 1, "precision": ""},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: any kind, sizes spread over their logarithm."""
    kind = rng.choice(["whole", "steps", "steps", "steps", "settle", "lists", "funnel", "batch", "grad", "e2e", "scan"])
    prec = rng.choice(["f32", "f32", "f64"])
    if kind == "whole":
        return {"kind": kind, "scene": "lattice", "n": _log_int(rng, 500, 20000), "steps": rng.randint(50, 400),
                "precision": prec}
    if kind == "steps":
        n = _log_int(rng, 1000, 1000000)
        scene = rng.choice(["lattice", "pile"]) if n <= 20000 else rng.choice(["box", "pile"])
        return {"kind": kind, "scene": scene, "n": n, "steps": rng.randint(20, 100), "precision": prec}
    if kind == "settle":
        return {"kind": kind, "scene": "pile", "n": _log_int(rng, 2000, 200000), "steps": 4 * rng.randint(10, 50),
                "precision": prec}
    if kind == "lists":
        return {"kind": kind, "scene": rng.choice(["box", "pile"]), "n": _log_int(rng, 5000, 600000),
                "steps": rng.randint(50, 200), "precision": prec}
    if kind == "funnel":
        return {"kind": "steps", "scene": "funnel", "n": _log_int(rng, 5000, 262144), "steps": rng.randint(20, 100),
                "precision": prec}
    if kind == "batch":
        return {"kind": "steps", "scene": "batch", "n": _log_int(rng, 3, 200), "steps": rng.randint(20, 100),
                "precision": "f32"}
    if kind == "grad":
        return {"kind": kind, "scene": "pile", "n": _log_int(rng, 1000, 65536), "steps": rng.randint(20, 100),
                "precision": prec}
    if kind == "e2e":
        return {"kind": kind, "scene": "box", "n": _log_int(rng, 3000, 400000), "steps": rng.randint(5, 20),
                "precision": prec}
    return {"kind": "scan", "scene": "", "n": _log_int(rng, 1000, 16000000), "steps": 1, "precision": ""}


# ---- the scenes ------------------------------------------------------------------
def _lattice(n, seed):
    """The 4,096-sphere lattice scene, at any count (the first n sites of the smallest cube that holds them)."""
    side = 1
    while side ** 3 < n:
        side += 1
    sc = scenes.lattice_c1(seed, side)
    st = sc.state[:n].copy()
    st[:, 6] = 0.16 / side  # radius 0.01 at 16 per edge
    st[:, 7] = scenes.mass_of(st[:, 6], 1000.0)
    # at rest it meets nothing for thousands of steps: give it the speeds of one that moves already
    st[:, 3:6] = np.random.default_rng(seed + 77).normal(0.0, 0.3, size=(n, 3))
    return sc.copy(state=st, k_spring=0.5 * float(st[0, 7]) / sc.dt * 0.1)


def _box(n, seed, k_spring):
    """The 1M-sphere box scene; smaller counts in a box of the same filling."""
    if n == 1 << 20:
        return scenes.c2_scene(n, seed, k_spring)
    rng = np.random.default_rng(seed)
    d = max(4, int(round((n / (4 * 0.1336)) ** (1 / 3))))
    slot, dims = 0.008, (d, d, 4 * d)
    while n > 0.9 * dims[0] * dims[1] * dims[2]:
        dims = (dims[0], dims[1], dims[2] + d)
    r = np.clip(rng.lognormal(math.log(0.002), 0.25, size=n), 0.001, 0.004)
    chosen = rng.choice(dims[0] * dims[1] * dims[2], size=n, replace=False)
    ijk = np.stack([chosen // (dims[1] * dims[2]), (chosen // dims[2]) % dims[1], chosen % dims[2]], axis=1)
    st = np.empty((n, 8))
    st[:, 0:3] = (ijk + 0.5) * slot + rng.uniform(-1.0, 1.0, size=(n, 3)) * (slot / 2 - r)[:, None]
    st[:, 3:6] = rng.normal(0.0, 0.05, size=(n, 3))
    st[:, 6] = r
    st[:, 7] = scenes.mass_of(r, 1000.0)
    return scenes.Scene(st, (0, 0, 0), tuple(slot * x for x in dims), (0, 0, -9.8), (0.7,) * 6, k_spring, 0.4, 5e-6,
                        interval=slot)


def _funnel(n, seed):
    """Spheres of radius 0.003 on a jittered lattice filling the funnel from the neck up, the outermost against the
    wall (a spring that the scheme integrates stably, as the repository's wall scene)."""
    rng = np.random.default_rng(seed)
    r, pitch = 0.003, 0.0066
    layers, count, z = [], 0, 0.31
    g = np.arange(-0.5, 0.5, pitch)
    gx, gy = (a.ravel() for a in np.meshgrid(g, g, indexing="ij"))
    rad = np.hypot(gx, gy)
    slope = math.hypot(0.7, 0.42) / 0.7  # distance along the radius of a unit distance to the cone's wall
    while count < n:
        wall = 0.08 + 0.42 * (z - 0.3) / 0.7
        keep = rad <= wall - 0.97 * r * slope
        layers.append(np.column_stack([gx[keep], gy[keep], np.full(int(keep.sum()), z)]))
        count += len(layers[-1])
        z += pitch
    pos = np.concatenate(layers)[:n] + rng.uniform(-2e-4, 2e-4, size=(n, 3))
    st = np.empty((n, 8))
    st[:, 0:3] = pos
    st[:, 3:6] = rng.normal(0.0, 0.1, size=(n, 3))
    st[:, 6] = r
    st[:, 7] = scenes.mass_of(st[:, 6], 1000.0)
    return scenes.Scene(st, (-0.5, -0.5, 0.0), (0.5, 0.5, 1.0), (0, 0, -9.8), (0.6,) * 6, 2e-2, 0.5, 5e-6,
                        tri=scenes.funnel_triangles(), widen_domain=1)


def _batch_shapes(n):
    """(spheres, box edge) of each scene of a batch: uneven, the same for every seed."""
    rng = np.random.default_rng(6)
    out = []
    for _ in range(n):
        m = int(round(math.exp(rng.uniform(math.log(1024), math.log(65536)))))
        edge = float(rng.uniform(0.2, 1.0))
        out.append((min(m, int(edge / 0.012) ** 3), edge))
    return out


def _batch(n, seed):
    """The batching workload (independent scenes of uneven counts, radii, boxes and coefficients; stable springs)."""
    rng = np.random.default_rng(seed)
    out = []
    for m, edge in _batch_shapes(n):
        slot = 0.012
        d = int(edge / slot)
        r = rng.uniform(0.002, 0.006, size=m)
        chosen = rng.choice(d ** 3, size=m, replace=False, shuffle=False)
        ijk = np.stack([chosen // (d * d), (chosen // d) % d, chosen % d], axis=1)
        st = np.empty((m, 8))
        st[:, 0:3] = (ijk + 0.5) * slot + rng.uniform(-1, 1, size=(m, 3)) * (slot / 2 - r)[:, None]
        st[:, 3:6] = rng.normal(0.0, 0.05, size=(m, 3))
        st[:, 6] = r
        st[:, 7] = scenes.mass_of(r, 1000.0)
        k = float(math.exp(rng.uniform(math.log(0.25), math.log(2.5))))
        out.append(scenes.Scene(st, (0, 0, 0), (edge,) * 3, (0, 0, -9.8),
                                tuple(float(x) for x in rng.uniform(0.3, 0.9, size=6)), k,
                                float(rng.uniform(0.3, 0.9)), 5e-6))
    return out


def _scenes(case, seed):
    n, kind = case["n"], case["scene"]
    if kind == "lattice":
        return [_lattice(n, seed)]
    if kind == "pile":
        return [scenes.pile(n, seed)]
    if kind == "box":
        return [_box(n, seed, 0.25)]
    if kind == "box_hard":
        return [_box(n, seed, 5e4)]
    if kind == "funnel":
        return [_funnel(n, seed)]
    return _batch(n, seed)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _scan_input(n, seed):
    """Cell counts: mostly empty cells, a few spheres in the others."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.poisson(torch.full((n,), 0.13, device="cuda"), generator=g).to(torch.int32)


def _loss_gradient(state):
    """dL/d(state) of the settling loss that the differentiation workload uses."""
    return psb200.height_loss(state)[1]


# ---- the passes ------------------------------------------------------------------
def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "scan":
        n = case["n"]
        s["in"] = _scan_input(n, seed)
        s["out"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["scratch"] = torch.empty(psb200.exclusive_scan_scratch_bytes(n), dtype=torch.uint8, device="cuda")
        return s
    scs = _scenes(case, seed)
    if case["kind"] == "whole":
        s["scene"] = scs[0]
        return s
    sim = psb200.Simulation(scs, case["precision"])
    sim.set_state()
    if case["kind"] == "lists":
        sim.set_neighbor_lists(0.05, 48)
    sim.checkpoint_save(0)
    sim.sync()
    s["sim"] = sim
    s["out"] = _pinned((sim.n, 8))
    if case["kind"] == "e2e":
        s["in"] = _pinned((sim.n, 8))
        s["in"][:] = scs[0].state
    if case["kind"] == "grad":
        s["every"] = max(1, case["steps"] // 4)
    return s


def run(s):
    case = s["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "scan":
        psb200.exclusive_scan_u32(s["in"].data_ptr(), s["out"].data_ptr(), case["n"], s["scratch"].data_ptr(),
                                  torch.cuda.current_stream().cuda_stream)
        return s["out"]
    if kind == "whole":
        return psb200.simulate(s["scene"], steps, case["precision"])
    sim = s["sim"]
    if kind == "e2e":
        sim.set_state(s["in"])
        sim.step(steps)
        return sim.get_state(s["out"])
    sim.checkpoint_load(0)
    if kind == "settle":
        told = []
        for _ in range(4):
            sim.step(steps // 4)
            t = sim.stats()
            told.append([t.kinetic_energy, *t.min_pos, *t.max_pos, t.max_overlap])
        return {"stats": np.array(told), "collided": t.n_collided, "state": sim.get_state(s["out"])}
    if kind == "grad":
        sim.forward_checkpointed(steps, s["every"])
        state = sim.get_state(s["out"])
        grads, g0 = sim.backward(_loss_gradient(state))
        # the parameters that the program updates are held in the simulation's precision
        real = np.float32 if case["precision"] == "f32" else np.float64
        return {"state": state, "parameters": grads[0].astype(real), "initial": g0.astype(real)}
    sim.step(steps)
    return sim.get_state(s["out"])


def _particles(case):
    if case["scene"] == "batch":
        return sum(m for m, _ in _batch_shapes(case["n"]))
    return case["n"]


def work(case):
    """A step reads the 8 reals of every sphere and writes the 6 that change, and tests each sphere against a few
    neighbours; the result crosses to the host once."""
    n = _particles(case)
    if case["kind"] == "scan":
        return {"bytes": 8 * n, "flops": n}
    real = 4 if case["precision"] == "f32" else 8
    per_step, flops = 14 * real, 100
    if case["kind"] == "grad":  # forward, recompute and reverse
        per_step, flops = 3 * per_step, 500
    return {"bytes": n * (per_step * case["steps"] + 64), "flops": n * flops * case["steps"]}


# ---- the same in 64 bits with plain torch ------------------------------------------
def _pairs(pos, r_max, scene_id):
    """(i, j) of every pair whose centres are within 2 r_max on each axis and some beyond, each pair once."""
    n = pos.shape[0]
    h = 2.0 * float(r_max) * 1.0001
    c = torch.floor((pos - pos.min(0).values) / h).long() + 1
    d = c.max(0).values + 2
    key = ((scene_id * d[0] + c[:, 0]) * d[1] + c[:, 1]) * d[2] + c[:, 2]
    skey, order = torch.sort(key)
    ii, jj = [], []
    for dx, dy, z0, z1 in ((0, 0, 0, 1), (0, 1, -1, 1), (1, -1, -1, 1), (1, 0, -1, 1), (1, 1, -1, 1)):
        base = skey + (dx * d[1] + dy) * d[2]
        lo = torch.searchsorted(skey, base + z0)
        hi = torch.searchsorted(skey, base + z1, right=True)
        if dx == 0 and dy == 0:
            lo = torch.arange(n, device=pos.device) + 1  # the rest of the own cell, and the next
        cnt = (hi - lo).clamp(min=0)
        a = torch.repeat_interleave(torch.arange(n, device=pos.device), cnt)
        b = torch.arange(a.numel(), device=pos.device) - torch.repeat_interleave(cnt.cumsum(0) - cnt, cnt) + lo[a]
        ii.append(order[a])
        jj.append(order[b])
    return torch.cat(ii), torch.cat(jj)


def _triangle_bins(tri, h, reach):
    """Triangles by the cells of edge h that their boxes, widened by `reach`, touch: (origin, dims, offsets, ids)."""
    t = tri.view(-1, 3, 3)
    lo, hi = t.min(1).values - reach, t.max(1).values + reach
    org = lo.min(0).values
    a, b = torch.floor((lo - org) / h).long(), torch.floor((hi - org) / h).long()
    dims = b.max(0).values + 1
    keys, ids = [], []
    span = (b - a).max(0).values
    for x in range(int(span[0]) + 1):
        for y in range(int(span[1]) + 1):
            for z in range(int(span[2]) + 1):
                c = a + torch.tensor([x, y, z], device=tri.device)
                ok = (c <= b).all(1)
                keys.append(((c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2])[ok])
                ids.append(torch.nonzero(ok).flatten())
    key, order = torch.sort(torch.cat(keys))
    total = int(dims.prod())
    off = torch.searchsorted(key, torch.arange(total + 1, device=tri.device))
    return org, dims, off, torch.cat(ids)[order]


def _segment(p, a, b):
    ab = b - a
    t = (((p - a) * ab).sum(1) / (ab * ab).sum(1)).clamp(0.0, 1.0)
    return a + ab * t[:, None]


def _triangles(pos, vel, r, tri, bins, h, e):
    """The triangle container: every triangle within a sphere's radius reflects its velocity (mean over them) and
    pushes it back; of the three edges the one with the smallest <centre, point> counts, as the reference has it."""
    org, dims, off, ids = bins
    c = torch.floor((pos - org) / h).long()
    inside = ((c >= 0) & (c < dims)).all(1)
    cell = torch.where(inside, (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2], torch.zeros_like(c[:, 0]))
    cnt = torch.where(inside, off[cell + 1] - off[cell], torch.zeros_like(cell))
    s = torch.repeat_interleave(torch.arange(pos.shape[0], device=pos.device), cnt)
    k = torch.arange(s.numel(), device=pos.device) - torch.repeat_interleave(cnt.cumsum(0) - cnt, cnt) + off[cell[s]]
    t = tri.view(-1, 3, 3)[ids[k]]
    p, a, b, d = pos[s], t[:, 0], t[:, 1], t[:, 2]
    nrm = torch.linalg.cross(b - a, d - a)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    q = p - nrm * ((p - a) * nrm).sum(1, keepdim=True)
    v0, v1, v2 = d - a, b - a, q - a
    d00, d01, d02 = (v0 * v0).sum(1), (v0 * v1).sum(1), (v0 * v2).sum(1)
    d11, d12 = (v1 * v1).sum(1), (v1 * v2).sum(1)
    inv = 1.0 / (d00 * d11 - d01 * d01)
    u, w = (d11 * d02 - d01 * d12) * inv, (d00 * d12 - d01 * d02) * inv
    e3 = torch.stack([_segment(p, a, b), _segment(p, b, d), _segment(p, d, a)], 1)
    pick = (e3 * p[:, None, :]).sum(2).argmin(1)
    edge = e3[torch.arange(len(pick), device=pos.device), pick]
    near = torch.where(((u >= 0) & (w >= 0) & (u + w <= 1))[:, None], q, edge)
    hit = ((near - p) ** 2).sum(1) < r[s] ** 2
    boxes = ((t.min(1).values <= p + r[s, None]) & (t.max(1).values >= p - r[s, None])).all(1)
    hit &= boxes
    s, nrm, p, a = s[hit], nrm[hit], p[hit], a[hit]
    refl = e * (vel[s] - 2.0 * (vel[s] * nrm).sum(1, keepdim=True) * nrm)
    push = -(r[s] + ((p - a) * nrm).sum(1))[:, None] * nrm
    hits = torch.zeros(pos.shape[0], dtype=pos.dtype, device=pos.device).index_add(0, s, torch.ones_like(r[s]))
    mean = torch.zeros_like(vel).index_add(0, s, refl) / hits.clamp(min=1.0)[:, None]
    return pos.index_add(0, s, push), torch.where((hits > 0)[:, None], mean, vel)


class _Exact:
    """The scenes' parameters as tensors, and one step of the scheme (functional, so that autograd follows it)."""

    def __init__(self, scs):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda x: torch.as_tensor(np.asarray(x, dtype=np.float64), device=dev)  # noqa: E731
        self.state = t(np.concatenate([s.state for s in scs]))
        self.sid = torch.repeat_interleave(torch.arange(len(scs), device=dev), torch.tensor([s.n for s in scs], device=dev))
        self.lo, self.hi = t([s.box_min for s in scs]), t([s.box_max for s in scs])
        e = t([s.e_wall for s in scs])  # zMin, zMax, xMin, xMax, yMin, yMax
        self.e_wall = e
        self.k, self.e = t([s.k_spring for s in scs]), t([s.e_sphere for s in scs])
        self.g, self.dt = t(scs[0].gravity), float(scs[0].dt)
        self.r, self.m = self.state[:, 6], self.state[:, 7]
        self.tri = t(scs[0].tri) if scs[0].tri is not None else None
        if self.tri is not None:
            self.h = 0.012
            self.bins = _triangle_bins(self.tri, self.h, float(self.r.max()) * 1.01)

    def step(self, x, v):
        r = self.r[:, None]
        x, v = x + v * self.dt, v + self.g * self.dt
        if self.tri is not None:
            x, v = _triangles(x, v, self.r, self.tri, self.bins, self.h, self.e_wall[0, 0])
        else:
            lo, hi = self.lo[self.sid], self.hi[self.sid]
            e_lo, e_hi = self.e_wall[:, [2, 4, 0]][self.sid], self.e_wall[:, [3, 5, 1]][self.sid]
            under, over = x - r < lo, x + r > hi
            v = torch.where(under, -v * e_lo, v)
            v = torch.where(over, -v * e_hi, v)
            x = torch.where(over, hi - r, torch.where(under, lo + r, x))
        with torch.no_grad():
            i, j = _pairs(x, self.r.max(), self.sid)
            near = ((x[i] - x[j]) ** 2).sum(1) < (self.r[i] + self.r[j]) ** 2
            i, j = i[near], j[near]
        d, u = x[i] - x[j], v[i] - v[j]
        dist = d.norm(dim=1)
        ov = self.r[i] + self.r[j] - dist
        ud = (u * d).sum(1)
        k, e, mi, mj = self.k[self.sid[i]], self.e[self.sid[i]], self.m[i], self.m[j]
        damp = 2.0 * e * ud / ((mi + mj) * dist * dist)
        fi, fj = k * ov / (dist * mi) - mj * damp, k * ov / (dist * mj) - mi * damp
        v = v.index_add(0, i, fi[:, None] * d).index_add(0, j, -fj[:, None] * d)
        return x, v

    def stats(self, x, v):
        i, j = _pairs(x, self.r.max(), self.sid)
        ov = (self.r[i] + self.r[j] - (x[i] - x[j]).norm(dim=1)).max() if len(i) else torch.zeros((), device=x.device)
        r = self.r[:, None]
        return [float((0.5 * self.m * (v * v).sum(1)).sum()), *(x - r).min(0).values.tolist(),
                *(x + r).max(0).values.tolist(), max(0.0, float(ov))]

    def records(self, x, v):
        return torch.cat([x, v, self.state[:, 6:]], 1).cpu().numpy()


def exact(case, seed):
    if case["kind"] == "scan":
        return None  # whole numbers
    if case["scene"] == "box_hard":
        return None  # this spring amplifies every rounding without bound: no value in another precision compares
    scs = _scenes(case, seed)
    E = _Exact(scs)
    x, v = E.state[:, 0:3], E.state[:, 3:6]
    if case["kind"] == "grad":
        E.k.requires_grad_(True)
        E.e.requires_grad_(True)
        E.e_wall.requires_grad_(True)
        x = x.clone().requires_grad_(True)
        v = v.clone().requires_grad_(True)
        x1, v1 = x, v
        for _ in range(case["steps"]):
            x1, v1 = E.step(x1, v1)
        state = E.records(x1.detach(), v1.detach())
        w = 2.0 * math.pi / 0.5  # the settling loss: mean (z - h(x))^2 with h(x) = 0.1 + 0.02 sin(w x)
        ((x1[:, 2] - (0.1 + 0.02 * torch.sin(w * x1[:, 0]))) ** 2).mean().backward()
        real = np.float32 if case["precision"] == "f32" else np.float64
        par = torch.cat([E.k.grad, E.e.grad, E.e_wall.grad[0]]).cpu().numpy()
        return {"state": state, "parameters": par, "initial": torch.cat([x.grad, v.grad], 1).cpu().numpy()}
    with torch.no_grad():
        told = []
        for k in range(case["steps"]):
            x, v = E.step(x, v)
            if case["kind"] == "settle" and (k + 1) % (case["steps"] // 4) == 0:
                told.append(E.stats(x, v))
        if case["kind"] == "settle":
            return {"stats": np.array(told), "collided": None, "state": E.records(x, v)}
        return E.records(x, v)
