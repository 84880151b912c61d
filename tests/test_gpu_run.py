"""Calls of many steps (one launch, lists between grid rebuilds) against the
step kernels, which ps_profile_steps always takes: the same scenes in the same
calls must give the same state and the same buckets bit for bit."""
import numpy as np
import pytest

import psb200
from psb200 import scenes
from oracle import ps_oracle as O

pytestmark = pytest.mark.gpu


def crowd(n_small: int = 300, seed: int = 51) -> scenes.Scene:
    """A large sphere inside a shell of small ones that touch it and each
    other: more neighbours than a list holds."""
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n_small, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    r = np.full(n_small + 1, 0.003)
    r[0] = 0.02
    pos = np.concatenate([np.zeros((1, 3)), d * rng.uniform(0.0229, 0.024, size=(n_small, 1))]) + 0.1
    st = np.zeros((n_small + 1, 8))
    st[:, :3] = pos
    st[:, 3:6] = rng.normal(0, 0.05, size=(n_small + 1, 3))
    st[:, 6] = r
    st[:, 7] = scenes.mass_of(r, 1000.0)
    return scenes.Scene(st, (0, 0, 0), (0.2, 0.2, 0.2), (0, 0, -9.8), (0.5,) * 6, 0.02, 0.3, 1e-5)


def faster(sc: scenes.Scene, f: float) -> scenes.Scene:
    st = sc.state.copy()
    st[:, 3:6] *= f
    return sc.copy(state=st)


SCENES = {
    "pile": lambda: [scenes.pile(1500, seed=11, k_spring=1.0)],
    "settle": lambda: [scenes.settle_pile(side=10)],
    "warm": lambda: [faster(scenes.pile(3000, seed=31, k_spring=1.0), 5.0)],      # spheres leave their cells
    "fast": lambda: [faster(scenes.pile(1000, seed=21, k_spring=1.0), 500.0)],    # no list would last
    "diverging": lambda: [scenes.pile(1000, seed=14, k_spring=1e4)],              # non-finite states
    "crowd": lambda: [crowd()],
    "cells of 2 r_max": lambda: [scenes.pile(2000, seed=32, k_spring=1.0).copy(interval=0.012)],
    "wide cells": lambda: [scenes.pile(2000, seed=33, k_spring=1.0).copy(interval=0.03)],
    "batch": lambda: [scenes.pile(300, seed=15, k_spring=0.5), scenes.pile(1, seed=25), scenes.settle_pile(side=8),
                      scenes.pile(1, seed=25).copy(state=np.zeros((0, 8))), scenes.pile(900, seed=16, k_spring=2.0),
                      scenes.pile(64, seed=17, k_spring=1e4)],
    "box mesh": lambda: [scenes.box_mesh_scene()],
    "funnel": lambda: [scenes.funnel_wall_scene(1500)],
    "fan": lambda: [scenes.fan_floor_scene()],                                    # more triangles than a sphere's list
    "fine mesh": lambda: [scenes.box_mesh_scene(100, seed=46).copy(tri=scenes.box_container(n=16))],
    "more than a CTA's share aside": lambda: [faster(scenes.pile(70000, seed=34, k_spring=1.0), 20.0)],
    "batch with a mesh": lambda: [scenes.pile(300, seed=28, k_spring=1.0), scenes.box_mesh_scene(),
                                  scenes.pile(500, seed=29, k_spring=1.0)],
}


def both(scs, prec, calls):
    out = []
    for name in ("step", "profile_steps"):
        with psb200.Simulation(scs, prec) as sim:
            sim.set_state()
            for n in calls:
                getattr(sim, name)(n)
            out.append((sim.get_state(), *sim.buckets()))
    return out


def same(a, b):
    return all(np.array_equal(x, y, equal_nan=x.dtype.kind == "f") for x, y in zip(a, b))


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("name", list(SCENES))
def test_runs_equal_step_kernels(need_gpu, name, prec):
    # the first probe, a call shorter than a run, a call past it, one of several launches
    a, b = both(SCENES[name](), prec, (60, 3, 9, 700))
    assert same(a, b)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 1025])
@pytest.mark.parametrize("steps", [8, 12, 13])
def test_runs_of_few_spheres_and_steps(need_gpu, n, steps):
    sc = scenes.pile(max(n, 8), seed=40 + n, k_spring=1.0)
    a, b = both([sc.copy(state=sc.state[:n])], "f32", (steps,))
    assert same(a, b)


def test_run_equals_oracle(need_gpu):
    sc = faster(scenes.pile(800, seed=12, k_spring=1.0), 3.0)
    with psb200.Simulation(sc, "f32") as sim:
        sim.set_state()
        sim.step(120)
        got = sim.get_state()
    assert np.array_equal(got.astype(np.float32), O.run(sc, 120, "f32"))


@pytest.mark.parametrize("skin", [None, 0.2])
def test_adjoint_of_runs_whose_order_is_an_earlier_grids(need_gpu, skin):
    # spheres change cells inside the blocks, so a block does not end in the
    # order of its last build; blocks of 5 steps take the step kernels and
    # their recording, whose sums differ in order alone
    sc = faster(scenes.pile(1000, seed=24, k_spring=1.0), 20.0)
    out = []
    for every in (5, 50):
        with psb200.Simulation(sc, "f64") as sim:
            sim.set_state()
            if skin is not None and every == 50:
                sim.set_neighbor_lists(skin, 64)
            sim.forward_checkpointed(100, every)
            final = sim.get_state()
            grads, g0 = sim.backward(psb200.height_loss(final)[1])
            out.append((final, grads[0], g0))
    assert np.array_equal(out[0][0], out[1][0])
    for k in (1, 2):
        np.testing.assert_allclose(out[0][k], out[1][k], rtol=1e-9, atol=1e-10 * np.abs(out[0][k]).max())


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("name", ["pile", "fast", "crowd", "batch", "cells of 2 r_max"])
def test_backward_on_recorded_runs(need_gpu, name, prec):
    """The backward pass recomputes blocks as recorded runs, or on the grid
    where lists do not last (fast) or overflow (crowd): blocks of 40 steps
    against blocks of 7, which are always recomputed on the grid, and two
    passes of the same against each other."""
    scs = SCENES[name]()
    if name == "batch":
        scs = scs[:-1]  # without the scene that diverges
    out = []
    for every in (7, 40):
        with psb200.Simulation(scs, prec) as sim:
            sim.set_state()
            sim.forward_checkpointed(84, every)
            g = psb200.height_loss(sim.get_state())[1]
            first, again = sim.backward(g), sim.backward(g)
            assert all(np.array_equal(x, y) for x, y in zip(first[0], again[0])) and np.array_equal(first[1], again[1])
            out.append(first)
    tol = 1e-9 if prec == "f64" else 2e-4
    for x, y in zip([*out[0][0], out[0][1]], [*out[1][0], out[1][1]]):
        np.testing.assert_allclose(x, y, rtol=tol, atol=tol * max(np.abs(x).max(), 1e-300))


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("n", [1, 31, 255, 257, 2000])
def test_statistics_at_the_edges_of_the_reduction(need_gpu, prec, n):
    sc = scenes.pile(max(n, 8), seed=60 + n, k_spring=1.0)
    sc = sc.copy(state=sc.state[:n])
    with psb200.Simulation([scenes.pile(300, seed=61), sc], prec) as sim:
        sim.set_state()
        sim.step(9)
        got = [sim.stats(1) for _ in range(2)]
        state = sim.get_state()[300:]
    o = O.stats(state)
    for s in got:
        assert s.n_collided == o.n_collided
        assert s.max_overlap == pytest.approx(o.max_overlap, rel=1e-12, abs=0)
        assert s.kinetic_energy == pytest.approx(o.kinetic_energy, rel=1e-12)
        assert list(s.min_pos) == list(o.min_pos) and list(s.max_pos) == list(o.max_pos)


@pytest.mark.parametrize("cap", [1, 31, 33, 64, 255, 4000])
def test_set_lists_of_any_capacity(need_gpu, cap):
    # shorter than the lists, one entry per lane and more, beyond the count word
    sc = faster(crowd(200), 30.0)
    want, _ = both([sc], "f32", (90, 40))
    with psb200.Simulation(sc, "f32") as sim:
        sim.set_state()
        sim.set_neighbor_lists(0.3, cap)
        sim.step(90)
        sim.step(40)
        got = (sim.get_state(), *sim.buckets())
        overflows = sim.list_stats()[1]
    assert same(got, want)
    assert (overflows > 0) == (cap < 200)  # all 200 small spheres are neighbours of the large one


def heap(k: int, n: int = 8000) -> scenes.Scene:
    """k spheres on top of one another, all in contact until their collisions
    part them, among n slow ones."""
    sc = scenes.pile(n, seed=81, k_spring=1e-4)
    st = sc.state.copy()
    st[:, 3:6] *= 0.02
    st[:k, :3] = st[n // 2, :3] + np.random.default_rng(82).normal(0, 2e-4, size=(k, 3))
    return sc.copy(state=st, dt=1e-6)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("k", [32, 33, 34, 64, 65, 66, 97, 400])
def test_lists_shorter_than_the_spheres_in_contact(need_gpu, k, prec):
    # contacts of a sphere beyond its list are taken 32 at a time; 400 such
    # spheres are too many, and the run goes on without lists
    sc = heap(k)
    want = both([sc], prec, (40, 9))[1]  # of the step kernels
    for skin in (0.0, 0.05):
        with psb200.Simulation(sc, prec) as sim:
            sim.set_state()
            sim.set_neighbor_lists(skin, 16)
            sim.step(40)
            sim.step(9)
            got = (sim.get_state(), *sim.buckets())
            overflows = sim.list_stats()[1]
        assert same(got, want)
        assert skin == 0.0 or overflows > 0
