"""The triangle bins against the oracle where their lists are special: spheres
larger than the bins were made for (a later upload), spheres beside and above
the bins, a mesh coarser and one finer than a bin."""
import numpy as np
import pytest

import psb200
from psb200 import scenes
from oracle import ps_oracle as O

pytestmark = pytest.mark.gpu


def same(got, want, prec):
    want = want.astype(np.float64)
    return np.array_equal(got.astype(np.float32) if prec == "f32" else got, want.astype(np.float32) if prec == "f32" else want)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("steps", [1, 20])
def test_spheres_larger_than_the_first_upload(need_gpu, prec, steps):
    # cell 0.03: radii up to 0.015 may be uploaded later; the bins are made for 2.2 * 0.0042
    big = scenes.box_mesh_scene(60, seed=44).copy(interval=0.03)
    st = big.state.copy()
    st[:, 6] *= 0.35
    small = big.copy(state=st)
    with psb200.Simulation(small, prec) as sim:
        sim.set_state()
        sim.set_state(big.state)
        sim.step(steps)
        got = sim.get_state()
    assert same(got, O.run(big, steps, prec), prec)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("n", [1, 12])
def test_coarse_and_fine_triangles(need_gpu, prec, n):
    # two triangles a face (many bins each) and 288 (several triangles a bin)
    sc = scenes.box_mesh_scene(100, seed=45).copy(tri=scenes.box_container(n=n))
    st = sc.state.copy()
    st[:5, 0] = 0.5                       # beside the bins
    st[5:10, 2] = np.linspace(0.26, 0.9, 5)  # above them
    st[10:15, 0] = -0.0999                # centre within a thousandth of a radius of the wall
    sc = sc.copy(state=st, widen_domain=1)
    with psb200.Simulation(sc, prec) as sim:
        sim.set_state()
        sim.step(25)
        got = sim.get_state()
    assert same(got, O.run(sc, 25, prec), prec)


def flat_triangles_scene(seed: int, kind: str, n: int = 200, length: float = 0.12) -> scenes.Scene:
    """Triangles without area among a box's, and a small sphere on each."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(-0.04, 0.04, (n, 3)) + (0.0, 0.0, 0.12)
    d = rng.normal(size=(n, 3))
    d *= length / 2 / np.linalg.norm(d, axis=1)[:, None]
    a -= d / 2
    third = {"collinear": a + 0.37 * d, "two equal corners": a, "sliver": a + 0.37 * d + rng.normal(0, 1e-12, (n, 3))}[kind]
    off = rng.normal(size=(n, 3))
    off *= 0.001 / np.linalg.norm(off, axis=1)[:, None]
    base = scenes.box_mesh_scene()
    st = np.zeros((n, 8))
    st[:, :3] = a + rng.uniform(0.0, 1.0, n)[:, None] * d + off
    st[:, 3:6] = rng.normal(0, 0.05, (n, 3))
    st[:, 6] = 0.002
    st[:, 7] = scenes.mass_of(st[:, 6], 1000.0)
    return base.copy(state=st, tri=np.concatenate([base.tri, np.concatenate([a, a + d, third], axis=1)]), k_spring=1e-6,
                     dt=1e-6)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("kind", ["collinear", "two equal corners", "sliver"])
@pytest.mark.parametrize("steps,skin", [(1, 0.0), (12, 0.0), (12, 0.2)])
def test_triangles_without_area(need_gpu, kind, steps, skin, prec):
    # their normals are rounding, or not numbers, but their edges are touched all the same
    sc = flat_triangles_scene(3, kind)
    with psb200.Simulation(sc, prec) as sim:
        sim.set_state()
        sim.set_neighbor_lists(skin, 64)
        sim.step(steps)
        got = sim.get_state()
    want = O.run(sc, steps, prec)
    assert np.array_equal(got.astype(want.dtype), want, equal_nan=True)
