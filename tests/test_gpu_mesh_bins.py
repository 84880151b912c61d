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
