"""Sequences of calls on one simulation whose later calls depend on what the
earlier ones left on the device: grids resized between runs, and the like.
States are compared bit for bit with the oracle or with the step kernels,
which ps_profile_steps always takes."""
import numpy as np
import pytest

import psb200
from psb200 import scenes
from oracle import ps_oracle as O

pytestmark = pytest.mark.gpu


def same(got, want, prec):
    return np.array_equal(got.astype(np.float32) if prec == "f32" else got, want, equal_nan=True)


def sparse_pile(seed: int) -> scenes.Scene:
    """Spheres in contact in a box of many more grid tiles than sphere blocks."""
    return scenes.pile(1000, seed=seed, k_spring=1.0).copy(box_max=(0.6, 0.6, 0.6))


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("lists_first", [True, False])
@pytest.mark.parametrize("make", [scenes.lattice_c1, lambda: sparse_pile(71)], ids=["lattice", "sparse pile"])
def test_cell_size_changed_between_runs(need_gpu, make, lists_first, prec):
    # the tuner's grids have other numbers of CTAs than the first one
    sc = make()
    with psb200.Simulation(sc, prec) as sim:
        sim.set_state()
        if lists_first:
            sim.set_neighbor_lists(0.1, 64)
        sim.step(60)
        sim.step(3)
        sim.set_state()
        for factors in ((1.0, 1.05, 1.25, 1.5, 2.0), (1.1,)):
            sim.autotune(trial_steps=10, cell_factors=factors, graph_blocks=(5, 20))
        sim.set_neighbor_lists(0.1, 64)
        sim.step(40)
        sim.set_neighbor_lists(0.0, 0)
        sim.step(40)
        got, grid = sim.get_state(), sim.grid(0)
    assert same(got, O.run(sc.copy(interval=grid.interval), 80, prec), prec)
