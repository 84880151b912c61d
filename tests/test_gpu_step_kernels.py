"""The step kernels where calls reach them: calls of fewer than 8 steps, and
longer ones on scenes too fast for lists (graph blocks, and the same launches
one by one on large scenes).  Calm scenes take runs in calls of 8 steps and
more, so the contact kernel's walks are tested in calls of 7 here."""
import os
import subprocess
import sys

import numpy as np
import pytest

import psb200
from psb200 import scenes
from oracle import ps_oracle as O
from conftest import ROOT

pytestmark = pytest.mark.gpu

WALKS_BY_SEVEN = r"""
import sys
import numpy as np
import psb200
from psb200 import scenes
from oracle import ps_oracle as O

if sys.argv[1] == "bounds":
    psb200.LIB_PATH = psb200.DEBUG_LIB_PATH
    assert psb200.bounds_checked()
batch = [scenes.pile(1500, seed=41, k_spring=1.0), scenes.lattice_c1(side=10), scenes.box_mesh_scene(),
         scenes.funnel_wall_scene(700, seed=9)]
sims = [batch, batch[:2], batch[:1], batch[2:3]]  # with and without a mesh, many scenes and one
for prec in ("f32", "f64"):
    want = [O.run(sc, 42, prec) for sc in batch]
    for scs in sims:
        for walk, block in psb200.CONTACT_KERNELS:
            with psb200.Simulation(scs, prec) as sim:
                sim.set_contact_kernel(walk, block)
                sim.set_state()
                for _ in range(6):
                    sim.step(7)
                    assert sim.launches() == 1 + 4 * 7
                sim.sync()
                got = sim.get_state()
            off = 0
            for sc in scs:
                w = want[[x is sc for x in batch].index(True)]
                assert np.array_equal(got[off:off + sc.n].astype(w.dtype), w), (prec, len(scs), walk, block, sc.name)
                off += sc.n
print("DONE", flush=True)
"""


@pytest.mark.parametrize("build", ["product", "bounds"])
def test_every_walk_in_calls_of_seven_steps(need_gpu, build):
    env = dict(os.environ)
    env["PYTHONPATH"] = os.pathsep.join([ROOT, os.path.join(ROOT, "particle-stabilizer_b200", "python"),
                                         env.get("PYTHONPATH", "")])
    r = subprocess.run([sys.executable, "-c", WALKS_BY_SEVEN, build], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=900)
    assert r.returncode == 0 and r.stdout.rstrip().endswith("DONE"), r.stdout[-3000:] + r.stderr[-3000:]


def fast_pile() -> scenes.Scene:
    sc = scenes.pile(1000, seed=21, k_spring=1.0)
    st = sc.state.copy()
    st[:, 3:6] *= 500.0
    return sc.copy(state=st)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("calls", [(706,), (1, 33, 200, 16, 200, 256), (206, 200, 300)])
def test_graph_blocks_of_a_fast_scene(need_gpu, calls, prec):
    # blocks of 200 steps, their remainders, and lengths that come again
    with psb200.Simulation(fast_pile(), prec) as sim:
        sim.set_state()
        for n in calls:
            sim.step(n)
            assert sim.launches() > 3 * n or n < 8
        got = sim.get_state()
    with psb200.Simulation(fast_pile(), prec) as sim:
        sim.set_state()
        sim.profile_steps(706)
        want = sim.get_state()
    assert np.array_equal(got, want, equal_nan=True)


def test_blocks_of_a_large_scene_launched_one_by_one_and_captured(need_gpu):
    # the first time a length comes its kernels are launched one by one, the
    # second time they are captured
    sc = scenes.c2_scene(n=300007)
    with psb200.Simulation(sc, "f32") as sim:
        sim.set_state()
        for n in (6, 6, 6, 50, 44, 44, 44):
            sim.step(n)
        got = sim.get_state()
    with psb200.Simulation(sc, "f32") as sim:
        sim.set_state()
        sim.profile_steps(200)
        want = sim.get_state()
    assert np.array_equal(got, want, equal_nan=True)
