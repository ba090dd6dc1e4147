"""A pick behind queued frames: the result is of the state those frames leave,
also where they take far longer than the host watches for it."""
import numpy as np
import pytest

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames", [1, 60])
def test_pick_waits_for_the_frames_before_it(frames):
    sc = S.gpu_default()
    sim = sim_from_scene(sc)
    ro = np.array([0.3, 0.2, 6.0])
    c = np.array(list(sc.desc.cube_center))
    rd = (c - ro) / np.linalg.norm(c - ro)
    for _ in range(2):  # graphs are captured
        sim.step(sc.dt, sc.substeps)
    sim.sync()
    before = sim.pick(ro, rd, 0.3)
    for _ in range(frames):
        sim.step(sc.dt, sc.substeps)
    got = sim.pick(ro, rd, 0.3)
    sim.sync()
    assert got == sim.pick(ro, rd, 0.3)
    assert got[0] >= 0 and got != before  # the body falls
    sim.close()
