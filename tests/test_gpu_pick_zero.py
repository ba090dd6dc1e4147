"""Pick at t = 0: a particle at the ray's origin, whose t is -0 when every
component of the direction is negative, is the nearest one, and ties with the
others there by index."""
import numpy as np
import pytest

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene
from helpers import load_state
from oracle.oracle import o2_from_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [[5], [5, 2], [0, 7]])
@pytest.mark.parametrize("sign", [(-1, -1, -1), (1, 1, 1), (-1, 1, -1), (0, -1, 0)])
def test_particle_at_the_origin_of_the_ray(at, sign):
    d, p, opts = S.gpu_scene(2, 16, 30)
    sc = S.Scene("pick", d, p, np.zeros((0, 3), np.float32), np.zeros((0, 3), np.float32), opts["fluidMass"], 1 / 60, 5, 1)
    sim, o2 = sim_from_scene(sc), o2_from_scene(sc)
    st = sim.read_state()
    ro = np.array([0.25, 1.5, -0.75])
    rd = np.array([0.5, 0.75, 0.625]) * sign
    rd /= np.linalg.norm(rd)
    far = [k for k in range(sc.solid_n) if k not in at]
    st["pos"][at, :3] = ro
    st["pos"][far, :3] = ro + np.outer(0.1 + 0.1 * np.arange(len(far)), rd)  # further along the ray
    load_state(sim, st)
    o2.write_state(**st)
    got = sim.pick(ro, rd, 0.05)
    assert got == o2.pick(ro, rd, 0.05)
    assert got == (min(at), 0.0)
    sim.close()
