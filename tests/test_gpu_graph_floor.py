"""The launch floor measures the graph that frames run: it is captured where
upbd_step captures, so a handle on a stream that cannot be captured (the legacy
default stream) steps and is measured alike, with the same kernels."""
import pytest

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene

pytestmark = pytest.mark.gpu
LEGACY = 1  # cudaStreamLegacy


def test_floor_on_the_legacy_stream():
    sc = S.cpu_scene()
    own, legacy = sim_from_scene(sc), sim_from_scene(sc)
    legacy.set_stream(LEGACY)
    for sim in (own, legacy):
        n = sim.launches
        sim.step(sc.dt, sc.substeps)
        sim.sync()
        ms, nodes = sim.graph_floor(sc.dt, sc.substeps, 20)
        assert nodes == sim.launches - n and ms > 0
        sim.close()
