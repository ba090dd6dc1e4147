"""A batch whose scenes are replaced by others of the same particle count and
another mix: the frame's launch grids follow every pass's own size, not only the
count (a graph captured over nearly all fluid has a handful of CTAs for the
solids), and a graph whose grids cover the scenes is used again."""
import pytest

from fluidphysics_b200 import batch as B
from helpers import assert_states_equal

pytestmark = pytest.mark.gpu
DT, NSUB = 1 / 60, 5


def fluid_heavy():
    return B.batch_scene(4, 9000, 1)  # 64 + 9,000


def body_heavy():
    return B.batch_scene(20, 1064, 2)  # 8,000 + 1,064


def frame(b):
    b.step(DT, NSUB)
    b.sync()


@pytest.mark.parametrize("block,per_sm", [(128, 128), (256, 8), (64, 256)])
def test_grids_follow_the_mix(block, per_sm):
    with B.Batch(max_scenes=4, block_threads=block, ctas_per_sm=per_sm) as b, \
         B.Batch(max_scenes=4, block_threads=block, ctas_per_sm=per_sm) as fresh:
        a = b.add_scene(fluid_heavy())
        frame(b)
        frame(b)
        assert b.info().captures == 1
        b.remove_scene(a)
        a = b.add_scene(body_heavy())
        frame(b)
        assert b.info().captures == 2  # the solids' passes have outgrown the first one's grids
        frame(b)
        assert b.info().captures == 2
        f = fresh.add_scene(body_heavy())
        frame(fresh)
        frame(fresh)
        assert_states_equal(b.read_state(a), fresh.read_state(f), "after the change")
        b.remove_scene(a)
        a = b.add_scene(fluid_heavy())
        frame(b)
        assert b.info().captures == 2  # both mixes are covered now
