"""upbd_read_grid where its two forms meet: tables up to, at and past the list
memory its offsets are gathered in, against numpy."""
import numpy as np
import pytest

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene
from test_gpu_density_nonfinite import buckets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n,table", [(1, 1, 1), (1, 1, 128), (1, 1, 256), (1, 1, 1 << 12), (2, 300, 1 << 15), (2, 300, 1 << 16)])
def test_offsets_counts_and_entries(dim, n, table):
    d, p, opts = S.gpu_scene(dim, n, 30)
    d.table_size = table
    rng = np.random.default_rng(table)
    fluid = rng.uniform(0, 0.6, (n, 3)).astype(np.float32)
    sim = sim_from_scene(S.Scene("grid", d, p, fluid, np.zeros((n, 3), np.float32), opts["fluidMass"], 1 / 60, 5, 1))
    for _ in range(2):
        sim.rebuild_grid()
        counts, offsets, entries = sim.read_grid()
        st = sim.read_state()
        own, _ = buckets(st["pos"][:, :3], 1.0 / p.cell_size, table)
        want = np.bincount(own, minlength=table)
        assert np.array_equal(counts, want)
        assert np.array_equal(offsets, np.concatenate([[0], np.cumsum(want)]))
        assert np.array_equal(entries[:len(own)], np.lexsort((-np.arange(len(own)), own)))
        sim.step(1 / 60, 2)
    sim.close()
