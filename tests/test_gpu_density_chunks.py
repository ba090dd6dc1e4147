"""The density pass's chunks where they can go wrong, parity build against the
oracle bit for bit (densities, and the neighbour lists through the displacement
that reads them): scenes of one particle, below and above a window, with several
blocks of every window size; crowded cells (chunks of every size, more
candidates than one round stages, lists that overflow); small hash tables, where
a bucket holds many cells and some of a particle's 27 buckets coincide; cells far
out whose hashes and keys are equal although the cells are not."""
import numpy as np
import pytest

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene
from helpers import load_state
from oracle.oracle import o2_from_scene

pytestmark = pytest.mark.gpu
DENSITY, APPLY_FLUID = 3, 5


def cloud(n, kind, H, rng):
    side = H * max(1.0, (n / 6.0) ** (1 / 3))
    p = rng.uniform(0, side, (n, 3)) + [0, 0.3, 0]
    if kind == "crowded":  # a third of them in one spot of half a cell
        p[: n // 3] = [0.31, 0.62, 0.17] + rng.uniform(0, 0.5 * H, (n // 3, 3))
    if kind == "far":
        p[: n // 2, 0] = np.float32(2.0) ** (100 + np.arange(n // 2) % 5)
        p[: n // 2, 1:] = 0.5 + rng.uniform(0, 0.2 * H, (n // 2, 2))
    return p.astype(np.float32)


@pytest.mark.parametrize("n,table,kind", [
    (1, 1 << 10, "plain"), (5, 1 << 10, "plain"), (130, 1 << 12, "plain"), (700, 1, "plain"), (900, 8, "plain"),
    (2100, 64, "crowded"), (2100, 1 << 13, "crowded"), (64, 1 << 10, "far"), (6007, 1 << 14, "plain"),
    (11003, 1 << 12, "plain"), (23001, 1 << 16, "crowded"), (45001, 1 << 18, "plain")])
def test_density_and_lists_bit_exact(n, table, kind):
    d, p, opts = S.gpu_scene(3, n, 30)
    d.table_size = table
    rng = np.random.default_rng(n + table)
    sc = S.Scene("chunks", d, p, cloud(n, kind, p.fluid_h, rng), np.zeros((n, 3), np.float32), opts["fluidMass"],
                 1 / 60, 5, 1)
    sim, o2 = sim_from_scene(sc, "parity"), o2_from_scene(sc)
    st = sim.read_state()
    dead = rng.random(n) < 0.1  # inactive slots have no place in the grid
    dead[0] = False
    st["flags"][sc.solid_n:][dead] = 0
    for last in (DENSITY, APPLY_FLUID):
        load_state(sim, st)
        o2.write_state(**st)
        sim.substep_partial(1 / 300, last)
        o2.substep_partial(1 / 300, last)
        g, r = sim.read_state(), o2.read_state()
        for k in ("density", "pos"):
            a, b = g[k], r[k].astype(np.float32)
            bad = np.flatnonzero(~((a == b) | (np.isnan(a) & np.isnan(b))).all(axis=1))
            assert bad.size == 0, (last, k, bad[:8], a[bad[:2]], b[bad[:2]])
    sim.close()
