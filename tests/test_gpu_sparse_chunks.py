"""Density and xsph over windows of small chunks (two to a warp), parity build
against the oracle bit for bit: cells of one and two particles, with a share of
fuller ones on either side of the rule (fewer than a quarter of a window's chunks
over four particles), an odd number of chunks, a crowded cell whose sparse
neighbours stage more than a half's rows, cells with equal keys, every window
size; at rest (lists are read) and moving (buckets are walked again)."""
import numpy as np
import pytest

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene
from helpers import load_state
from oracle.oracle import o2_from_scene

pytestmark = pytest.mark.gpu
DENSITY, XSPH_APPLY = 3, 15


def drops(n, full, crowd, H, rng):
    side = 28 if n < 28**3 else 36
    cells = rng.permutation(side**3)[:n]
    per = np.where(rng.random(n) < full, rng.integers(3, 10, n), rng.integers(1, 3, n))
    of = np.repeat(cells, per)[: n - crowd]
    c = np.stack([of % side, of // side % side, of // side**2], 1).astype(np.float64)
    p = (c + rng.uniform(0.05, 0.95, c.shape)) * H + [0, 0.3, 0]
    spot = np.array([5.5, 5.5, 5.5]) * H + [0, 0.3, 0] + rng.uniform(0, 0.4 * H, (crowd, 3))
    return np.concatenate([p, spot]).astype(np.float32)


@pytest.mark.parametrize("n,table,full,crowd,speed", [
    (9, 1 << 10, 0.0, 0, 0.0), (203, 1 << 12, 0.0, 0, 4.0), (901, 64, 0.1, 0, 4.0), (4001, 1 << 14, 0.1, 170, 0.0),
    (4001, 1 << 14, 0.25, 170, 6.0), (9003, 1 << 15, 0.0, 300, 6.0), (21001, 1 << 16, 0.1, 0, 4.0),
    (40001, 1 << 17, 0.05, 400, 6.0)])
def test_small_chunks_bit_exact(n, table, full, crowd, speed):
    d, p, opts = S.gpu_scene(3, n, 30)
    d.table_size = table
    rng = np.random.default_rng(n + table)
    vel = (speed * rng.standard_normal((n, 3))).astype(np.float32)
    sc = S.Scene("drops", d, p, drops(n, full, crowd, p.fluid_h, rng), vel, opts["fluidMass"], 1 / 60, 5, 1)
    sim, o2 = sim_from_scene(sc, "parity"), o2_from_scene(sc)
    st = sim.read_state()
    for last in (DENSITY, XSPH_APPLY):
        load_state(sim, st)
        o2.write_state(**st)
        sim.substep_partial(1 / 300, last)
        o2.substep_partial(1 / 300, last)
        g, r = sim.read_state(), o2.read_state()
        for k in ("density", "pos", "vel"):
            a, b = g[k], r[k].astype(np.float32)
            bad = np.flatnonzero(~((a == b) | (np.isnan(a) & np.isnan(b))).all(axis=1))
            assert bad.size == 0, (last, k, bad[:8], a[bad[:2]], b[bad[:2]])
    sim.close()
