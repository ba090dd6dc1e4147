"""The shipped float build over the chunk cases of test_gpu_density_chunks.py and
test_gpu_sparse_chunks.py, whose parity build picks its candidates by other code:
densities against 64 bits at the pass's own positions, and a substep against the
oracle.

Tolerances. A term's q = 1 - d / H: the differences of two float positions are
exact to 2^-24, d2 to 3 * 2^-24, the approximate square root to 2^-22, times
1 / H and the subtraction 2^-24 each: 1e-6 covers them for d <= H. A density is a
sum of q^2 (2 q dq each) and q^3 (3 q^2 dq), and each of its n additions and
products rounds once or twice (2^-23 of the sum each). The substep has the
tolerances of the per-substep tests; xsph counts its neighbours unweighted, so a
particle with a neighbour within 1e-5 m of H may count another number of them and
is left out."""
import numpy as np
import pytest
from scipy.spatial import cKDTree

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene
from helpers import POS_RTOL, POS_SCALE, VEL_RTOL, VEL_SCALE, load_state
from oracle.oracle import o2_from_scene
from test_gpu_density_chunks import cloud
from test_gpu_density_nonfinite import buckets
from test_gpu_sparse_chunks import drops

pytestmark = pytest.mark.gpu
DENSITY, APPLY_FLUID, XSPH_APPLY = 3, 5, 15


def scene(n, table, fluid, vel):
    d, p, opts = S.gpu_scene(3, n, 30)
    d.table_size = table
    return S.Scene("chunks", d, p, fluid, vel, opts["fluidMass"], 1 / 60, 5, 1)


def check_density(g, sc, table):
    """rho and near density of the active fluid against 64 bits"""
    H = float(np.float32(sc.params.fluid_h))
    act = np.flatnonzero(g["flags"][sc.solid_n:] & 1) + sc.solid_n
    pos = g["pos"][act, :3].astype(np.float64)
    own, around = buckets(g["pos"][act, :3], 1.0 / sc.params.cell_size, table)
    order = np.argsort(own, kind="stable")
    start = np.searchsorted(own[order], np.arange(table + 1))
    for i in range(len(act)):
        j = np.concatenate([order[start[b]:start[b + 1]] for b in around[i]])
        q = 1.0 - np.sqrt(((pos[j[j != i]] - pos[i]) ** 2).sum(1)) / H
        q = q[q > 0]
        rho, near = g["density"][act[i]]
        assert abs(rho - (q * q).sum()) <= 2e-6 * q.sum() + len(q) * 2.0**-23 * (q * q).sum() + 1e-12, (i, rho, (q * q).sum())
        assert abs(near - (q**3).sum()) <= 3e-6 * (q * q).sum() + len(q) * 2.0**-22 * (q**3).sum() + 1e-12, (i, near)


def check_state(g, r, what, keep=None):
    assert np.array_equal(g["flags"], r["flags"]), what
    act = (g["flags"] & 1).astype(bool)
    assert np.abs(g["pos"][act, :3] - r["pos"][act, :3]).max() <= POS_RTOL * POS_SCALE, what
    if keep is not None:
        assert np.abs(g["vel"][keep, :3] - r["vel"][keep, :3]).max() <= VEL_RTOL * VEL_SCALE, what


@pytest.mark.parametrize("n,table,kind", [
    (1, 1 << 10, "plain"), (5, 1 << 10, "plain"), (130, 1 << 12, "plain"), (700, 1, "plain"), (900, 8, "plain"),
    (2100, 64, "crowded"), (2100, 1 << 13, "crowded"), (6007, 1 << 14, "plain")])
def test_density_and_lists(n, table, kind):
    d, p, _ = S.gpu_scene(3, n, 30)
    rng = np.random.default_rng(n + table)
    sc = scene(n, table, cloud(n, kind, p.fluid_h, rng), np.zeros((n, 3), np.float32))
    sim, o2 = sim_from_scene(sc), o2_from_scene(sc)
    st = sim.read_state()
    dead = rng.random(n) < 0.1
    dead[0] = False
    st["flags"][sc.solid_n:][dead] = 0
    for last in (DENSITY, APPLY_FLUID):
        load_state(sim, st)
        o2.write_state(**st)
        sim.substep_partial(1 / 300, last)
        o2.substep_partial(1 / 300, last)
        g = sim.read_state()
        if last == DENSITY:
            check_density(g, sc, table)
        check_state(g, o2.read_state(), last)
    sim.close()


@pytest.mark.parametrize("n,table,full,crowd,speed", [
    (9, 1 << 10, 0.0, 0, 0.0), (203, 1 << 12, 0.0, 0, 4.0), (901, 64, 0.1, 0, 4.0), (4001, 1 << 14, 0.1, 170, 0.0),
    (4001, 1 << 14, 0.25, 170, 6.0), (9003, 1 << 15, 0.0, 300, 6.0)])
def test_small_chunks(n, table, full, crowd, speed):
    d, p, _ = S.gpu_scene(3, n, 30)
    rng = np.random.default_rng(n + table)
    vel = (speed * rng.standard_normal((n, 3))).astype(np.float32)
    sc = scene(n, table, drops(n, full, crowd, p.fluid_h, rng), vel)
    sim, o2 = sim_from_scene(sc), o2_from_scene(sc)
    st = sim.read_state()
    for last in (DENSITY, XSPH_APPLY):
        load_state(sim, st)
        o2.write_state(**st)
        sim.substep_partial(1 / 300, last)
        o2.substep_partial(1 / 300, last)
        g, r = sim.read_state(), o2.read_state()
        if last == DENSITY:
            check_density(g, sc, table)
        act = np.flatnonzero(g["flags"] & 1)
        fl = act[act >= sc.solid_n]
        t = cKDTree(r["pos"][fl, :3].astype(np.float64))
        q = r["pos"][fl, :3].astype(np.float64)
        edge = t.query_ball_point(q, p.fluid_h + 1e-5, return_length=True) != t.query_ball_point(q, p.fluid_h - 1e-5, return_length=True)
        check_state(g, r, last, np.concatenate([act[act < sc.solid_n], fl[~edge]]))
        assert edge.mean() < 0.02
    sim.close()
