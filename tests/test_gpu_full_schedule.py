"""The folded solve's phases (distance solve, tets, solid contacts) and the
warp-wide contact collection where they can go wrong, parity build against
the oracle bit for bit: one iteration (two or three phases), one-lattice and
tiny bodies, a body cut in half (contacts between former neighbours), and
bodies squeezed until a solid has more than the cache's 40 candidates and its
buckets hold dozens of solids."""
import numpy as np
import pytest

from fluidphysics_b200 import _lib as L
from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene
from helpers import assert_states_equal, load_state
from oracle.oracle import o2_from_scene

pytestmark = pytest.mark.gpu
BOTH = L.FEAT_TETS | L.FEAT_SOLID_CONTACTS


@pytest.mark.parametrize("features,iters,dim,dim2,squeeze,cut", [
    (BOTH, 1, 7, 3, 1.0, False), (L.FEAT_TETS, 1, 6, 0, 1.0, False), (L.FEAT_SOLID_CONTACTS, 1, 6, 0, 1.0, True),
    (BOTH, 2, 1, 0, 1.0, False), (BOTH, 2, 2, 1, 1.0, False), (BOTH, 0, 5, 2, 1.0, False),
    (BOTH, 3, 9, 4, 0.55, True), (L.FEAT_SOLID_CONTACTS, 2, 12, 0, 0.35, True), (BOTH, 4, 11, 5, 0.8, True)])
def test_solid_phases_bit_exact(features, iters, dim, dim2, squeeze, cut):
    d, p, opts = S.gpu_scene(dim, 700, 30, iters=iters, features=features)
    d.solid_dim2 = dim2
    d.cube2_center[:] = [0.1, opts["cubeCenter"][1] + 0.05, 0.07]  # overlapping the body
    fp = S.jittered_block(10, 7, 10, 0.066, 0.1, 4)
    sc = S.Scene("phases", d, p, fp, np.zeros_like(fp), opts["fluidMass"], 1 / 60, 5, 1)
    sim, o2 = sim_from_scene(sc, "parity"), o2_from_scene(sc)
    st = sim.read_state()
    n = sc.solid_n
    c = st["pos"][:n, :3].mean(0)
    rng = np.random.default_rng(dim)
    st["pos"][:n, :3] = c + (st["pos"][:n, :3] - c) * squeeze + rng.uniform(-0.002, 0.002, (n, 3))
    st["prev"][:n, :3] = st["pos"][:n, :3]
    cons = sim.read_constraints()
    if cut:
        side = st["pos"][:n, 0] > c[0] + 0.001
        cons[side[cons[:, 0]] != side[cons[:, 1]], 3] = 0
    load_state(sim, st, cons)
    o2.write_state(**st)
    o2.write_constraints(cons)
    for k in range(2):
        sim.step(1 / 60, 3)
        o2.step(1 / 60, 3)
        assert_states_equal(sim.read_state(), o2.read_state(), f"frame {k}")
    assert np.array_equal(sim.read_constraints(), o2.read_constraints()[0])
    assert np.array_equal(sim.read_tets(), o2.read_tets())
    if features & L.FEAT_SOLID_CONTACTS and squeeze < 0.6:
        assert o2.read_contact_cache()[0].max() == 40  # the cache was full somewhere
    sim.close()


@pytest.mark.parametrize("dim,dim2", [(1, 0), (2, 0), (5, 2), (9, 4)])
def test_solid_viscosity_bit_exact_and_batched(dim, dim2):
    """Solid viscosity on its lanes: single scene against the oracle (cut body,
    stirred velocities), and the same scene in a batch beside one without it."""
    from fluidphysics_b200 import batch as B
    d, p, opts = S.gpu_scene(dim, 300, 30, iters=2)
    d.solid_dim2 = dim2
    d.cube2_center[:] = [0.9, 1.0, 0.7]
    S.set_params(p, {"solidViscosity": 0.3})
    fp = S.jittered_block(8, 5, 8, 0.066, 0.1, 4)[:300]
    sc = S.Scene("visc", d, p, fp, np.zeros_like(fp), opts["fluidMass"], 1 / 60, 5, 1)
    sim, o2 = sim_from_scene(sc, "parity"), o2_from_scene(sc)
    st, cons = sim.read_state(), sim.read_constraints()
    n = sc.solid_n
    rng = np.random.default_rng(dim)
    st["vel"][:n, :3] = rng.normal(0, 1, (n, 3))
    side = st["pos"][:n, 0] > st["pos"][:n, 0].mean() + 0.001
    cons[side[cons[:, 0]] != side[cons[:, 1]], 3] = 0
    load_state(sim, st, cons)
    o2.write_state(**st)
    o2.write_constraints(cons)
    sim.step(1 / 60, 3)
    o2.step(1 / 60, 3)
    g = sim.read_state()
    assert_states_equal(g, o2.read_state(), "visc")
    with B.Batch(solid_iters=2, max_scenes=2, variant="parity") as b:
        sid = b.add_scene(sc)
        b.add_scene(B.batch_scene(4, 500, 3, iters=2))
        b.write_state(sid, **st)
        b.write_constraints(sid, cons)
        b.step(1 / 60, 3)
        b.sync()
        h = b.read_state(sid)
    for k in ("pos", "vel", "flags"):
        assert np.array_equal(g[k], h[k]), k
    sim.close()
