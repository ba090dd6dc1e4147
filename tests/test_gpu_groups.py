"""upbd_groups against the oracle's sequential union-find (the labels are
whole numbers: equal) where its parallel form can go wrong: bodies smaller
than a warp, two lattices, planar cuts (few seeds, many constraints between
their trees), heavy random damage (many seeds, joins of joins), all or no
constraints alive."""
import numpy as np
import pytest

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene
from oracle.oracle import o2_from_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,dim2", [(1, 0), (2, 0), (3, 2), (5, 3), (11, 4), (20, 8)])
def test_groups_cuts_and_damage(dim, dim2):
    d, p, opts = S.gpu_scene(dim, 1024, 30)
    d.solid_dim2 = dim2
    sc = S.Scene("groups", d, p, np.zeros((0, 3), np.float32), np.zeros((0, 3), np.float32), opts["fluidMass"],
                 1 / 60, 5, 1)
    sim, o2 = sim_from_scene(sc), o2_from_scene(sc)
    cons = sim.read_constraints()
    pos = sim.read_state()["pos"][:sc.solid_n, :3].astype(np.float64)
    rng = np.random.default_rng(dim)
    for trial in range(12):
        side = np.zeros(sc.solid_n, np.int64)
        for k in range(trial % 5):
            side += ((pos - pos.mean(0) + rng.normal(0, 0.05, 3)) @ rng.normal(size=3) > 0).astype(np.int64) << k
        c = cons.copy()
        c[:, 3] = side[c[:, 0]] == side[c[:, 1]]
        c[:, 3] &= rng.random(len(c)) >= (0.0, 0.6, 0.9)[trial % 3]
        if trial == 11:
            c[:, 3] = 0
        sim.write_constraints(c)
        o2.write_constraints(c)
        g, ref = sim.groups(), o2.groups()
        assert np.array_equal(g, ref), (dim, dim2, trial, int((g != ref).sum()))
    sim.close()
