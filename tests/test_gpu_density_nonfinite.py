"""Fluid that is not at a finite distance (NaN, infinite, or so far out that the
squared distance overflows) in the product build's density: it is in nobody's
density or list, and leaves the near density of every particle that meets it in
its 27 buckets NaN, whatever form of the pass the window takes (crowded cells,
drops, tables of one bucket)."""
import numpy as np
import pytest

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene
from helpers import load_state

pytestmark = pytest.mark.gpu
DENSITY = 3
K = (92837111.0, 689287499.0, 283923481.0)


def toint32(x):
    """JavaScript's ToInt32 of an array of doubles, as unsigned 32 bits"""
    return np.array([int(v) % (1 << 32) if np.isfinite(v) else 0 for v in x.ravel()], np.int64).reshape(x.shape)


def buckets(pos, inv, table):
    """own bucket, and the 27 around, of each position"""
    c = np.floor(pos.astype(np.float64) * inv)
    part = [[toint32((c[:, a] + o) * K[a]) for o in (-1.0, 0.0, 1.0)] for a in range(3)]
    around = [(x ^ y ^ z) & (table - 1) for x in part[0] for y in part[1] for z in part[2]]
    return around[13], np.stack(around, 1)


@pytest.mark.parametrize("n,table,spread", [(40, 1, 1.0), (300, 1 << 10, 1.0), (900, 1 << 12, 3.0), (2100, 1 << 6, 0.6)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 3e19, -1e30])
def test_near_density_of_what_is_not_at_a_finite_distance(n, table, spread, bad):
    d, p, opts = S.gpu_scene(3, n, 30)
    d.table_size = table
    rng = np.random.default_rng(n + table)
    side = spread * p.fluid_h * (n / 6.0) ** (1 / 3)
    fluid = (rng.uniform(0, side, (n, 3)) + [0, 0.3, 0]).astype(np.float32)
    sc = S.Scene("far", d, p, fluid, np.zeros((n, 3), np.float32), opts["fluidMass"], 1 / 60, 5, 1)
    st0 = None
    dens = []
    for with_bad in (False, True):
        sim = sim_from_scene(sc)
        st = sim.read_state()
        if st0 is None:
            st0 = {k: a.copy() for k, a in st.items()}
        st = {k: a.copy() for k, a in st0.items()}
        out = sc.solid_n + np.array([1, n // 2])  # one coordinate of each
        if with_bad:
            st["pos"][out, [0, 2]] = bad
        else:
            st["flags"][out] = 0
        load_state(sim, st)
        sim.substep_partial(1 / 300, DENSITY)
        dens.append(sim.read_state())
        sim.close()
    g = dens[1]
    act = np.flatnonzero(g["flags"][sc.solid_n:] & 1) + sc.solid_n
    pos = g["pos"][act, :3]
    own, around = buckets(pos, 1.0 / p.cell_size, table)
    far = np.zeros(len(act), bool)
    with np.errstate(over="ignore", invalid="ignore"):
        for k in range(len(act)):
            met = np.isin(own, around[k])
            e = pos[met] - pos[k]
            far[k] = not np.isfinite((e * e).sum(1, dtype=np.float32)).all()
    rho, near = g["density"][act, 0], g["density"][act, 1]
    assert far.any()
    assert np.array_equal(np.isnan(near), far)
    assert np.isfinite(rho).all()
    # the others' densities are those without the two, but for the order of the
    # sums: fewer than n terms (each up to 27 times), one rounding each
    ok = np.isin(act, np.flatnonzero(dens[0]["flags"] & 1))
    ref = dens[0]["density"][act[ok]]
    tol = 2.0 * min(27 * n, 3000) * 2.0**-24
    assert np.allclose(rho[ok], ref[:, 0], rtol=tol, atol=0)
    assert np.allclose(near[ok & ~far], ref[~far[ok], 1], rtol=tol, atol=0)
