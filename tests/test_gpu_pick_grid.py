"""Pick and the stateless grid build at the edges of their launches: bodies from
one particle to several per thread of the pick's grid, ties (the lowest index
wins), rays that hit nothing; grids of one bucket, of a ragged last tile, with
and without counts and into buffers that are not 16-byte aligned. Ids, t and
grids are compared with the oracle's / numpy's exactly."""
import ctypes as C

import numpy as np
import pytest

from fluidphysics_b200 import _lib as L
from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import sim_from_scene
from helpers import load_state
from oracle.oracle import o2_from_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1, 2, 7, 20, 45])
def test_pick_matches_oracle(dim):
    d, p, opts = S.gpu_scene(dim, 16, 30)
    sc = S.Scene("pick", d, p, np.zeros((0, 3), np.float32), np.zeros((0, 3), np.float32), opts["fluidMass"], 1 / 60, 5, 1)
    sim, o2 = sim_from_scene(sc), o2_from_scene(sc)
    st = sim.read_state()
    rng = np.random.default_rng(dim)
    n = sc.solid_n
    st["pos"][:n, :3] += rng.normal(0, 0.01, (n, 3))
    if n > 4:  # three particles in one place, one of them inactive
        st["pos"][[n - 1, n // 2, 1], :3] = st["pos"][n // 3, :3]
        st["flags"][1] = 0
    load_state(sim, st)
    o2.write_state(**st)
    hits = 0
    for k in range(20):
        q = st["pos"][n // 3 if k % 4 == 0 else int(rng.integers(n)), :3].astype(np.float64)
        ro = np.array([rng.uniform(-3, 3), 2.5, 4.0])
        rd = q - ro if k % 5 else ro - q  # every fifth ray points away
        rd /= np.linalg.norm(rd)
        a, b = sim.pick(ro, rd, 0.05), o2.pick(ro, rd, 0.05)
        assert a == b or (a[0] == b[0] == -1), (dim, k, a, b)
        hits += a[0] >= 0
    assert hits >= 12
    sim.close()


@pytest.mark.parametrize("n,table,shift", [(0, 16, 0), (1, 1, 0), (777, 1, 0), (5000, 2, 1), (4097, 2048, 0),
                                           (6001, 4096, 3), (100003, 1 << 18, 0), (20000, 1 << 12, 2)])
def test_stateless_grid_matches_numpy(n, table, shift):
    import torch
    lib = L.load()
    rng = np.random.default_rng(n + table)
    cell = 0.078
    pos = rng.uniform(-3, 3, (n, 4)).astype(np.float32)
    act = rng.random(n) < 0.9
    c = np.floor(pos[:, :3].astype(np.float64) * (1.0 / cell)).astype(np.int64)
    h = ((c[:, 0] * 92837111) ^ (c[:, 1] * 689287499) ^ (c[:, 2] * 283923481)) & (table - 1)
    idx = np.flatnonzero(act)
    order = idx[np.lexsort((-idx, h[idx]))]  # by bucket, descending index inside
    counts = np.bincount(h[idx], minlength=table)
    dp = torch.from_numpy(pos).cuda() if n else torch.zeros(1, 4, device="cuda")
    df = torch.from_numpy(act.astype(np.int32)).cuda() if n else torch.zeros(1, dtype=torch.int32, device="cuda")
    for fn in (lib.upbd_grid_build, lib.upbd_grid_build_noalloc):
        for with_counts in (True, False):
            off = torch.full((table + 1 + shift,), -1, dtype=torch.int32, device="cuda")
            ent = torch.full((n + shift + 1,), -1, dtype=torch.int32, device="cuda")
            cnt = torch.full((table + shift,), -1, dtype=torch.int32, device="cuda")
            p = lambda t: C.c_void_p(t.data_ptr() + 4 * shift)
            rc = fn(C.c_void_p(dp.data_ptr()), C.c_void_p(df.data_ptr()), n, table, cell, p(cnt) if with_counts else None,
                    p(off), p(ent), None)
            assert rc == 0
            torch.cuda.synchronize()
            assert np.array_equal(off.cpu().numpy()[shift:], np.concatenate([[0], np.cumsum(counts)]))
            assert np.array_equal(ent.cpu().numpy()[shift:shift + len(order)], order)
            if with_counts:
                assert np.array_equal(cnt.cpu().numpy()[shift:], counts)
