"""The stateless grid build reads the caller's flags once, in its count. Here the
flags lie in the buffer that the same call fills with the bucket counts, so they
change between its passes: the grid is that of the flags as they were, and the
scratch, which outlives the call, is clear for the next ones."""
import ctypes as C

import numpy as np
import pytest

from fluidphysics_b200 import _lib as L

pytestmark = pytest.mark.gpu
CELL = 0.078


def expected(pos, act, table):
    c = np.floor(pos[:, :3].astype(np.float64) * (1.0 / CELL)).astype(np.int64)
    h = ((c[:, 0] * 92837111) ^ (c[:, 1] * 689287499) ^ (c[:, 2] * 283923481)) & (table - 1)
    idx = np.flatnonzero(act)
    counts = np.bincount(h[idx], minlength=table)
    return counts, np.concatenate([[0], np.cumsum(counts)]), idx[np.lexsort((-idx, h[idx]))]


@pytest.mark.parametrize("n,table", [(777, 1), (5000, 4096), (100003, 1 << 15)])
@pytest.mark.parametrize("entry", ["upbd_grid_build", "upbd_grid_build_noalloc"])
def test_flags_that_change_during_a_build(n, table, entry):
    import torch
    fn = getattr(L.load(), entry)
    rng = np.random.default_rng(n)
    pos = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    act = rng.random(n) < 0.9
    dp = torch.from_numpy(pos).cuda()
    p = lambda t: C.c_void_p(t.data_ptr())
    for shared in (True, False, True, False):
        df = torch.from_numpy(act.astype(np.int32)).cuda()
        cnt = df if shared else torch.zeros(table, dtype=torch.int32, device="cuda")
        off = torch.full((table + 1,), -1, dtype=torch.int32, device="cuda")
        ent = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        assert fn(p(dp), p(df), n, table, CELL, p(cnt), p(off), p(ent), None) == 0
        torch.cuda.synchronize()
        counts, offsets, entries = expected(pos, act, table)
        assert np.array_equal(off.cpu().numpy(), offsets)
        assert np.array_equal(ent.cpu().numpy()[:len(entries)], entries)
        assert np.array_equal(cnt.cpu().numpy()[:table], counts)
