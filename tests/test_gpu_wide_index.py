"""A scene with so many slots (45 million, 29 GB) that a neighbour list's row
times the slot count passes 2^32: the same 2,500 crowded particles in its last
slots take the same substep, bit for bit, as in a scene of 2,500 slots."""
import numpy as np
import pytest

from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import Sim

pytestmark = pytest.mark.gpu
SLOTS, ALL = 45_000_000, 1000


class Rows:
    def __init__(self, ptr, rows, comps, ty):
        self.__cuda_array_interface__ = dict(shape=(rows, comps), typestr=ty, data=(ptr, False), version=2)


def substep(slots, fluid, vel, mass):
    import torch
    d, p, _ = S.gpu_scene(3, slots, 30)
    d.table_size = 1 << 14
    sim = Sim(d, p)
    n, total = len(fluid), sim.info.total
    ptr = sim.device_ptrs()
    view = lambda q, c, ty="<f4": torch.as_tensor(Rows(q, total, c, ty), device="cuda")[total - n:]
    pos, prev, v, flags, dens = view(ptr.pos, 4), view(ptr.prev, 4), view(ptr.vel, 4), view(ptr.flags, 1, "<i4"), view(ptr.density, 2)
    sim.sync()
    f, w = torch.from_numpy(fluid).cuda(), torch.from_numpy(vel).cuda()
    pos[:, :3], prev[:, :3], v[:, :3] = f, f, w
    pos[:, 3] = 1.0 / mass
    flags[:] = 1
    torch.cuda.synchronize()
    sim.substep_partial(1 / 300, ALL)
    sim.sync()
    torch.cuda.synchronize()
    out = [t.cpu().numpy().copy() for t in (pos, v, dens, flags)]
    assert sim.health() == 0
    del pos, prev, v, flags, dens
    sim.close()
    return out


def test_list_rows_past_32_bits():
    import torch
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of free device memory")
    rng = np.random.default_rng(5)
    d, p, opts = S.gpu_scene(3, 16, 30)
    H, n = p.fluid_h, 2500
    # balls of 60 to 130 particles within half a list radius: lists up to the last row, some that overflow
    centre = np.stack(np.meshgrid(*[np.arange(3)] * 3, indexing="ij"), -1).reshape(-1, 3) * 3.1 * H + [0.5, 0.6, 0.5]
    of = np.repeat(np.arange(27), rng.integers(60, 131, 27))[:n]
    fluid = np.zeros((n, 3))
    fluid[:len(of)] = centre[of]
    fluid[len(of):] = centre[0] - [0, 0, 4 * H]
    u = rng.normal(size=(n, 3))
    fluid += u / np.linalg.norm(u, axis=1, keepdims=True) * (0.5 * H * rng.random((n, 1)) ** (1 / 3))
    fluid, vel = fluid.astype(np.float32), rng.normal(0, 0.2, (n, 3)).astype(np.float32)
    small, wide = substep(n, fluid, vel, opts["fluidMass"]), substep(SLOTS, fluid, vel, opts["fluidMass"])
    for a, b in zip(small, wide):
        assert np.array_equal(a, b)
