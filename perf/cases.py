"""Performance cases: the work a program has this package do, through its public entry points.

  frame   GpuSim.encode's frame of one resident scene (Sim.step): substeps x (grid, fluid, solid
          solve, contacts, bounds, xsph), from the CPU solver's small scene to 276k particles, plain and
          with the app's full schedule (tets, solid contact cache, companion cube, solid viscosity),
          with the hose and a grab, and with the state read back to the host every frame
  batch   many uneven scenes stepped together, then read back (what the frame server does per request)
  grid    the stateless hash-grid build over a caller's buffers
  groups  the connected pieces of a sliced body (Solver._recomputeGroups)
  pick    the ray pick behind every click

Scenes use the repository's own derivations (scenes.gpu_scene: 30 mm particles, 5 substeps;
scenes.solver_params for the CPU solver's scene). `pool` states are a settled basin: fluid in
layers on the floor (about 20 neighbours within H where the basin is full), moving at a few dm/s, the
body standing in it; `fall` states are the initial block dropping onto it. Inputs come from the seed alone (no simulated history).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from fluidphysics_b200 import _lib as L
from fluidphysics_b200 import batch as B
from fluidphysics_b200 import scenes as S
from fluidphysics_b200.sim import Sim

# One working stream for every handle, as a program that shares the GPU with torch sets it up.
_STREAM = None


def _stream() -> int:
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM.cuda_stream


# ------------------------------------------------------------------ the cases
def _frame(name, **kw):
    c = dict(name=name, kind="frame", rules="gpu", dim=20, fluid=65536, slots=0, radius_mm=30.0, iters=3, substeps=5,
             full=False, visc=0.0, state="pool", cut=False, hose=0, grab=0, read=False)
    c.update(kw)
    return c


def listed():
    return [
        # a click in the app: the smallest call, host-synchronous
        dict(name="pick_20", kind="pick", dim=20, reach=0.25),
        # the CPU solver's own scene (7^3 + 2,600), the page's first scene: launches and latency
        _frame("frame_cpu_scene", rules="cpu", dim=7, fluid=2600, state="fall"),
        # a phone-sized scene with odd counts and a ring buffer that is not full
        _frame("frame_ragged", dim=11, fluid=5003, slots=6007, iters=4),
        # the default scene settled in its basin, body sliced: the headline workload
        _frame("frame_default", cut=True),
        # the same frame with positions and flags read into pinned host memory (a CPU renderer)
        _frame("frame_default_read", read=True),
        # the largest interactive scene: block dropping, hose on, 64 particles grabbed
        _frame("frame_large", dim=24, fluid=262144, state="fall", hose=120, grab=64),
        # the app's own schedule: GpuSim's defaults (tets, contact cache, companion cube, 8 iterations)
        _frame("frame_full", full=True, iters=8),
        # the same schedule at a small odd size, solid viscosity on
        _frame("frame_full_small", full=True, iters=8, dim=9, fluid=7001, visc=0.05, cut=True),
        # served requests: 48 uneven scenes, two frames, state read back
        dict(name="batch_48", kind="batch", scenes=48, iters=3, frames=2),
        # the grid build alone over a caller's particles
        dict(name="grid_262k", kind="grid", n=262139, table=1 << 19),
        # the pieces of the default body after two cuts
        dict(name="groups_20", kind="groups", dim=20, cuts=2),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["frame", "frame", "frame", "full", "batch", "grid", "groups", "pick"])
    if kind == "frame":
        c = _frame("", dim=rng.randint(4, 22), fluid=log(600, 150000), iters=rng.randint(1, 8), substeps=rng.randint(4, 6),
                   state=rng.choice(["pool", "fall"]), cut=rng.random() < 0.5, read=rng.random() < 0.25,
                   radius_mm=rng.choice([25.0, 30.0, 36.0]))
    elif kind == "full":
        c = _frame("", full=True, dim=rng.randint(5, 20), fluid=log(600, 60000), iters=rng.randint(2, 8),
                   visc=rng.choice([0.0, 0.05]), cut=rng.random() < 0.5)
    elif kind == "batch":
        c = dict(kind="batch", scenes=rng.randint(3, 40), iters=rng.randint(2, 4), frames=rng.randint(1, 2))
    elif kind == "grid":
        n = log(1000, 262144)
        c = dict(kind="grid", n=n, table=1 << (math.ceil(math.log2(2 * n)) + rng.randint(0, 1)))
    elif kind == "groups":
        c = dict(kind="groups", dim=rng.randint(5, 24), cuts=rng.randint(0, 3))
    else:
        c = dict(kind="pick", dim=rng.randint(5, 24), reach=round(rng.uniform(0.1, 0.4), 4))
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ scenes
def _lattice(dim, spacing, centre, base):
    """Lattice positions and 26-neighbour constraints (a, b, rest) in the scene builder's order."""
    g = np.stack(np.meshgrid(*[np.arange(dim)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = np.asarray(centre)[None] - (dim - 1) * spacing / 2 + g * spacing
    a, b, r = [], [], []
    off = [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1) if (x, y, z) > (0, 0, 0)]
    for o in off:
        h = g + o
        ok = ((h >= 0) & (h < dim)).all(1)
        a.append(np.flatnonzero(ok))
        b.append((h[ok] * [dim * dim, dim, 1]).sum(1))
        r.append(np.full(ok.sum(), math.sqrt(sum(x * x for x in o) * spacing * spacing)))
    a, b, r = np.concatenate(a), np.concatenate(b), np.concatenate(r)
    o = np.lexsort((b, a))  # neighbours of one particle come in ascending index
    return pos, a[o] + base, b[o] + base, r[o]


def _tets(dim, base):
    idx = lambda x, y, z: base + (x * dim + y) * dim + z
    c = np.stack(np.meshgrid(*[np.arange(dim - 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x, y, z = c.T
    v = dict(A=idx(x, y, z), B=idx(x + 1, y, z), C=idx(x + 1, y + 1, z), D=idx(x, y + 1, z), E=idx(x, y, z + 1),
             F=idx(x + 1, y, z + 1), G=idx(x + 1, y + 1, z + 1), H=idx(x, y + 1, z + 1))
    pick = lambda names: np.stack([np.stack([v[k] for k in t], -1) for t in names], 1)
    even, odd = pick(["ACFH", "ABCF", "ACDH", "AEFH", "CFGH"]), pick(["BDEG", "ABDE", "BCDG", "DEHG", "BEFG"])
    return np.where((c.sum(1) % 2 == 0)[:, None, None], even, odd).reshape(-1, 4)


def _pool(rng, n, H, r, half, top):
    """n fluid particles in floor layers of a 6.8 m basin (as a settled pool packs them), clear of a
    body of half width `half` and height `top` standing at the origin."""
    s, out, have, layer = 0.62 * H, [], 0, 0
    side = min(6.8, s * math.ceil(math.sqrt(n + (2 * half / s) ** 2)) + 2 * s)
    while have < n:
        k = np.arange(-side / 2 + s / 2, side / 2 - s / 4, s) + rng.uniform(-0.25, 0.25) * s
        x, z = [q.ravel() for q in np.meshgrid(k, k, indexing="ij")]
        y = np.full(x.size, r + layer * 0.4 * H)
        p = np.stack([x, y, z], 1) + rng.uniform(-0.12, 0.12, (x.size, 3)) * s
        p[:, 1] = np.maximum(p[:, 1], r)
        p = p[~((np.abs(p[:, 0]) < half + r) & (np.abs(p[:, 2]) < half + r) & (p[:, 1] < top + r))]
        out.append(p)
        have += len(p)
        layer += 1
    return rng.permutation(np.concatenate(out)[:n])  # the ring buffer holds them in no spatial order


def _build(case, seed):
    """Descriptor, constants and initial state (float32, the layout of Sim.write_state) of a frame case."""
    rng = np.random.default_rng([int(seed), 17])
    if case["rules"] == "cpu":
        sc = S.cpu_scene(iters=case["iters"])
        d, p, fluid_mass = sc.desc, sc.params, 0.03
        d.solid_dim, d.max_fluid, d.substeps = case["dim"], max(case["slots"], case["fluid"]), case["substeps"]
    else:
        d, p, _ = S.gpu_scene(case["dim"], max(case["slots"], case["fluid"]), case["radius_mm"], iters=case["iters"],
                              substeps=case["substeps"], features=L.FEAT_TETS | L.FEAT_SOLID_CONTACTS if case["full"] else 0)
        if case["full"]:  # the companion cube of GpuSim's constructor
            d.solid_dim2 = max(2, S.js_round((d.solid_dim - 1) / 20 ** (1 / 3)) + 1)
            d.cube2_center[:] = [1.1, (d.solid_dim2 - 1) * d.spacing / 2 + p.solid_radius, 0.7]
        S.set_params(p, {"solidViscosity": case["visc"]})
        fluid_mass = d.fluid_mass
    half = (d.solid_dim - 1) * d.spacing / 2
    if case["state"] == "pool":
        d.cube_center[:] = [0.0, half + p.solid_radius, 0.0]
    pos, a, b, rest = _lattice(d.solid_dim, d.spacing, list(d.cube_center), 0)
    tets = _tets(d.solid_dim, 0)
    if d.solid_dim2:
        q, a2, b2, r2 = _lattice(d.solid_dim2, d.spacing, list(d.cube2_center), len(pos))
        tets = np.concatenate([tets, _tets(d.solid_dim2, len(pos))])
        pos, a, b, rest = np.concatenate([pos, q]), np.concatenate([a, a2]), np.concatenate([b, b2]), np.concatenate([rest, r2])
    n_s, n_f = len(pos), case["fluid"]
    lattice = pos.astype(np.float32)
    alive = np.ones(len(a), np.uint32)
    if case["cut"]:  # the body is already sliced once, through a random plane near its centre
        nrm = rng.normal(size=3)
        side = (pos - np.asarray(list(d.cube_center)) - 0.2 * d.spacing) @ nrm > 0
        alive[side[a] != side[b]] = 0
    body = pos + rng.uniform(-0.02, 0.02, pos.shape) * d.spacing
    body_v = rng.normal(0, 0.1, pos.shape)
    if case["state"] == "pool":
        fp = _pool(rng, n_f, p.fluid_h, p.fluid_radius, half, 2 * half + p.solid_radius)
        fv = 0.35 * np.sin(fp[:, [2, 0, 1]] * 1.7 + rng.uniform(0, 6.28, 3)) + rng.normal(0, 0.05, fp.shape)
        fv[:, 1] *= 0.1
    else:  # a jittered block dropping from above the body
        ny = 16 if n_f < 200000 else 64
        nx = max(1, math.ceil(math.sqrt(n_f / ny)))
        y0 = max(1.7, d.cube_center[1] + half + 3 * p.fluid_radius)
        fp = S.jittered_block(nx, ny, nx, 2.2 * p.fluid_radius, y0, int(seed))[:n_f]
        fv = np.zeros((n_f, 3)) + [0, -1.5, 0] + rng.normal(0, 0.2, (n_f, 3))
        body_v[:, 1] -= 1.0
    N = n_s + d.max_fluid
    st = dict(pos=np.zeros((N, 4), np.float32), prev=np.zeros((N, 4), np.float32), vel=np.zeros((N, 4), np.float32),
              density=np.zeros((N, 2), np.float32), flags=np.zeros(N, np.uint32))
    st["pos"][:n_s, :3], st["pos"][:n_s, 3] = body, 1 / d.solid_mass
    st["pos"][n_s:, 3] = 1 / fluid_mass
    st["pos"][n_s:n_s + n_f, :3] = fp
    st["prev"][:, :3] = st["pos"][:, :3]
    st["vel"][:n_s, :3], st["vel"][n_s:n_s + n_f, :3] = body_v, fv
    st["flags"][:n_s] = 1
    st["flags"][n_s:n_s + n_f] = 1
    cons = np.stack([a, b, rest.astype(np.float32).view(np.uint32), alive], 1).astype(np.uint32)
    return dict(desc=d, params=p, state=st, cons=cons, tets=tets, lattice=lattice, n_s=n_s)


class _Buffer:
    """A device buffer of the handle, for torch.as_tensor (no copy); the tensor keeps the handle open."""

    def __init__(self, sim, ptr, shape, typestr):
        self.sim = sim
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=2)


def _open(bld):
    sim = Sim(bld["desc"], bld["params"])
    sim.set_stream(_stream())
    sim.write_state(**bld["state"])
    sim.write_constraints(bld["cons"])
    return sim


def _views(sim):
    """The resident state as tensors over the handle's own buffers, as a renderer reads it."""
    p, n, c = sim.device_ptrs(), sim.info.total, sim.info.num_cons
    t = lambda ptr, shape, ty: torch.as_tensor(_Buffer(sim, ptr, shape, ty), device="cuda")
    cons = t(p.cons, (c, 4), "<i4")
    return dict(pos=t(p.pos, (n, 4), "<f4"), vel=t(p.vel, (n, 4), "<f4"), density=t(p.density, (n, 2), "<f4"),
                flags=t(p.flags, (n,), "<i4"), rest=cons.view(torch.float32)[:, 2], alive=cons[:, 3])


def _batch_sizes(case):
    """Body edge and fluid count of each scene: the case's own, whatever the seed."""
    rng = np.random.default_rng(case["scenes"])
    return [(int(rng.integers(6, 21)), int(2 ** rng.uniform(11, 15.5))) for _ in range(case["scenes"])]


def _batch_scenes(case, seed):
    rng = np.random.default_rng([int(seed), 23])
    out = []
    for k, (dim, nf) in enumerate(_batch_sizes(case)):
        sc = B.batch_scene(dim, nf, int(seed) * 1000 + k, iters=case["iters"])
        if k % 2:  # every other scene is settled
            half = (dim - 1) * sc.desc.spacing / 2
            sc.desc.cube_center[:] = [0.0, half + sc.params.solid_radius, 0.0]
            sc.fluid_pos = _pool(rng, nf, sc.params.fluid_h, sc.params.fluid_radius, half, 2 * half + sc.params.solid_radius).astype(np.float32)
        sc.fluid_vel = rng.normal(0, 0.3, (nf, 3)).astype(np.float32)
        out.append(sc)
    return out


def _body(case, seed):
    return _build(_frame("", dim=case["dim"], fluid=600, state="pool"), seed)


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        bld = _build(case, seed)
        sim = _open(bld)
        st = dict(kind=kind, sim=sim, dt=1 / 60, substeps=case["substeps"], out=_views(sim), frame=0, hose=None, grab=False)
        if case["hose"]:
            sc = S.Scene("", bld["desc"], bld["params"], None, None, 0.0, 1 / 60, 5, 0, hose_per_frame=case["hose"], hose_seed=int(seed))
            st["hose"], st["count"] = S.hose_script(sc, 64), case["hose"]
        if case["grab"]:
            sim.grab_indices(S.grab_set(bld["lattice"], case["dim"] ** 3, case["dim"], case["grab"]))
            st["grab"] = True
        if case["read"]:
            n = sim.info.total
            st["host"] = (torch.empty(n, 4, pin_memory=True), torch.empty(n, dtype=torch.int32, pin_memory=True))
            st["np"] = (st["host"][0].numpy(), st["host"][1].numpy().view(np.uint32))
        return st
    if kind == "batch":
        scenes = _batch_scenes(case, seed)
        b = B.Batch(solid_iters=case["iters"], max_scenes=64, block_threads=128, ctas_per_sm=128)
        b.set_stream(_stream())
        ids = [b.add_scene(s) for s in scenes]
        n = [s.total for s in scenes]
        at = np.concatenate([[0], np.cumsum(n)])
        host = [torch.empty(at[-1], 4, pin_memory=True), torch.empty(at[-1], 4, pin_memory=True),
                torch.empty(at[-1], dtype=torch.int32, pin_memory=True)]
        flat = [h.numpy() for h in host]
        ptrs = [(i, L.fptr(flat[0][at[k]:at[k + 1]]), L.fptr(flat[1][at[k]:at[k + 1]]), L.uptr(flat[2].view(np.uint32)[at[k]:at[k + 1]]))
                for k, i in enumerate(ids)]
        return dict(kind=kind, batch=b, frames=case["frames"], ptrs=ptrs, out=dict(pos=host[0], vel=host[1], flags=host[2]))
    if kind == "grid":
        n, T = case["n"], case["table"]
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        H = 0.078
        side = 6.8
        pos = torch.rand(n, 4, generator=g, device="cuda")
        pos[:, 0] = (pos[:, 0] - 0.5) * side
        pos[:, 2] = (pos[:, 2] - 0.5) * side
        pos[:, 1] *= n / (7.0 / H ** 3 * side * side)  # about 7 to a cell, a pool's packing
        flags = (torch.rand(n, generator=g, device="cuda") < 0.97).to(torch.int32)
        out = dict(counts=torch.empty(T, dtype=torch.int32, device="cuda"), offsets=torch.empty(T + 1, dtype=torch.int32, device="cuda"),
                   entries=torch.zeros(n, dtype=torch.int32, device="cuda"))
        p = lambda t: C.c_void_p(t.data_ptr())
        args = (p(pos), p(flags), n, T, H, p(out["counts"]), p(out["offsets"]), p(out["entries"]), C.c_void_p(_stream()))
        return dict(kind=kind, lib=L.load(), args=args, keep=(pos, flags), out=out)
    bld = _body(case, seed)
    rng = np.random.default_rng([int(seed), 29])
    if kind == "groups":
        side = np.zeros(bld["n_s"], np.int64)
        ctr = bld["lattice"].mean(0)
        for k in range(case["cuts"]):
            side += ((bld["lattice"] - ctr + rng.normal(0, 0.05, 3)) @ rng.normal(size=3) > 0).astype(np.int64) << k
        a, b = bld["cons"][:, 0], bld["cons"][:, 1]
        bld["cons"][side[a] != side[b], 3] = 0
        sim = _open(bld)
        out = torch.empty(bld["n_s"], dtype=torch.int32, device="cuda")
        return dict(kind=kind, sim=sim, out=out)
    ro, rd = _ray(bld, rng)
    return dict(kind=kind, sim=_open(bld), ro=ro, rd=rd, reach=case["reach"])


def _ray(bld, rng):
    target = bld["state"]["pos"][int(rng.integers(bld["n_s"])), :3].astype(np.float64) + rng.normal(0, 0.01, 3)
    ro = np.array([rng.uniform(-3, 3), 2.5, 4.0])
    rd = target - ro
    return ro, rd / np.linalg.norm(rd)


def run(state):
    kind = state["kind"]
    if kind == "frame":
        sim = state["sim"]
        if state["hose"] is not None:
            sim.emit(state["count"], *state["hose"][state["frame"] % 64])
        if state["grab"]:
            k = state["frame"]
            sim.grab_move([0.0, 0.3 * (math.sin(math.pi * (k + 1) / 60) - math.sin(math.pi * k / 60)), 0.0])
        sim.step(state["dt"], state["substeps"])
        state["frame"] += 1
        if "host" not in state:
            return state["out"]
        sim.read_state_async(*state["np"])
        sim.read_wait()
        return dict(state["out"], host_pos=state["host"][0], host_flags=state["host"][1])
    if kind == "batch":
        b = state["batch"]
        for _ in range(state["frames"]):
            b.step(1 / 60, 5)
        for i, pos, vel, flags in state["ptrs"]:
            L.check_batch(b.lib, b.h, b.lib.upbd_batch_read_state(b.h, i, pos, None, vel, None, flags))
        return state["out"]
    if kind == "grid":
        L.check(state["lib"], None, state["lib"].upbd_grid_build(*state["args"]))
        return state["out"]
    if kind == "groups":
        state["sim"].groups_device(state["out"].data_ptr())
        return state["out"]
    i, t = state["sim"].pick(state["ro"], state["rd"], state["reach"])
    return dict(id=int(i), t=float(t))


# ------------------------------------------------------------------ compulsory work
def _sizes(case):
    n1 = case["dim"] ** 3
    n2 = (max(2, S.js_round((case["dim"] - 1) / 20 ** (1 / 3)) + 1) ** 3) if case.get("full") else 0
    cons = lambda m: 3 * m * m * (m - 1) + 6 * m * (m - 1) ** 2 + 4 * (m - 1) ** 3
    m2 = round(n2 ** (1 / 3))
    return n1 + n2, cons(case["dim"]) + (cons(m2) if n2 else 0), 5 * ((case["dim"] - 1) ** 3 + (max(m2 - 1, 0)) ** 3)


def _frame_work(s_n, c_n, t_n, fluid, slots, iters, substeps, full, read):
    """One frame reads and writes the persistent state once (pos, prev, vel: 48 B a particle in, 48 out; density
    8 out; flags 4; constraints 16 in, tets 20 in). Its arithmetic: per substep about 30 neighbours a fluid
    particle at 60 operations over the three gathers, 30 a constraint end and iteration, 150 a tet corner."""
    n = s_n + fluid
    by = n * (96 + 8 + 4) + 16 * c_n + (20 * t_n if full else 0)
    if read:
        by += (s_n + slots) * 20
    fl = substeps * (fluid * 30 * 60 + n * 80 + 2 * c_n * 30 * iters + (4 * t_n * 150 * iters if full else 0))
    return dict(bytes=by, flops=fl)


def work(case):
    kind = case["kind"]
    if kind == "frame":
        s_n, c_n, t_n = _sizes(case)
        return _frame_work(s_n, c_n, t_n, case["fluid"], max(case["slots"], case["fluid"]), case["iters"], case["substeps"],
                           case["full"], case["read"])
    if kind == "batch":
        by, fl = 0.0, 0.0
        for dim, nf in _batch_sizes(case):
            s_n, c_n, t_n = _sizes(dict(dim=dim))
            w = _frame_work(s_n, c_n, t_n, nf, 0, case["iters"], 5, False, False)
            by, fl = by + w["bytes"] * case["frames"], fl + w["flops"] * case["frames"]
        return dict(bytes=by, flops=fl)
    if kind == "grid":
        return dict(bytes=case["n"] * (16 + 4 + 4) + case["table"] * 8, flops=case["n"] * 20)
    s_n, c_n, _ = _sizes(case)
    if kind == "groups":
        return dict(bytes=c_n * 16 + s_n * 4, flops=c_n * 4)
    return dict(bytes=s_n * 20, flops=s_n * 25)


# ------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    """The outputs in 64-bit arithmetic. Whole numbers (grid, groups) have no other value than the exact one.
    The hose has none (its jitter is a hash of the low bits of a 32-bit sine), and a batch takes too long."""
    if case["kind"] == "pick":
        bld = _body(case, seed)
        ro, rd = _ray(bld, np.random.default_rng([int(seed), 29]))
        mp = case["reach"]
        p = bld["state"]["pos"][:bld["n_s"], :3].astype(np.float64) - ro
        t = p @ rd
        hit = (t >= 0) & (((p - t[:, None] * rd) ** 2).sum(1) <= mp * mp)
        return dict(id=None, t=float(t[hit].min()) if hit.any() else math.inf)
    if case["kind"] != "frame" or case["hose"] or case["grab"]:
        return None
    r = _exact_frame(_build(case, seed), case)
    out = dict(pos=r["pos"], vel=r["vel"], density=r["density"], flags=None, rest=r["rest"], alive=None)
    if case["read"]:
        out.update(host_pos=r["pos"], host_flags=None)
    return out


class _Grid64:
    """Particles by hash bucket (the three primes of Solver._hash); pairs() walks the 27 cells around points."""
    K = (92837111, 689287499, 283923481)

    def __init__(self, pos, ids, inv, table):
        self.inv, self.mask, self.ids, dev = inv, table - 1, ids, pos.device
        c = torch.floor(pos[ids] * inv).long()
        h = self._hash(c[:, 0], c[:, 1], c[:, 2])
        self.order = ids[torch.argsort(h, stable=True)]
        self.count = torch.bincount(h, minlength=table)
        self.start = torch.cumsum(self.count, 0) - self.count
        self.dev = dev

    def _hash(self, x, y, z):
        return ((x * self.K[0]) ^ (y * self.K[1]) ^ (z * self.K[2])) & self.mask

    def pairs(self, who, p):
        c = torch.floor(p[who] * self.inv).long()
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dz in (-1, 0, 1):
                    h = self._hash(c[:, 0] + dx, c[:, 1] + dy, c[:, 2] + dz)
                    n = self.count[h]
                    k = torch.repeat_interleave(torch.arange(len(who), device=self.dev), n)
                    if k.numel() == 0:
                        continue
                    at = torch.arange(k.numel(), device=self.dev) - (torch.cumsum(n, 0) - n)[k] + self.start[h][k]
                    yield who[k], self.order[at]


def _clamp_len(d, lim):
    n = d.norm(dim=1, keepdim=True)
    return torch.where(n > lim, d * (lim / n.clamp_min(1e-300)), d)


def _exact_frame(bld, case):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    D = torch.float64
    f32 = lambda x: float(np.float32(x))
    P, d, S_n = bld["params"], bld["desc"], bld["n_s"]
    g = {k: f32(getattr(P, k)) for k in S.PARAM_NAMES.values() if k not in ("tear_mode", "plastic_clamp")}
    up = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
    pos4, vel4 = up(bld["state"]["pos"]).to(D), up(bld["state"]["vel"]).to(D)
    pos, w, vel = pos4[:, :3].clone(), pos4[:, 3].clone(), vel4[:, :3].clone()
    act = up(bld["state"]["flags"].astype(np.int64)) > 0
    N = len(pos)
    solid = torch.arange(N, device=dev) < S_n
    rho2 = torch.zeros(N, 2, dtype=D, device=dev)
    ca, cb = up(bld["cons"][:, 0].astype(np.int64)), up(bld["cons"][:, 1].astype(np.int64))
    rest = up(bld["cons"][:, 2].astype(np.uint32).view(np.float32).astype(np.float64))
    alive = up(bld["cons"][:, 3].astype(np.int64)) > 0
    deg = torch.bincount(torch.cat([ca, cb]), minlength=max(S_n, 1))
    pair = 1.0 / torch.maximum(deg[ca], deg[cb]).to(D)
    rest0 = rest.clone()  # lattice rest lengths
    lat = up(bld["lattice"]).to(D)
    n1 = case["dim"] ** 3
    tet = up(bld["tets"].astype(np.int64))
    if case["full"]:
        q = [lat[tet[:, k]] for k in range(4)]
        vol = (torch.cross(q[1] - q[0], q[2] - q[0], dim=1) * (q[3] - q[0])).sum(1) / 6
        tdeg = torch.bincount(tet.reshape(-1), minlength=S_n)
        tscale = 1.0 / tdeg[tet].max(1).values.to(D)
        bonded = lambda: torch.cat([ca[alive] * S_n + cb[alive], cb[alive] * S_n + ca[alive]]).sort().values

    def cell_of(i):  # lattice coordinates and the lattice of a solid
        second = i >= n1
        dim = torch.where(second, torch.full_like(i, max(d.solid_dim2, 1)), torch.full_like(i, d.solid_dim))
        k = torch.where(second, i - n1, i)
        return second, torch.stack([k // (dim * dim), (k // dim) % dim, k % dim], 1)

    def rsum_of(i, j):
        (si, gi), (sj, gj) = cell_of(i), cell_of(j)
        near = (si == sj) & ((gi - gj).abs().max(1).values <= 1)
        full = 2 * g["solid_radius"]
        return torch.where(near, torch.full((len(i),), min(full, f32(d.spacing) * 0.97), dtype=D, device=dev),
                           torch.full((len(i),), full, dtype=D, device=dev))

    H, rs, rf = g["fluid_h"], g["solid_radius"], g["fluid_radius"]
    inv, h = 1.0 / P.cell_size, f32((1 / 60) / case["substeps"])
    sol = torch.arange(S_n, device=dev)
    for _ in range(case["substeps"]):
        fluid = torch.nonzero(act & ~solid)[:, 0]
        prev = pos.clone()
        vel = torch.where(act[:, None], vel + torch.tensor([0, g["gravity"] * h, 0], dtype=D, device=dev), vel)
        pos = torch.where(act[:, None], pos + vel * h, pos)
        F, Sg = _Grid64(pos, fluid, inv, d.table_size), _Grid64(pos, sol, inv, d.table_size)
        # density
        rho = torch.zeros(N, 2, dtype=D, device=dev)
        for i, j in F.pairs(fluid, pos):
            r2 = ((pos[j] - pos[i]) ** 2).sum(1)
            k = (r2 < H * H) & (i != j)
            q = 1 - r2[k].sqrt() / H
            rho.index_add_(0, i[k], torch.stack([q * q, q ** 3], 1))
        rho2[fluid] = rho[fluid]
        # displacement
        Pr, Pn = g["stiffness"] * (rho[:, 0] - g["rest_density"]), g["near_stiffness"] * rho[:, 1]
        dsp = torch.zeros(N, 3, dtype=D, device=dev)
        for i, j in F.pairs(fluid, pos):
            e = pos[j] - pos[i]
            r2 = (e ** 2).sum(1)
            k = (r2 < H * H) & (r2 >= 1e-12) & (i != j)
            i, j, e, r = i[k], j[k], e[k], r2[k].sqrt()
            q = 1 - r / H
            m = (0.25 * ((Pr[i] + Pr[j]) * q + (Pn[i] + Pn[j]) * q * q)).clamp(-0.05 * H, 0.05 * H)
            dsp.index_add_(0, i, -e * (m / r)[:, None])
        pos = torch.where((act & ~solid)[:, None], pos + _clamp_len(dsp, 0.35 * H), pos)
        # solids
        contacts = []
        if case["full"]:
            bd = bonded()
            for i, j in Sg.pairs(sol, pos):
                lim = rsum_of(i, j) + 2 * rs
                k = (((pos[i] - pos[j]) ** 2).sum(1) < lim * lim) & (i != j)
                i, j = i[k], j[k]
                key = i * S_n + j
                at = torch.searchsorted(bd, key).clamp_max(max(len(bd) - 1, 0))
                k = bd[at] != key if len(bd) else torch.ones_like(key, dtype=torch.bool)
                contacts.append((i[k], j[k]))
        alpha = g["compliance"] / (h * h)
        for _ in range(case["iters"]):
            e = pos[ca] - pos[cb]
            r = e.norm(dim=1)
            k = alive & (r >= 1e-9)
            f = torch.where(k, -(r - rest) / (w[ca] + w[cb] + alpha) / r.clamp_min(1e-9) * pair, torch.zeros_like(r))
            dl = torch.zeros(N, 3, dtype=D, device=dev)
            dl.index_add_(0, ca, e * (f * w[ca])[:, None])
            dl.index_add_(0, cb, -e * (f * w[cb])[:, None])
            pos = pos + dl * g["omega"]
            if case["full"]:
                q = [pos[tet[:, k]] for k in range(4)]
                b_, c_, d_ = q[1] - q[0], q[2] - q[0], q[3] - q[0]
                V = (torch.cross(b_, c_, dim=1) * d_).sum(1) / 6
                gb, gc, gd = [torch.cross(x, y, dim=1) / 6 for x, y in ((c_, d_), (d_, b_), (b_, c_))]
                gs = [-(gb + gc + gd), gb, gc, gd]
                wa = w[tet[:, 0]]
                den = wa * sum((x ** 2).sum(1) for x in gs)
                ok = (vol > 0) & (den >= 1e-12)
                fac = torch.where(ok, -(V - vol) / den.clamp_min(1e-300) * wa * tscale, torch.zeros_like(V))
                dl = torch.zeros(N, 3, dtype=D, device=dev)
                for k in range(4):
                    dl.index_add_(0, tet[:, k], _clamp_len(gs[k] * fac[:, None], 0.5 * rs))
                pos = pos + _clamp_len(dl, 0.5 * rs)
                dl = torch.zeros(N, 3, dtype=D, device=dev)
                for i, j in contacts:
                    e, lim = pos[i] - pos[j], rsum_of(i, j)
                    r2 = (e ** 2).sum(1)
                    k = (r2 < lim * lim) & (r2 >= 1e-12)
                    i, j, e, r, lim = i[k], j[k], e[k], r2[k].sqrt(), lim[k]
                    dl.index_add_(0, i, e * ((lim - r) / r * w[i] / (w[i] + w[j]) * 0.5)[:, None])
                pos = pos + _clamp_len(dl, 0.5 * rs)
        # bonds (and tets) on the solved positions
        r = (pos[ca] - pos[cb]).norm(dim=1)
        tear = r > rest * g["break_strain"] if P.tear_mode == 1 else r > rest + g["tear_gap"] * 2 * rs
        nr = torch.where(((r - rest) / rest).abs() > g["plastic_threshold"], rest + (r - rest) * g["plastic_rate"], rest)
        if P.plastic_clamp:
            nr = torch.minimum(torch.maximum(nr, 0.9 * rest0), 1.25 * rest0)
        rest = torch.where(alive & ~tear, nr, rest)
        alive = alive & ~tear
        if case["full"]:
            for a in range(3):
                for b in range(a + 1, 4):
                    r0 = (lat[tet[:, a]] - lat[tet[:, b]]).norm(dim=1)
                    far = (pos[tet[:, a]] - pos[tet[:, b]]).norm(dim=1) > r0 + g["tear_gap"] * 2 * rs
                    vol = torch.where(far, -vol.abs(), vol)
        # solid-fluid contacts
        dl = torch.zeros(N, 3, dtype=D, device=dev)
        for grid, who in ((F, sol), (Sg, fluid)):
            for i, j in grid.pairs(who, pos):
                e = pos[i] - pos[j]
                r2 = (e ** 2).sum(1)
                k = (r2 < (rs + rf) ** 2) & (r2 >= 1e-12)
                i, j, e, r = i[k], j[k], e[k], r2[k].sqrt()
                dl.index_add_(0, i, e * ((rs + rf - r) / r * w[i] / (w[i] + w[j]) * g["contact_scale"])[:, None])
        rad = torch.where(solid, rs, rf).to(D)
        p = torch.where(act[:, None], pos + _clamp_len(dl, rad[:, None]), pos)
        # bounds
        low = p[:, 1] < rad
        mu = torch.where(solid, g["friction_solid"], g["friction_fluid"]).to(D)
        x, y, z = p[:, 0], torch.where(low, rad, p[:, 1]), p[:, 2]
        x = torch.where(low, x - (x - prev[:, 0]) * mu, x)
        z = torch.where(low, z - (z - prev[:, 2]) * mu, z)
        wallish = y < g["wall_h"] + rad
        lim = rad + g["wall_t"]
        for ax, wl in ((0, g["wall_x"]), (1, g["wall_z"])):
            c = x if ax == 0 else z
            hit = wallish & ((c.abs() - wl).abs() < lim)
            c = torch.where(hit, torch.sign(c) * torch.where(c.abs() < wl, wl - lim, wl + lim), c)
            x, z = (c, z) if ax == 0 else (x, c)
        p = torch.stack([x, y, z], 1)
        was = act
        cull = act & ~solid & ((y < -3.0) | (x * x + z * z > g["cull_r"] ** 2))
        pos = torch.where(was[:, None], p, pos)
        act = act & ~cull
        # velocities
        damp = torch.where(solid, g["damp_solid"], g["damp_fluid"]).to(D)
        nv = _clamp_len((pos - prev) / h * (1 - damp * h).clamp_min(0)[:, None], g["max_speed"])
        vel = torch.where(act[:, None], nv, vel)
        if case["visc"] > 0:
            k = alive
            m, s = torch.zeros(N, dtype=D, device=dev), torch.zeros(N, 3, dtype=D, device=dev)
            for i, j in ((ca[k], cb[k]), (cb[k], ca[k])):
                m.index_add_(0, i, torch.ones(len(i), dtype=D, device=dev))
                s.index_add_(0, i, vel[j])
            has = (m > 0) & solid
            sv = torch.where(has[:, None], vel + g["solid_viscosity"] * (s / m.clamp_min(1)[:, None] - vel), vel)
        # xsph on the fluid (the solids' smoothed velocities take no part)
        m, s = torch.zeros(N, dtype=D, device=dev), torch.zeros(N, 3, dtype=D, device=dev)
        mine = torch.nonzero(act & ~solid)[:, 0]
        for i, j in F.pairs(mine, pos):
            k = (((pos[j] - pos[i]) ** 2).sum(1) < H * H) & (i != j)
            m.index_add_(0, i[k], torch.ones(int(k.sum()), dtype=D, device=dev))
            s.index_add_(0, i[k], vel[j[k]])
        has = (m > 0) & act & ~solid
        out = torch.where(has[:, None], vel + g["viscosity"] * (s / m.clamp_min(1)[:, None] - vel), vel)
        vel = torch.where(solid[:, None], sv, out) if case["visc"] > 0 else out
    return dict(pos=torch.cat([pos, w[:, None]], 1), vel=torch.cat([vel, vel4[:, 3:]], 1), density=rho2, rest=rest)
