"""Performance cases: the work a program has this library do, through its public entry points.

A case is a dict of plain values.  "frame" cases advance hair objects by one dynamic frame -- on the
batched path (one graph launch, path = "batch") or on the plain path (one dispatch per object per
stage, path = "plain") --, "sdf" rebuilds a collision grid, "quads" expands strands for a renderer,
"query" and "train" run the learned collision proxy.  Inputs come from the seed alone; sizes come from
the case.  Every frame starts from a moving state (positions and velocities, no reset), written with
the snapshot / restore calls.

exact() restates the same computations in 64 bits with plain torch.  Which cells a triangle visits is
decided in 32 bits there too, because that choice is part of the definition (a cell is set or not).
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

DEV = "cuda" if torch.cuda.is_available() else "cpu"
TICKS = 4          # frame inputs a state cycles through: a pose swinging there and back
DT = 1.0 / 60.0
FRAME0 = 10        # simulation frame of the first pass (frames below 2 reset the positions)


def listed():
    return [
        # the smallest frame a program issues: one short-haired object, nothing to collide with
        dict(name="strands_small", kind="frame", path="batch", objects=1, guides=2048, n=16, follow=0, tris=0, gx=0, gy=0,
             gz=0, local=1, length=1, wind=0.0, layout=0),
        # one game character: a shipped-asset-sized hair (2,240 guides, four follow hairs) on a 25k-triangle body
        dict(name="character", kind="frame", path="batch", objects=1, guides=2240, n=32, follow=4, tris=25800, gx=64, gy=96,
             gz=56, local=2, length=2, wind=1.0, layout=0),
        # the same character driven dispatch by dispatch, as a host that follows the reference's loop does
        dict(name="character_plain", kind="frame", path="plain", objects=1, guides=2240, n=32, follow=4, tris=25800, gx=64,
             gy=96, gz=56, local=2, length=2, wind=1.0, layout=0),
        # the film head: 20,000 guides with four follow hairs, 64^3 grid
        dict(name="head", kind="frame", path="batch", objects=1, guides=20000, n=32, follow=4, tris=20000, gx=64, gy=64, gz=64,
             local=3, length=3, wind=2.0, layout=0),
        # fur: many short strands, a fine grid
        dict(name="fur", kind="frame", path="batch", objects=1, guides=200000, n=16, follow=0, tris=50000, gx=128, gy=128,
             gz=128, local=2, length=2, wind=0.0, layout=0),
        # a crowd: sixteen uneven objects, each on its own mesh and grid, strand lengths mixed
        dict(name="crowd", kind="frame", path="batch", objects=16, guides=0, n=0, follow=0, tris=0, gx=0, gy=0, gz=0, local=2,
             length=2, wind=1.5, layout=6),
        # few odd-sized objects: strand counts off every tile, follow hairs on some, grids that are not cubes
        dict(name="ragged", kind="frame", path="batch", objects=3, guides=0, n=0, follow=0, tris=0, gx=0, gy=0, gz=0, local=2,
             length=2, wind=0.5, layout=-1),
        # long hair on the plain path, odd grid
        dict(name="long_plain", kind="frame", path="plain", objects=1, guides=6007, n=64, follow=1, tris=9000, gx=49, gy=53,
             gz=47, local=2, length=2, wind=1.0, layout=0),
        # a collision grid rebuilt from a skinned mesh every frame, on its own
        dict(name="sdf_rebuild", kind="sdf", tris=50000, gx=128, gy=128, gz=128),
        # the renderer's vertices of a head's strands
        dict(name="strand_quads", kind="quads", guides=20000, n=32, follow=4, shadow=0),
        # the learned proxy asked for the distances of a head's guide vertices
        dict(name="proxy_query", kind="query", points=640000),
        # a stretch of the proxy's training
        dict(name="proxy_train", kind="train", samples=262144, batch=8192, steps=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["sdf", "quads", "query", "train"])
    if kind == "frame":
        if rng.random() < 0.3:
            while True:   # no more than the listed crowd's vertices and triangles
                c = dict(kind="frame", path="batch", objects=rng.randint(2, 12), guides=0, n=0, follow=0, tris=0, gx=0, gy=0, gz=0,
                         local=rng.randint(1, 3), length=rng.randint(1, 3), wind=rng.choice([0.0, 1.5]),
                         layout=rng.randint(1, 1 << 20))
                o = _specs(c)
                if sum(x["guides"] * x["n"] for x in o) <= 5_000_000 and sum(x["tris"] for x in o) <= 180_000:
                    return c
        n = rng.choice([8, 16, 32, 64])
        follow = rng.choice([0, 0, 1, 2, 4])
        guides = _log(rng, 300, 1_600_000 // (n * (follow + 1)))
        collide = rng.random() < 0.85
        g = [_log(rng, 24, 128) for _ in range(3)] if collide else [0, 0, 0]
        return dict(kind="frame", path=rng.choice(["batch", "batch", "plain"]), objects=1, guides=guides, n=n, follow=follow,
                    tris=_log(rng, 1500, 40000) if collide else 0, gx=g[0], gy=g[1], gz=g[2], local=rng.randint(1, 3),
                    length=rng.randint(1, 3), wind=rng.choice([0.0, 2.0]), layout=0)
    if kind == "sdf":
        return dict(kind="sdf", tris=_log(rng, 1500, 50000), gx=_log(rng, 24, 128), gy=_log(rng, 24, 128), gz=_log(rng, 24, 128))
    if kind == "quads":
        n = rng.choice([8, 16, 32, 64])
        return dict(kind="quads", guides=_log(rng, 300, 600000 // n), n=n, follow=rng.randint(0, 4), shadow=rng.randint(0, 1))
    if kind == "query":
        return dict(kind="query", points=_log(rng, 500, 640000))
    return dict(kind="train", samples=_log(rng, 10000, 262144), batch=512 * rng.randint(1, 16), steps=rng.randint(16, 64))


# ------------------------------------------------------------------------------------------ what a case holds
def _specs(case):
    """One dict of sizes and settings per hair object."""
    if case["objects"] == 1:
        o = {k: case[k] for k in ("guides", "n", "follow", "tris", "local", "length", "wind")}
        return [dict(o, grid=(case["gx"], case["gy"], case["gz"]), damping=0.06, stiff=0.85, glob=0.35)]
    if case["layout"] == -1:
        rows = [(777, 64, 0, 6100, (37, 41, 53)), (1013, 8, 2, 3300, (33, 29, 47)), (131, 4, 1, 1700, (45, 31, 27))]
        return [dict(guides=g, n=n, follow=f, tris=t, grid=d, local=case["local"], length=case["length"], wind=case["wind"],
                     damping=0.05, stiff=0.7, glob=0.3) for g, n, f, t, d in rows]
    r = random.Random(case["layout"])
    out = []
    for _ in range(case["objects"]):
        cells = r.choice([32, 48, 64, 96, 128])
        out.append(dict(guides=(_log(r, 512, 50000) + 63) // 64 * 64, n=r.choice([8, 16, 32, 64]), follow=0, tris=_log(r, 5000, 30000),
                        grid=(cells,) * 3, local=case["local"], length=case["length"], wind=r.uniform(0.0, case["wind"]),
                        damping=r.uniform(0.01, 0.1), stiff=r.uniform(0.1, 0.9), glob=r.uniform(0.1, 0.9)))
    return out


def _settings(o):
    return dict(vsp_coeff=0.7, vsp_accel_threshold=1.2, local_constraint_stiffness=o["stiff"],
                local_constraints_iterations=o["local"], global_constraint_stiffness=o["glob"], global_constraints_range=0.3,
                length_constraints_iterations=o["length"], damping=o["damping"], gravity_magnitude=9.8, tip_separation=1.0,
                wind_magnitude=o["wind"])


def _bone(rot, pivot):
    """Row-vector 4x4 of a rotation about a pivot."""
    m = np.eye(4)
    m[:3, :3] = rot.T
    m[3, :3] = np.asarray(pivot) - np.asarray(pivot) @ rot.T
    return m.astype(np.float32).reshape(16)


def _pose(center, phase, tick):
    """Three joints: the neck (still), a nod and a turn of up to some degrees a tick."""
    pivot = (center[0], center[1] - 0.12, center[2])
    s = math.sin(2.0 * math.pi * (tick / TICKS + phase))
    a, b = math.radians(2.0) * s, math.radians(3.0) * s
    rx = np.array([[1, 0, 0], [0, math.cos(a), -math.sin(a)], [0, math.sin(a), math.cos(a)]])
    ry = np.array([[math.cos(b), 0, math.sin(b)], [0, 1, 0], [-math.sin(b), 0, math.cos(b)]])
    return np.stack([_bone(np.eye(3), pivot), _bone(rx, pivot), _bone(ry @ rx, pivot)])


def _ellipsoid(center, radii, tris):
    """UV ellipsoid with about `tris` triangles: positions, outward normals, indices."""
    lon = max(8, int(round(math.sqrt(tris))))
    lat = max(3, int(round(tris / (2 * lon))) + 1)
    th = np.linspace(0.0, math.pi, lat + 1)[1:-1]
    ph = np.linspace(0.0, 2.0 * math.pi, lon, endpoint=False)
    t, p = np.meshgrid(th, ph, indexing="ij")
    u = np.stack([np.sin(t) * np.cos(p), np.cos(t), np.sin(t) * np.sin(p)], -1).reshape(-1, 3)
    u = np.concatenate([[[0.0, 1.0, 0.0]], u, [[0.0, -1.0, 0.0]]])
    r = np.asarray(radii)
    nrm = u / r
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    i, k = np.meshgrid(np.arange(lat - 2), np.arange(lon), indexing="ij")
    a, b = 1 + i * lon + k, 1 + i * lon + (k + 1) % lon
    c, d = a + lon, b + lon
    k = np.arange(lon)
    last = len(u) - 1
    base = 1 + (lat - 2) * lon
    idx = np.concatenate([np.stack([0 * k, 1 + (k + 1) % lon, 1 + k], -1), np.stack([a, b, d], -1).reshape(-1, 3),
                          np.stack([a, d, c], -1).reshape(-1, 3),
                          np.stack([0 * k + last, base + k, base + (k + 1) % lon], -1)])
    return u * r + np.asarray(center), nrm, idx


def _mesh(center, tris, gen):
    """A head and a neck: {position, normal} rows, indices, {bone index, bone weight} rows."""
    v, nr, ix = _ellipsoid(center, (0.1, 0.11, 0.1), tris * 0.7)
    v2, nr2, ix2 = _ellipsoid((center[0], center[1] - 0.1, center[2] + 0.015), (0.06, 0.09, 0.07), tris * 0.3)
    v, nr, ix = np.concatenate([v, v2]), np.concatenate([nr, nr2]), np.concatenate([ix, ix2 + len(v)])
    v = v + 2e-4 * torch.randn(len(v), 3, generator=gen, device=gen.device).double().cpu().numpy()   # a sculpted surface, not an exact one
    out = np.zeros((len(v), 8), np.float32)
    out[:, :3], out[:, 3], out[:, 4:7] = v, 1.0, nr
    sk = np.zeros((len(v), 8), np.float32)
    w = np.clip((v[:, 1] - (center[1] - 0.18)) / 0.16, 0.0, 1.0)
    sk[:, 0], sk[:, 4] = 2.0, 1.0
    sk[-len(v2):, 0], sk[-len(v2):, 4], sk[-len(v2):, 5] = 1.0, np.maximum(w[-len(v2):], 1e-3), 1.0 - w[-len(v2):]
    return out, ix.astype(np.uint32).reshape(-1), sk


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _asset(o, center, gen):
    """Strands grown from the upper part of the head, follow hairs beside them, and a moving state."""
    from tressfx_gb300.synthetic import HairAsset
    G, n, F = o["guides"], o["n"], o["follow"]
    rnd = lambda *s: torch.randn(*s, generator=gen, device=gen.device, dtype=torch.float32)  # noqa: E731
    d = _unit(rnd(G, 3))
    d[:, 1] = torch.where(d[:, 1] < -0.2, -d[:, 1], d[:, 1])
    c = torch.tensor(center, device=gen.device, dtype=torch.float32)
    r = torch.tensor([0.1, 0.11, 0.1], device=gen.device)
    p = [d * r + c]
    down = torch.tensor([0.0, -1.0, 0.0], device=gen.device)
    for j in range(1, n):
        d = _unit(d + 0.26 * rnd(G, 3) + (0.1 * j / n) * down)
        p.append(p[-1] + (0.16 / n) * d)
    guide = torch.stack(p, 1)                                             # [G, n, 3]
    off = torch.zeros(G, F + 1, 4, device=gen.device)
    off[:, :, 3] = (torch.arange(G, device=gen.device) * (F + 1))[:, None]
    off[:, 1:, :3] = 0.002 * (2.0 * torch.rand(G, F, 3, generator=gen, device=gen.device) - 1.0)
    grow = 1.0 + torch.arange(n, device=gen.device) / n
    pos = torch.zeros(G, F + 1, n, 4, device=gen.device)
    pos[..., :3] = guide[:, None] + off[:, :, None, :3] * grow[None, None, :, None]
    pos[:, :, 2:, 3] = 1.0
    rest = torch.zeros(G, F + 1, n, device=gen.device)
    rest[:, :, :-1] = (pos[:, :, 1:, :3] - pos[:, :, :-1, :3]).norm(dim=-1)
    tan = torch.zeros_like(pos)
    tan[:, :, :-1, :3] = _unit(pos[:, :, 1:, :3] - pos[:, :, :-1, :3])
    tan[:, :, -1, :3] = tan[:, :, -2, :3]
    sk = torch.zeros(G, F + 1, 8, device=gen.device)
    sk[:, :, 0], sk[:, :, 1] = 2.0, 1.0
    sk[:, :, 4] = 0.5 + 0.5 * torch.rand(G, 1, generator=gen, device=gen.device)
    sk[:, :, 5] = 1.0 - sk[:, :, 4]
    sway = rnd(G, 1, 1, 3) * 0.003 * torch.arange(n, device=gen.device)[None, None, :, None] / n
    now, prev = pos.clone(), pos.clone()
    now[:, :, 2:, :3] += sway[:, :, 2:]
    prev[:, :, 2:, :3] += sway[:, :, 2:] * 0.5
    h = lambda t, w: t.reshape(-1, w).cpu().numpy()  # noqa: E731
    return (HairAsset(G, n, F, h(pos, 4), h(tan, 4), rest.reshape(-1).cpu().numpy(), h(off, 4), h(sk, 8)), h(now, 4), h(prev, 4))


def _grid_numbers(o, center):
    """(origin, cell, margin): the grid box around head and neck, margin half a cell."""
    ext = np.array([0.27, 0.36, 0.27])
    cell = np.float32(max(ext[k] / o["grid"][k] for k in range(3)))
    mid = np.array([center[0], center[1] - 0.04, center[2]])
    origin = (mid - 0.5 * np.array(o["grid"]) * float(cell)).astype(np.float32)
    return origin, cell, np.float32(0.5) * cell


def _objects(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    out = []
    for k, o in enumerate(_specs(case)):
        center = (0.9 * (k % 4) + 0.013, 1.6, 0.8 * (k // 4) - 0.007)
        phase = float(torch.rand(1, generator=gen, device=DEV))
        out.append((o, center, phase, _asset(o, center, gen), _mesh(center, o["tris"], gen) if o["tris"] else None))
    return out


# ------------------------------------------------------------------------------------------ the library side
class _Device:
    """Device memory of a library object as a torch tensor without a copy; the tensor keeps the object."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3)


def _view(owner, ptr, shape, typestr="<f4"):
    return torch.as_tensor(_Device(owner, ptr, shape, typestr), device="cuda")


class _State:
    pass


def _context():
    from tressfx_gb300.api import Context
    return Context(0)


def _grid_struct(o, center):
    from tressfx_gb300._capi import SdfGrid
    origin, cell, margin = _grid_numbers(o, center)
    g = SdfGrid()
    for k in range(3):
        g.origin[k] = float(origin[k])
    g.cell_size = float(cell)
    g.num_cells_x, g.num_cells_y, g.num_cells_z = o["grid"]
    return g, float(margin)


def prepare(case, seed):
    kind = case["kind"]
    return {"frame": _prepare_frame, "sdf": _prepare_sdf, "quads": _prepare_quads, "query": _prepare_query,
            "train": _prepare_train}[kind](case, seed)


def run(state):
    return state.go(state)


def _prepare_frame(case, seed):
    from tressfx_gb300 import _capi as A
    from tressfx_gb300 import api
    from tressfx_gb300.headless import settings_struct
    s = _State()
    s.ctx, s.tick, s.hair, s.mesh, s.sdf, s.grid, s.bones, s.params = _context(), 0, [], [], [], [], [], []
    s.settings, s.plain = [], api.Simulation()
    batch = s.batch = api.Batch(s.ctx) if case["path"] == "batch" else None
    s.out = []
    for k, (o, center, phase, (asset, now, prev), mesh) in enumerate(_objects(case, seed)):
        h = api.HairObject(s.ctx, asset)
        h.write(A.BUF_POSITIONS, now)
        h.write(A.BUF_POSITIONS_PREV, prev)
        h.frame = FRAME0
        for cb in h.sim_cb:
            cb.reset_positions = 0.0
        m = d = g = None
        if mesh is not None:
            m = api.CollisionMesh(s.ctx, *mesh)
            d = api.SDFCollision(s.ctx, int(np.prod(o["grid"])))
            d.bind_mesh(m)
            g = _grid_struct(o, center)
        if batch:
            si = batch.add_sdf(d, m, o["grid"]) if d else -1
            batch.add_hair(h, si)
        st = settings_struct(_settings(o))
        bones = [_pose(center, phase, t) for t in range(TICKS)]
        params = []
        for t in range(TICKS):
            p = A.SimParams()
            it = api.fill_sim_params(p, st, DT, o["n"], o["follow"], FRAME0 + t)
            p.bones_view()[:3] = bones[t]
            params.append((p, it))
        s.hair.append(h), s.mesh.append(m), s.sdf.append(d), s.grid.append(g), s.bones.append(bones), s.params.append(params)
        s.settings.append(st)
        for buf in (A.BUF_POSITIONS, A.BUF_POSITIONS_PREV, A.BUF_TANGENTS):
            s.out.append(_view(h, h.device_buffer(buf)[0], (h.num_vertices, 4)))
        if d:
            s.out.append(_view(d, _sdf_ptr(d), tuple(reversed(o["grid"]))))
    if batch:
        batch.build()
    s.ctx.synchronize()
    s.go = _run_batch if batch else _run_plain
    return s


def _sdf_ptr(d):
    from tressfx_gb300 import _capi as A
    p, n = C.c_void_p(), C.c_size_t()
    A.check(A.lib().tfx_sdf_get_buffer(d.handle, C.byref(p), C.byref(n)), "tfx_sdf_get_buffer")
    return p.value


def _run_batch(s):
    t, b = s.tick % TICKS, s.batch
    s.tick += 1
    for i in range(len(s.hair)):
        p, it = s.params[i][t]
        b.set_hair_constants(i, p, 3, it)
    si = 0
    for i, g in enumerate(s.grid):
        if g is not None:
            b.set_sdf_frame(si, g[0], g[1])
            b.set_mesh_bones(si, s.bones[i][t])
            si += 1
    b.run()
    return s.out


def _run_plain(s):
    t = s.tick % TICKS
    s.tick += 1
    for i, h in enumerate(s.hair):
        h.update_simulation_parameters(s.settings[i], DT)
        h.update_bone_matrices(s.bones[i][t])
        if s.mesh[i] is not None:
            s.mesh[i].skin(s.bones[i][t])
            s.sdf[i].update(s.grid[i][0])
    s.plain.simulate(s.hair)
    for i, h in enumerate(s.hair):
        if s.sdf[i] is not None:
            s.sdf[i].collide(h, *s.grid[i])
    return s.out


def _sdf_case(case):
    return dict(grid=(case["gx"], case["gy"], case["gz"]), tris=case["tris"])


def _prepare_sdf(case, seed):
    from tressfx_gb300 import api
    s = _State()
    s.ctx, s.tick = _context(), 0
    o, center = _sdf_case(case), (0.013, 1.6, -0.007)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    s.phase = float(torch.rand(1, generator=gen, device=DEV))
    s.mesh = api.CollisionMesh(s.ctx, *_mesh(center, o["tris"], gen))
    s.sdf = api.SDFCollision(s.ctx, int(np.prod(o["grid"])))
    s.sdf.bind_mesh(s.mesh)
    s.grid = _grid_struct(o, center)[0]
    s.bones = [_pose(center, s.phase, t) for t in range(TICKS)]
    s.out = [_view(s.sdf, _sdf_ptr(s.sdf), tuple(reversed(o["grid"])))]
    s.ctx.synchronize()
    s.go = _run_sdf
    return s


def _run_sdf(s):
    s.mesh.skin(s.bones[s.tick % TICKS])
    s.tick += 1
    s.sdf.update(s.grid)
    return s.out


_VIEW = dict(eye=(0.3, 1.7, 0.9), win=(1920.0, 1080.0),
             proj=(1.2, 0.05, -0.4, -0.2, 0.1, 1.9, -0.2, -3.0, 0.35, 0.1, 0.9, -0.5, 0.35, 0.1, 0.92, 0.9))
_STRAND = dict(base=(0.4, 0.25, 0.2, 1.0), tip=(0.6, 0.5, 0.4, 1.0), tip_percentage=0.3, ratio=0.5, radius=0.0021)


def _quads_object(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return _asset(dict(guides=case["guides"], n=case["n"], follow=case["follow"]), (0.013, 1.6, -0.007), gen)


def _prepare_quads(case, seed):
    from tressfx_gb300 import _capi as A
    from tressfx_gb300 import api
    s = _State()
    s.ctx = _context()
    asset, now, _ = _quads_object(case, seed)
    s.hair = api.HairObject(s.ctx, asset)
    s.hair.write(A.BUF_POSITIONS, now)
    p = s.params = A.StrandParams()
    p.mat_base_color[:], p.mat_tip_color[:] = _STRAND["base"], _STRAND["tip"]
    p.tip_percentage, p.fiber_ratio, p.fiber_radius = _STRAND["tip_percentage"], _STRAND["ratio"], _STRAND["radius"]
    p.num_vertices_per_strand, p.enable_thin_tip = case["n"], 1
    s.eye, s.win, s.proj = (C.c_float * 3)(*_VIEW["eye"]), (C.c_float * 2)(*_VIEW["win"]), (C.c_float * 16)(*_VIEW["proj"])
    s.shadow = case["shadow"]
    s.quads = torch.empty(2 * s.hair.num_vertices, 16, device="cuda")
    torch.cuda.synchronize()
    s.go = _run_quads
    return s


def _run_quads(s):
    from tressfx_gb300 import _capi as A
    A.check(A.lib().tfx_hair_expand_strands(s.hair.handle, C.byref(s.params), s.eye, s.win, s.proj, s.shadow, s.quads.data_ptr()),
            "tfx_hair_expand_strands")
    return s.quads


# the proxy's network: 102 inputs padded to 112, four hidden layers of 64, one output padded to 8
_IN, _PAD, _HID, _OUT = 102, 112, 64, 8
_BOX = ((-0.35, 1.15, -0.35), (0.35, 1.85, 0.35))
_CELL = 0.0021


def _proxy_weights(seed):
    gen = torch.Generator(device="cpu")
    gen.manual_seed(seed)

    def dense(rows, pad_rows, cols, used):
        w = torch.zeros(pad_rows, cols)
        w[:rows, :used] = (2.0 * torch.rand(rows, used, generator=gen) - 1.0) * math.sqrt(6.0 / rows)
        return w
    out = []
    for rows, pad in ((_IN, _PAD), (_HID, _HID), (_HID, _HID), (_HID, _HID)):
        out += [dense(rows, pad, _HID, _HID), 0.2 * (2.0 * torch.rand(_HID, generator=gen) - 1.0)]
    b = torch.zeros(_OUT)
    b[0] = 0.5
    return out + [dense(_HID, _HID, _OUT, 1), b]


def _proxy(s, samples):
    from tressfx_gb300 import api
    return api.NeuralSDF(s.ctx, *_BOX, _CELL, band_cells=3.0, seed=3, max_samples=max(samples, 1), max_eval_samples=1)


def _proxy_points(count, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    d = _unit(torch.randn(count, 3, generator=gen, device=DEV))
    r = 0.1 + 0.05 * torch.rand(count, 1, generator=gen, device=DEV)
    p = torch.zeros(count, 4, device=DEV)
    p[:, :3] = d * r + torch.tensor([0.0, 1.6, 0.0], device=DEV)
    pose = (torch.rand(3, generator=gen, device=DEV) - 0.5).tolist()
    return p, pose


def _prepare_query(case, seed):
    s = _State()
    s.ctx = _context()
    s.proxy = _proxy(s, 1)
    s.proxy.set_params(torch.cat([t.reshape(-1) for t in _proxy_weights(seed)]).numpy())
    s.points, s.pose = _proxy_points(case["points"], seed)
    s.dist = torch.empty(case["points"], device="cuda")
    torch.cuda.synchronize()
    s.go = _run_query
    return s


def _run_query(s):
    s.proxy.query_device(s.points.data_ptr(), len(s.points), s.pose, s.dist.data_ptr())
    return s.dist


def _prepare_train(case, seed):
    s = _State()
    s.ctx = _context()
    s.proxy = _proxy(s, case["samples"])
    s.proxy.set_params(torch.cat([t.reshape(-1) for t in _proxy_weights(seed)]).numpy())
    p, _ = _proxy_points(case["samples"], seed)
    rec = torch.zeros(case["samples"], 8, device=DEV)
    rec[:, :3] = p[:, :3]
    rec[:, 3] = (((p[:, :3] - torch.tensor([0.0, 1.6, 0.0], device=DEV)).norm(dim=1) - 0.12) / _CELL).clamp(-3.0, 3.0)
    rec[:, 4:7] = 0.1 * torch.sin(37.0 * p[:, :3])
    rec[:, 7] = 1.0
    s.proxy.set_samples(0, rec.cpu().numpy())
    s.steps, s.batch = case["steps"], case["batch"]
    s.ctx.synchronize()
    s.go = _run_train
    return s


def _run_train(s):
    loss = s.proxy.train(s.steps, s.batch, 2e-4)
    return {"loss": loss, "weights": s.proxy.params(), "gradients": s.proxy.gradients()}


# ------------------------------------------------------------------------------------------ work
def _sdf_work(o):
    cells = int(np.prod(o["grid"]))
    # vertices in (bind, skinning, skinned) once, indices once, the grid written once; about 150 cells a
    # triangle visits at 100 operations each
    return 96 * (o["tris"] / 2) + 12 * o["tris"] + 4 * cells, 150 * 100 * o["tris"]


def work(case):
    kind = case["kind"]
    if kind == "frame":
        b = f = 0.0
        for o in _specs(case):
            vg = o["guides"] * o["n"]
            # guides: positions, previous positions, rest pose, tangents, rest lengths in; positions, previous
            # twice and tangents out; the skinning record and strand-level data of a strand
            b += 132 * vg + 80 * o["guides"] + (36 * vg + 16 * o["guides"]) * o["follow"]
            f += vg * (150 + 110 * o["local"] + 40 * o["length"]) + 60 * vg * (1 + o["follow"])
            if o["tris"]:
                sb, sf = _sdf_work(o)
                b, f = b + sb + 4 * int(np.prod(o["grid"])), f + sf
        return {"bytes": b, "flops": f}
    if kind == "sdf":
        b, f = _sdf_work(_sdf_case(case))
        return {"bytes": b, "flops": f}
    if kind == "quads":
        v = case["guides"] * (case["follow"] + 1) * case["n"]
        return {"bytes": 160 * v, "flops": 200 * v}
    macs = _IN * _HID + 3 * _HID * _HID + _HID
    if kind == "query":
        return {"bytes": 20 * case["points"], "flops": 2 * macs * case["points"]}
    return {"bytes": 32 * case["batch"] * case["steps"], "flops": 6 * macs * case["batch"] * case["steps"]}


# ------------------------------------------------------------------------------------------ 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind == "frame":
        out = []
        for obj in _objects(case, seed):
            out += _exact_frame(*obj)
        return out
    if kind == "sdf":
        o, center = _sdf_case(case), (0.013, 1.6, -0.007)
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        phase = float(torch.rand(1, generator=gen, device=DEV))
        return [_exact_sdf(o, center, _mesh(center, o["tris"], gen), _pose(center, phase, 0))]
    if kind == "quads":
        return _exact_quads(case, seed)
    if kind == "query":
        return _exact_query(case, seed)
    return None   # which samples a training step takes is the library's own choice


def _t(a):
    return torch.as_tensor(np.asarray(a), device=DEV).double()


def _blend(bones, skin):
    w = skin[:, 4:8].clone()
    w[:, 1:] = w[:, 1:].clamp(min=0.0)
    m = sum(w[:, k, None, None] * bones[skin[:, k].long()] for k in range(4))
    return m / w.sum(1)[:, None, None]


def _xform(p, m, w=1.0):
    return torch.einsum("...i,...ij->...j", p, m[..., :3, :3]) + w * m[..., 3, :3]


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _exact_sdf(o, center, mesh, bones):
    verts, idx, skin = mesh
    origin, cell, _ = _grid_numbers(o, center)
    m = _blend(_t(bones).reshape(-1, 4, 4), _t(skin))
    v = _xform(_t(verts)[:, :3], m)
    tri = v[torch.as_tensor(idx.astype(np.int64), device=DEV)].reshape(-1, 3, 3)
    nx, ny, nz = o["grid"]
    dims = torch.tensor([nx, ny, nz], device=DEV)
    # the box of cells a triangle visits, in 32 bits
    t32, o32 = tri.float(), torch.as_tensor(origin, device=DEV)
    c32 = torch.tensor(float(cell), dtype=torch.float32, device=DEV)
    lo = ((t32.amin(1) - c32 - o32) / c32).to(torch.int64) - 1
    hi = ((t32.amax(1) + c32 - o32) / c32).to(torch.int64) + 1
    zero = torch.zeros_like(dims)
    lo, hi = torch.maximum(zero, torch.minimum(lo, dims - 1)), torch.maximum(zero, torch.minimum(hi, dims - 1))
    ext = hi - lo + 1
    vol = ext.prod(1)
    best = torch.full((nx * ny * nz,), float("inf"), dtype=torch.float64, device=DEV)
    neg = torch.ones(nx * ny * nz, dtype=torch.bool, device=DEV)
    h, org = float(cell), _t(origin)
    ends = vol.cumsum(0).cpu()
    first, parts = 0, []
    while first < len(tri):   # about 8M (triangle, cell) pairs at a time
        base = int(ends[first - 1]) if first else 0
        last = max(first + 1, int(torch.searchsorted(ends, base + (8 << 20))))
        n = vol[first:last]
        t = torch.repeat_interleave(torch.arange(first, last, device=DEV), n)
        k = torch.arange(len(t), device=DEV) - torch.repeat_interleave(n.cumsum(0) - n, n)
        e = ext[t]
        cc = lo[t] + torch.stack([k % e[:, 0], (k // e[:, 0]) % e[:, 1], k // (e[:, 0] * e[:, 1])], 1)
        d, s = _exact_tri(cc.double() * h + org, tri[t])
        lin = (cc[:, 2] * ny + cc[:, 1]) * nx + cc[:, 0]
        parts.append((lin, d, s))
        best.scatter_reduce_(0, lin, d, "amin")
        first = last
    for lin, d, s in parts:   # the sign of the nearest; on a tie the positive one wins
        at = (d <= best[lin]) & ~s
        neg[lin[at]] = False
    val = torch.where(neg, -best, best)
    return torch.where(torch.isinf(best), torch.full_like(best, 1e10), val).reshape(nz, ny, nx)


def _exact_tri(p, tri):
    """(|distance|, negative) of points to triangles, inside taken by the barycentric coordinates."""
    x0, x1, x2 = tri[:, 0], tri[:, 1], tri[:, 2]
    x02 = x0 - x2
    l0 = x02.norm(dim=1, keepdim=True) + 1e-30
    x02 = x02 / l0
    x12 = x1 - x2
    l1 = _dot(x12, x02)
    x12 = x12 - l1 * x02
    l2 = x12.norm(dim=1, keepdim=True) + 1e-30
    x12 = x12 / l2
    px2 = p - x2
    b = _dot(x12, px2) / l2
    a = (_dot(x02, px2) - l1 * b) / l0
    c = 1.0 - a - b
    face = (a >= -1e-8) & (b >= -1e-8) & (c >= -1e-8)
    d = (p - (a * x0 + b * x1 + c * x2)).norm(dim=1, keepdim=True)

    def edge(u, v):
        t = (_dot(v - p, v - u) / _dot(v - u, v - u)).clamp(0.0, 1.0)
        return (p - (t * u + (1.0 - t) * v)).norm(dim=1, keepdim=True)
    d = torch.where(face, d, torch.minimum(edge(x0, x1), torch.minimum(edge(x1, x2), edge(x0, x2))))
    side = _dot(p - x0, torch.linalg.cross(x1 - x0, x2 - x0))
    return d[:, 0], side[:, 0] < 0.0


def _quat_rot(q, v):
    u = q[..., :3]
    uv = torch.linalg.cross(u.expand_as(v), v)
    return v + uv * (2.0 * q[..., 3:]) + 2.0 * torch.linalg.cross(u.expand_as(v), uv)


def _quat_between(u, v):
    r = 1.0 + _dot(u, v)
    flip = r < 1e-7
    z = torch.zeros_like(r)
    other = torch.where(u[..., :1].abs() > u[..., 2:].abs(), torch.cat([-u[..., 1:2], u[..., :1], z], -1),
                        torch.cat([z, -u[..., 2:], u[..., 1:2]], -1))
    q = torch.cat([torch.where(flip, other, torch.linalg.cross(u, v)), torch.where(flip, z, r)], -1)
    return q / q.norm(dim=-1, keepdim=True)


def _quat_of(m):
    """Rotation quaternion of nearly orthonormal blends with a positive trace (small poses)."""
    r = torch.sqrt(m[:, 0, 0] + m[:, 1, 1] + m[:, 2, 2] + 1.0)
    w, r = 0.5 * r, 0.5 / r
    return torch.stack([(m[:, 1, 2] - m[:, 2, 1]) * r, (m[:, 2, 0] - m[:, 0, 2]) * r, (m[:, 0, 1] - m[:, 1, 0]) * r, w], 1)


def _exact_lookup(sdf, origin, cell, p):
    """Trilinear distance; 1e10 outside the grid or beside a cell that was never set."""
    nz, ny, nx = sdf.shape
    g = ((p - origin) / cell)
    i = g.to(torch.int64)
    ok = ((i >= 0) & (i < torch.tensor([nx - 2, ny - 2, nz - 2], device=p.device))).all(1)
    i = torch.where(ok[:, None], i, torch.zeros_like(i))
    f = (p - (i.double() * cell + origin)) / cell
    acc, unset = torch.zeros(len(p), dtype=torch.float64, device=p.device), torch.zeros(len(p), dtype=torch.bool, device=p.device)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                v = sdf[i[:, 2] + dz, i[:, 1] + dy, i[:, 0] + dx]
                unset |= v == 1e10
                w = (f[:, 0] if dx else 1 - f[:, 0]) * (f[:, 1] if dy else 1 - f[:, 1]) * (f[:, 2] if dz else 1 - f[:, 2])
                acc += w * v
    return torch.where(ok & ~unset, acc, torch.full_like(acc, 1e10))


def _exact_frame(o, center, phase, hair, mesh):
    asset, now, prev = hair
    G, n, F = o["guides"], o["n"], o["follow"]
    bones = _pose(center, phase, 0)
    f32 = lambda x: float(np.float32(x))  # noqa: E731
    dt, damping, kg, rng = f32(DT), f32(o["damping"]), f32(o["glob"]), f32(0.3)
    shape = lambda a, w: _t(a).reshape(G, F + 1, n, w)  # noqa: E731
    pos, old, tan, init = shape(now, 4), shape(prev, 4), shape(asset.tangents, 4), shape(asset.positions, 4)
    rest = _t(asset.rest_lengths).reshape(G, F + 1, n)[:, 0]
    w = pos[:, 0, :, 3:]
    free = w > 0
    m = _blend(_t(bones).reshape(-1, 4, 4), _t(asset.bone_skinning).reshape(G, F + 1, 8)[:, 0])
    target = _xform(init[:, 0, :, :3], m[:, None])
    cur, last = pos[:, 0, :, :3], old[:, 0, :, :3]
    fall = torch.tensor([0.0, -f32(9.8), 0.0], dtype=torch.float64, device=DEV)
    p = torch.where(free, cur + math.exp(-damping * dt * 60.0) * (cur - last) + fall * dt * dt, target)
    pull = free & (torch.arange(n, device=DEV)[None, :, None] < rng * n)
    p = torch.where(pull, p + kg * (target - p), p)
    was = cur.clone()
    # strand-level rotation and velocity shock propagation
    q = _quat_between(_unit(was[:, 1] - was[:, 0]), _unit(p[:, 1] - p[:, 0]))
    move = p[:, 0] - _quat_rot(q, was[:, 0])
    acc = torch.cat([p[:, 1] - 2.0 * was[:, 1] + last[:, 1], (w[:, 1] - 2.0 * w[:, 1] + old[:, 0, 1, 3:])], 1).norm(dim=1)
    k = torch.where(acc > f32(1.2), 1.0, f32(0.7))[:, None, None]
    for a in (p, was):
        a[:, 2:] = (1.0 - k) * a[:, 2:] + k * (_quat_rot(q[:, None], a[:, 2:]) + move[:, None])
    # local shape: sweeps from root to tip
    bind = _quat_rot(_quat_of(m)[:, None], init[:, 0, :, :3])
    stiff = 0.5 * min(f32(o["stiff"]), f32(0.95))
    sweeps = 1 if n >= 64 else o["local"]
    for _ in range(sweeps):
        for j in range(1, n - 1):
            r = _quat_between(_unit(bind[:, j] - bind[:, j - 1]), _unit(p[:, j] - p[:, j - 1]))
            d = stiff * (_quat_rot(r, bind[:, j + 1] - bind[:, j]) + p[:, j] - p[:, j + 1])
            p[:, j] = torch.where(free[:, j], p[:, j] - d, p[:, j])
            p[:, j + 1] = torch.where(free[:, j + 1], p[:, j + 1] + d, p[:, j + 1])
    if o["wind"] != 0.0:
        mag = o["wind"] * (math.sin(FRAME0 * 0.01) ** 2 + 0.5)
        ca, sa = math.cos(math.radians(40.0)) * mag, math.sin(math.radians(40.0)) * mag
        corner = torch.tensor([[ca, 0, -sa], [ca, 0, sa], [ca, sa, 0], [ca, -sa, 0]], dtype=torch.float64, device=DEV)
        a = ((torch.arange(G, device=DEV) * (F + 1)) % 20).double()[:, None] / 20.0
        wind = (a * corner[0] + (1 - a) * corner[1] + a * corner[2] + (1 - a) * corner[3])[:, None]
        v = p[:, 2:-1] - p[:, 3:]
        wind = wind.expand_as(v)
        p[:, 2:-1] -= torch.linalg.cross(torch.linalg.cross(v, wind), v) * dt * dt
    for _ in range(o["length"]):
        for s0 in (0, 1):   # edges (0,1) (2,3) .., then (1,2) (3,4) ..
            i = torch.arange(s0, n - 1, 2, device=DEV)
            d = p[:, i + 1] - p[:, i]
            d = (1.0 - rest[:, i, None] / d.norm(dim=-1, keepdim=True).clamp(min=1e-7)) * d
            a, b = free[:, i], free[:, i + 1]
            p[:, i] += torch.where(a & b, 0.5, torch.where(a, 1.0, 0.0)) * d
            p[:, i + 1] -= torch.where(a & b, 0.5, torch.where(b, 1.0, 0.0)) * d
    t = torch.cat([p[:, 1:] - p[:, :-1], p[:, -1:] - p[:, -2:-1]], 1)
    t = _unit(t)
    step = p - was
    sq = _dot(step, step)
    was = torch.where(sq > 400.0, p - step * (400.0 / sq), was)
    pos, old, tan = pos.clone(), old.clone(), tan.clone()
    pos[:, 0, :, :3], old[:, 0, :, :3], tan[:, 0, :, :3] = p, was, t
    grow = 1.0 + torch.arange(n, device=DEV).double() / n
    off = _t(asset.follow_root_offsets).reshape(G, F + 1, 1, 4)[..., :3]
    pos[:, 1:, :, :3] = p[:, None] + off[:, 1:] * grow[:, None]
    tan[:, 1:] = tan[:, :1]
    out = []
    if mesh is not None:
        sdf = _exact_sdf(o, center, mesh, bones)
        origin, cell, margin = (_t(x) for x in _grid_numbers(o, center))
        x = pos[:, :, 2:, :3].reshape(-1, 3)
        d = _exact_lookup(sdf, origin, cell, x)
        near = (d < margin).nonzero()[:, 0]
        if len(near):
            y, dn, h = x[near], d[near, None], 0.1 * cell
            g = torch.cat([(_exact_lookup(sdf, origin, cell, y + h * torch.eye(3, dtype=torch.float64, device=DEV)[a])[:, None] - dn) / h
                           for a in range(3)], 1)
            x = x.clone()
            x[near] = y + _unit(g) * (margin - dn)
            hit = torch.zeros(len(x), 1, dtype=torch.bool, device=DEV)
            hit[near] = True
            pos[:, :, 2:, :3] = x.reshape(G, F + 1, n - 2, 3)
            old[:, :, 2:, :3] = torch.where(hit.reshape(G, F + 1, n - 2, 1), pos[:, :, 2:, :3], old[:, :, 2:, :3])
        out = [sdf]
    return [a.reshape(-1, 4) for a in (pos, old, tan)] + out


def _exact_quads(case, seed):
    asset, now, _ = _quads_object(case, seed)
    n, v, t = case["n"], _t(now)[:, :3], _t(asset.tangents)[:, :3]
    f32 = lambda x: float(np.float32(x))  # noqa: E731
    frac = (torch.arange(len(v), device=DEV) % n).double()[:, None] / (n - 1)
    ratio = 1.0 + frac * (f32(_STRAND["ratio"]) - 1.0)
    right = _unit(torch.linalg.cross(t, _unit(v - _t(np.float32(_VIEW["eye"])))))
    proj = _t(np.float32(_VIEW["proj"])).reshape(4, 4)
    mv = lambda a, w: a @ proj[:, :3].T + w * proj[:, 3]  # noqa: E731
    side = _unit(mv(right, 0.0)[:, :2])
    reach = right * ratio * f32(_STRAND["radius"])
    e0, e1 = mv(v - reach, 1.0), mv(v + reach, 1.0)
    px = side * (1.0 if case["shadow"] else f32(0.71)) / f32(_VIEW["win"][1])
    out = torch.zeros(len(v), 2, 16, dtype=torch.float64, device=DEV)
    out[:, 0, :4], out[:, 1, :4] = e1, e0
    out[:, 0, :2] += px * e1[:, 3:]
    out[:, 1, :2] -= px * e0[:, 3:]
    if not case["shadow"]:
        out[:, :, 4:7] = t[:, None]
        out[:, 0, 7] = 1.0
        ndc = torch.cat([e0[:, :2] / e0[:, 3:].clamp(min=1e-7), e1[:, :2] / e1[:, 3:].clamp(min=1e-7)], 1)
        out[:, :, 8:12] = ndc[:, None]
        root, tip = _t(np.float32(_STRAND["base"]))[:3], _t(np.float32(_STRAND["tip"]))[:3]
        out[:, :, 12:15] = torch.where(frac > 1.0 - f32(_STRAND["tip_percentage"]), root + frac * (tip - root), root)[:, None]
        out[:, :, 15] = frac
    return out.reshape(-1, 16)


def _exact_query(case, seed):
    p, pose = _proxy_points(case["points"], seed)
    lo, hi = _t(np.float32(_BOX[0])), _t(np.float32(_BOX[1]))
    u = (p[:, :3].double() - 0.5 * (lo + hi)) / (0.5 * (hi - lo))
    a = torch.tensor(pose, dtype=torch.float64, device=DEV) / 0.7
    f = torch.pow(2.0, torch.arange(16, dtype=torch.float64, device=DEV) / 3.0)
    ang = math.pi * u[:, None, :] * f[None, :, None]
    x = torch.cat([u, a.expand(len(u), 3), torch.stack([torch.sin(ang), torch.cos(ang)], -1).reshape(len(u), -1)], 1)
    w = [t.double().to(DEV) for t in _proxy_weights(seed)]
    w[0] = w[0][:_IN]
    for k in range(4):
        z = x @ w[2 * k] + w[2 * k + 1]
        x = z * torch.sigmoid(z)
    return (x @ w[8][:, 0] + w[9][0]) * float(np.float32(_CELL))
