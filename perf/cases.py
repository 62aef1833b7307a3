"""Performance cases of the GI library: what a renderer or a serving program has it do for one frame, through the public
host objects (rtgi.gpu, rtgi.batch), over the sizes, formats and options the library takes.

A case is a dict of plain values.  ``prepare`` builds what such a program holds before the frame (the scene on the
device, the voxel world, the cascades, the G-buffer, a captured graph where it replays one), ``run`` is one frame.

Kinds:
  solve    gi_solve over a given G-buffer: the voxel rebuild and the cascades (screen or world probes), call by call
  frame    a whole frame replayed from one CUDA graph: moved objects posed, G-buffer drawn, solve, irradiance copied
  objects  a frame with a dynamic layer, called one by one: pose, G-buffer, sun shadow map, layer, multi-bounce, solve
  batch    several uneven solves in one graph (capture_passes, or parallel chains)
  rebuild  the voxel rebuild into the caller's own device memory (gi_vox_build_noalloc)
"""
import ctypes
import dataclasses
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "real-time-gi-lab_b200"))
from rtgi import _lib, batch, configs, frame as fr, gpu, movers, scenes  # noqa: E402

_SHARED = {}


def _ctx():
    if "ctx" not in _SHARED:
        _SHARED["ctx"] = gpu.Context(0)
        _SHARED["stream"] = torch.cuda.Stream()   # a program's render stream (graphs need one that is not the default)
    return _SHARED["ctx"]


def _stream():
    _ctx()
    return _SHARED["stream"]


# Clipmaps by name: v0, levels, G, maxBricks, maxVoxels, as the repository's benchmark, tests and runner use them
_CLIPMAPS = {
    "small": {"v0": 0.16, "levels": 1, "G": 8, "maxBricks": 512, "maxVoxels": 1 << 18},
    "room": {"v0": 0.08, "levels": 3, "G": 16, "maxBricks": 8192, "maxVoxels": 1 << 20},
    "leak": {"v0": 0.1, "levels": 5, "G": 64, "maxBricks": 32768, "maxVoxels": 1 << 22},
    "large": {"v0": 0.1, "levels": 4, "G": 16, "maxBricks": 16384, "maxVoxels": 1 << 22},
    "default": {"v0": 0.2, "levels": 5, "G": 32, "maxBricks": 4608, "maxVoxels": 524288},
    "pool": {"v0": 0.2, "levels": 4, "G": 16, "maxBricks": 4096, "maxVoxels": 524288},
}
_SCENE_TRIS = {"room": 2414, "leak": 1212, "colonnade": 261784, "textured": 742}


def listed():
    return [
        # The smallest call: the benchmark's small room at 256 x 256, two cascades, under sun and sky.  Launches and
        # latency are all of it.
        {"name": "room-256", "kind": "solve", "scene": "room", "clipmap": "small", "config": "screen-8-voxel-f32-dda64",
         "cascades": 2, "width": 256, "height": 256, "shadow": 0, "bounce": False},
        # A small viewport of the reference's leak room with its recorded clipmap (5 levels of 512^3), bf16 atlas, an
        # odd size, the sun's shadow map: a big empty clipmap around little geometry.
        {"name": "leak-641x361", "kind": "solve", "scene": "leak", "clipmap": "leak", "config": "screen-8-voxel-bf16",
         "cascades": 5, "width": 641, "height": 361, "shadow": 1024, "bounce": False},
        # The headline workload: the colonnade at 1920 x 1080, f32 atlas, irradiance stored as the reference stores it.
        {"name": "colonnade-1080p", "kind": "solve", "scene": "colonnade", "clipmap": "large",
         "config": "screen-8-voxel-f32-dda256-irr16", "cascades": 5, "width": 1920, "height": 1080, "shadow": 4096,
         "bounce": False},
        # The same world for a viewer that replays whole frames (raster included) from one graph, f16 atlas.
        {"name": "frame-colonnade-1080p", "kind": "frame", "scene": "colonnade", "clipmap": "large",
         "config": "screen-8-voxel-f16-dda256", "cascades": 5, "width": 1920, "height": 1080, "objects": 16},
        # A served request: a small scene with many moving boxes, posed and replayed.
        {"name": "frame-served-640x360", "kind": "frame", "scene": "mixed", "tris": 25000, "clipmap": "room",
         "config": "screen-8-voxel-f16-dda256", "cascades": 4, "width": 640, "height": 360, "objects": 80},
        # Ragged: probe tiles of 12 pixels, an odd size, textures with alpha-masked panels, f32 outputs of an f16 atlas.
        {"name": "textured-1001x563", "kind": "solve", "scene": "textured", "clipmap": "room",
         "config": "screen-12-voxel-f16-f32out", "cascades": 5, "width": 1001, "height": 563, "shadow": 2048,
         "bounce": False},
        # World probes with voxel relocation, the benchmark's world configuration at 1920 x 1080.
        {"name": "world-1080p", "kind": "solve", "scene": "colonnade", "clipmap": "large",
         "config": "world-48-voxel-rc2-vrel-f32-dda256", "cascades": 5, "width": 1920, "height": 1080, "shadow": 4096,
         "bounce": False},
        # The reference renderer's default transport in a room: world probes, G-buffer relocation, multi-bounce, f16.
        {"name": "world-bounce-720p", "kind": "solve", "scene": "room", "clipmap": "default", "config": "world-24-voxel-rc2",
         "cascades": 5, "width": 1280, "height": 720, "shadow": 2048, "bounce": True},
        # Screen probes with multi-bounce at the runner's default clipmap.
        {"name": "bounce-900p", "kind": "solve", "scene": "mixed", "tris": 120000, "clipmap": "default",
         "config": "screen-8-voxel-f16", "cascades": 5, "width": 1600, "height": 900, "shadow": 4096, "bounce": True},
        # Moving objects through the dynamic layer, receiving and blocking the bounce (token obj), every pass called.
        {"name": "objects-720p", "kind": "objects", "scene": "colonnade", "clipmap": "large",
         "config": "screen-8-voxel-f16-dda256-obj", "cascades": 5, "width": 1280, "height": 720, "shadow": 2048,
         "objects": 64},
        # The largest: eight uneven solves of the batch distribution, one launch per pass.
        {"name": "batch-8", "kind": "batch", "first": 0, "count": 8, "atlas": "f32", "passes": True},
        # The rebuild alone in the caller's memory, at the upper end of the triangles its fixed big-triangle lists hold.
        {"name": "rebuild-200k", "kind": "rebuild", "scene": "mixed", "tris": 200000, "clipmap": "pool"},
    ]


def draw(rng):
    logu = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind = rng.choice(["solve", "solve", "solve", "frame", "objects", "batch", "rebuild"])
    if kind == "batch":
        return {"kind": "batch", "first": rng.randrange(8, 200), "count": rng.randrange(2, 6),
                "atlas": rng.choice(["f32", "f16", "bf16"]), "passes": rng.random() < 0.7}
    if kind == "rebuild":
        return {"kind": "rebuild", "scene": "mixed", "tris": logu(5000, 200000), "clipmap": "pool"}
    W = logu(200, 1900)
    c = {"kind": kind, "width": W, "height": max(64, int(W * rng.uniform(0.5, 0.62))), "cascades": rng.randrange(2, 6)}
    atlas = rng.choice(["f32", "f16", "f16", "bf16"]) + rng.choice(["", "", "-irr16", "-f32out"])
    P = rng.choice([8, 8, 8, 12, 16, 32])
    if kind == "solve":
        c["scene"] = rng.choice(["room", "leak", "colonnade", "mixed", "textured"])
        c["clipmap"] = rng.choice(["small", "room", "large", "default"])
        if rng.random() < 0.35:
            c["config"] = f"world-{rng.choice([24, 32, 48])}-voxel-rc2{rng.choice(['', '-vrel', '-norel'])}-{atlas}"
        else:
            c["config"] = f"screen-{P}-voxel-{atlas}-dda{rng.choice([64, 256, 1024])}"
        c["shadow"] = rng.choice([0, 1024, 2048, 4096])
        c["bounce"] = rng.random() < 0.4
    else:
        c["scene"] = rng.choice(["room", "colonnade", "mixed"])
        c["clipmap"] = rng.choice(["room", "large"])
        c["config"] = f"screen-{P}-voxel-{atlas}-dda256" + ("-obj" if kind == "objects" else "")
        c["objects"] = logu(1, 200)
        if kind == "objects":
            c["shadow"] = rng.choice([1024, 2048])
    if c["scene"] == "mixed":
        c["tris"] = logu(5000, 300000)
    return c


def _scene(case, seed):
    """The case's scene and camera: geometry, lamps and colours from the seeded generators, the camera moved a little."""
    rng = random.Random(seed)
    name = case["scene"]
    if name == "room":
        s = scenes.room_scene(seed & 0xffff)
        eye, at = s.camera.eye, s.camera.target
    elif name == "leak":
        s = scenes.leak_room(rng.uniform(0.08, 0.3))
        eye, at = s.camera.eye, s.camera.target
    elif name == "textured":
        s = scenes.textured_scene()
        s = dataclasses.replace(s, textures=np.roll(s.textures, rng.randrange(1, 60), axis=2))
        eye, at = s.camera.eye, s.camera.target
    elif name == "colonnade":
        s = scenes.colonnade_scene(seed & 0xffff)
        x, z = 2.5 * rng.randrange(-4, 5), 2.5 * rng.randrange(-2, 3)   # an aisle between four columns
        eye, at = (x, 1.7, z), (x + rng.uniform(15, 25), rng.uniform(1.0, 2.0), z + rng.uniform(-6, 6))
    else:
        s = scenes.mixed_scene(seed & 0xffff, case["tris"])
        eye, at = s.camera.eye, s.camera.target
    eye = tuple(float(c) + rng.uniform(-0.15, 0.15) for c in eye)
    cam = dataclasses.replace(s.camera, eye=eye, target=tuple(float(c) for c in at))
    sun = tuple(float(a) + rng.uniform(-0.1, 0.1) for a in s.sun_dir)
    return dataclasses.replace(s, camera=cam, sun_dir=sun, sun_e=fr.SUN_E, sky=fr.SKY)


def _frame(case, s, p):
    lvp, bias = [0.0] * 16, (0.0, 0.0)
    if case.get("shadow"):
        bmin, bmax = fr.scene_bounds(s.positions)
        lvp, bias = fr.scene_sun_view_proj(bmin, bmax, s.sun_dir), fr.SHADOW_BIAS
    return fr.pack_frame(fr.FrameParams(cam=s.camera, width=case["width"], height=case["height"], sun_dir=s.sun_dir,
                                        sun_e=s.sun_e, sky=s.sky, cascades=p.cascades, P=p.P, s_min=p.sMin, lift=p.lift,
                                        light_view_proj=lvp, shadow_bias=bias))


class _State:
    """Device handles of one prepared case, freed with it."""

    def __init__(self, case):
        self.case, self.own, self.n = case, [], 0

    def hold(self, h):
        self.own.append(h)
        return h

    def __del__(self, sync=torch.cuda.synchronize):
        sync()
        for h in reversed(self.own):
            h.destroy()


def _irradiance(rc):
    wide = rc.irr_bytes() == rc.width * rc.height * 16
    return torch.zeros((rc.height, rc.width, 4), dtype=torch.float32 if wide else torch.float16, device="cuda")


def _with_objects(case, seed):
    base = _scene(case, seed)
    area = (base.camera.eye[0], base.camera.eye[2], 4.0, 4.0) if case["scene"] == "room" else (0.0, 0.0, 12.0, 12.0)
    s, objs = movers.with_moving_boxes(base, case["objects"], scenes.PCG32(seed & 0xffff, stream=9), area=area)
    poses = [torch.from_numpy(objs.transforms(0.4 * k + 0.1 * (seed % 7))).contiguous().pin_memory() for k in range(4)]
    return base, s, objs, poses


def prepare(case, seed):
    ctx, st = _ctx(), _stream()
    S = _State(case)
    kind = case["kind"]
    if kind == "batch":
        S.solves, S.out = [], []
        for i in range(case["count"]):
            spec = scenes.batch_spec(case["first"] + i)
            scene = scenes.mixed_scene((seed * 31 + i) & 0xffff, spec["tris"])
            x = S.hold(batch.make_solve(ctx, spec, case["atlas"], st, scene))
            S.solves.append(x)
            S.out.append(_irradiance(x.rc))
        b = S.hold(gpu.Batch(ctx, [x.rc for x in S.solves], [x.vox for x in S.solves]))
        if case["passes"]:
            b.capture_passes(st)
        else:
            b.capture(st)
        S.batch = b
        return S
    v = configs.vox_params(_CLIPMAPS[case["clipmap"]])
    if kind == "rebuild":
        s = _scene(case, seed)
        dev = torch.device("cuda", 0)
        S.pos, S.nrm = (torch.zeros((a.shape[0], 4), dtype=torch.float32, device=dev) for a in (s.positions, s.normals))
        S.pos[:, :3] = torch.from_numpy(s.positions).to(dev)
        S.nrm[:, :3] = torch.from_numpy(s.normals).to(dev)
        S.tri = torch.from_numpy(np.ascontiguousarray(s.tri, np.uint32).view(np.int32)).to(dev)
        S.mats = torch.from_numpy(s.material_array().view(np.uint8)).to(dev)
        S.nmats = len(s.materials)
        words = {"hdr": 64, "ptr": v.levels * v.G ** 3, "occ": v.maxBricks * 16, "base": v.maxBricks, "code": v.maxBricks,
                 "attr": v.maxVoxels * 4}
        S.out = {k: torch.zeros(n, dtype=torch.int32, device=dev) for k, n in words.items()}
        S.out.update({k: torch.zeros(v.maxVoxels, dtype=torch.float32, device=dev) for k in ("plane", "sunvis")})
        S.params = _lib.GiVoxParams(float(v.v0), v.levels, v.G, v.maxBricks, v.maxVoxels, v.dynBricks, 0)
        S.eye = (ctypes.c_double * 3)(*[float(c) for c in s.camera.eye])
        torch.cuda.synchronize()
        return S
    p = configs.parse_config(case["config"], {"cascades": case["cascades"]})
    if kind == "solve":
        s = _scene(case, seed)
        sg = S.hold(gpu.SceneGpu(ctx, s))
    else:
        base, s, objs, S.poses = _with_objects(case, seed)
        sg = S.hold(gpu.SceneGpu(ctx, s))
        sg.rigid_define(objs.first, objs.per, objs.centres.shape[0])
        if kind == "objects":
            sg.set_static_count(base.triangle_count)
    vw = S.hold(gpu.VoxWorld(sg, v))
    if kind == "objects":
        dyn = S.hold(gpu.DynLayer(vw, base.triangle_count, bricks=2048, albedo=True))
    rc = S.hold(gpu.Rc(ctx, p, case["width"], case["height"]))
    S.sg, S.vw, S.rc, S.eye, S.frame, S.out = sg, vw, rc, s.camera.eye, _frame(case, s, p), _irradiance(rc)
    rc.set_frame(S.frame, st)
    vw.update(S.eye)
    if kind == "frame":
        sg.rigid_upload(S.poses[0].data_ptr(), st)
        rc.graph_capture_frame(vw, sg, S.out.data_ptr(), st)
    elif kind == "objects":
        rc.set_dyn(dyn)
        rc.set_bounce(vw)
    else:
        rc.render_gbuffer(sg, st)
        if case["shadow"]:
            rc.render_shadow(sg, case["shadow"], st)
        if case["bounce"]:
            rc.set_bounce(vw)
    torch.cuda.synchronize()
    return S


def run(S):
    st, case = _SHARED["stream"], S.case
    kind = case["kind"]
    S.n += 1
    if kind == "batch":
        S.batch.launch(st)
        for x, o in zip(S.solves, S.out):
            x.rc.read_irradiance_async(o.data_ptr(), st)
        return S.out
    if kind == "rebuild":
        o = S.out
        _lib.call("gi_vox_build_noalloc", ctypes.byref(S.params), S.eye, S.pos.data_ptr(), S.nrm.data_ptr(), S.pos.shape[0],
                  S.tri.data_ptr(), S.tri.shape[0], S.mats.data_ptr(), S.nmats, o["hdr"].data_ptr(), o["ptr"].data_ptr(),
                  o["occ"].data_ptr(), o["base"].data_ptr(), o["code"].data_ptr(), o["attr"].data_ptr(),
                  o["plane"].data_ptr(), o["sunvis"].data_ptr(), int(st.cuda_stream))
        return o
    if kind == "frame":
        S.sg.rigid_upload(S.poses[S.n % len(S.poses)].data_ptr(), st)
        S.rc.graph_launch(st)
        return S.out
    S.rc.set_frame(S.frame, st)
    S.vw.update(S.eye)
    if kind == "objects":
        S.sg.rigid_upload(S.poses[S.n % len(S.poses)].data_ptr(), st)
        S.sg.rigid_apply(st)
        S.rc.render_gbuffer(S.sg, st)
        S.rc.render_shadow(S.sg, case["shadow"], st)
    S.rc.solve(S.vw, st)
    S.rc.read_irradiance_async(S.out.data_ptr(), st)
    return S.out


def _screen(P, cascades, W, H):
    """Probes and rays of the screen cascades."""
    probes = [(-(-W // (P << c))) * (-(-H // (P << c))) for c in range(cascades)]
    return sum(probes), sum(n * (4 << c) ** 2 for c, n in enumerate(probes))


def work(case):
    """The scene read once, the G-buffer (10 bytes a pixel) read once, or written once where the frame draws it, the
    irradiance written once; the operations of a ray's set-up and six cells, a pixel's four probes, a triangle's tests."""
    if case["kind"] == "batch":
        parts = []
        for i in range(case["count"]):
            sp = scenes.batch_spec(case["first"] + i)
            parts.append((sp["tris"], sp["width"], sp["height"], sp["cascades"], 8, 16 if case["atlas"] == "f32" else 8))
    else:
        tris = case.get("tris") or _SCENE_TRIS[case["scene"]]
        tris += 12 * case.get("objects", 0)
        if case["kind"] == "rebuild":
            return {"bytes": tris * (16 + 18) + 6.0e6, "flops": tris * 400.0}
        p = configs.parse_config(case["config"], {"cascades": case["cascades"]})
        wide = (p.atlas == "f32" or p.f32Out) and not p.irr16
        parts = [(tris, case["width"], case["height"], case["cascades"], min(p.P, 16), 16 if wide else 8)]
    out = {"bytes": 0.0, "flops": 0.0}
    for tris, W, H, cascades, P, irr in parts:
        probes, rays = _screen(P, cascades, W, H)
        out["bytes"] += tris * (16 + 18) + W * H * (10 + irr)
        out["flops"] += tris * 400.0 + rays * 300.0 + W * H * 250.0
    return out


def exact(case, seed):
    """The irradiance of the one-level room in 64 bits, from the scene and camera alone.  The other cases have no such
    value: several levels, dropped bricks, histories and quantised voxel records make their result a property of the
    32-bit decisions, and a 64-bit walk over their scenes takes far over 20 seconds."""
    if case["kind"] != "solve" or case["scene"] != "room" or case["clipmap"] != "small" or case["shadow"] or case["bounce"]:
        return None
    if not case["config"].startswith("screen") or case["width"] * case["height"] > 400000:
        return None
    p = configs.parse_config(case["config"], {"cascades": case["cascades"]})
    return _exact_room(_scene(case, seed), _CLIPMAPS["small"], p, case["width"], case["height"])


def _hits(o, d, V, chunk=1 << 24):
    """Nearest triangle along o + t d (t > 0.05 along the unit forward axis is the caller's scaling): t, index."""
    a, e1, e2 = V[:, 0], V[:, 1] - V[:, 0], V[:, 2] - V[:, 0]
    best, idx = [], []
    step = max(1, chunk // V.shape[0])
    for k in range(0, d.shape[0], step):
        dd = d[k:k + step, None, :]
        pv = torch.linalg.cross(dd, e2[None].expand(dd.shape[0], -1, -1))
        det = (pv * e1).sum(-1)
        tv = (o - a)[None]
        u = (tv * pv).sum(-1) / det
        qv = torch.linalg.cross(tv, e1[None])
        w = (dd * qv).sum(-1) / det
        t = (qv * e2).sum(-1) / det
        t = torch.where((u >= 0) & (w >= 0) & (u + w <= 1) & (t > 0.05), t, torch.full_like(t, math.inf))
        t, i = t.min(-1)
        best.append(t)
        idx.append(i)
    return torch.cat(best), torch.cat(idx)


def _exact_room(s, clip, p, W, H):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    T = lambda x: torch.as_tensor(np.asarray(x, np.float64), device=dev)  # noqa: E731
    pos, tri = T(s.positions), torch.as_tensor(s.tri.astype(np.int64), device=dev)
    V, nrm = pos[tri[:, :3]], T(s.normals)[tri[:, 0]]          # flat faces: one normal a triangle
    albedo = (torch.floor(T([m.base_color[:3] for m in s.materials]) * 255 + 0.5) / 255)[tri[:, 3]]
    emit = T([m.emissive for m in s.materials])[tri[:, 3]]
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)  # noqa: E731
    eye, sun, sky, sun_e = T(s.camera.eye), unit(T(s.sun_dir)), T(s.sky), T(s.sun_e)
    # the G-buffer: a primary ray per pixel centre
    fwd = unit(T(s.camera.target) - eye)
    right = unit(torch.linalg.cross(fwd, T([0.0, 1.0, 0.0])))
    up = torch.linalg.cross(right, fwd)
    th = math.tan(s.camera.fov_y_deg * math.pi / 360)
    px, py = torch.arange(W, device=dev, dtype=torch.float64), torch.arange(H, device=dev, dtype=torch.float64)
    gx, gy = ((px + 0.5) / W * 2 - 1) * th * W / H, (1 - (py + 0.5) / H * 2) * th
    d = (fwd + gx[None, :, None] * right + gy[:, None, None] * up).reshape(-1, 3)
    z, who = _hits(eye, d, V)
    ok = torch.isfinite(z)
    zz = torch.where(ok, z, torch.ones_like(z))
    X, N = (eye + d * zz[:, None]).reshape(H, W, 3), nrm[who].reshape(H, W, 3)
    ok, zz = ok.reshape(H, W), zz.reshape(H, W)
    # the voxels: every cell a triangle's box test takes keeps its last triangle
    n, vs = clip["G"] * 8, clip["v0"]
    lo = (torch.floor(eye / (8 * vs)) - clip["G"] // 2) * 8 * vs
    c0 = torch.floor((V.min(1).values - lo) / vs).clamp(0, n)
    m = ((torch.floor((V.max(1).values - lo) / vs) + 1).clamp(0, n) - c0).long().clamp(min=0)
    cnt = m.prod(-1)
    own = torch.repeat_interleave(torch.arange(V.shape[0], device=dev), cnt)
    q = torch.arange(own.shape[0], device=dev) - torch.repeat_interleave(cnt.cumsum(0) - cnt, cnt)
    mx, my = m[own, 0], m[own, 1]
    cell = c0[own].long() + torch.stack([q % mx, (q // mx) % my, q // (mx * my)], -1)
    w = V[own] - (lo + (cell + 0.5) * vs)[:, None, :]
    h = 0.5 * vs * 1.0001
    take = (w.min(1).values <= h).all(-1) & (w.max(1).values >= -h).all(-1)
    e = [w[:, 1] - w[:, 0], w[:, 2] - w[:, 1], w[:, 0] - w[:, 2]]
    axes = [torch.linalg.cross(e[0], e[1])] + [torch.linalg.cross(T(np.eye(3)[k]).expand_as(x), x) for x in e for k in range(3)]
    for ax in axes:
        pr, r = (w * ax[:, None, :]).sum(-1), h * ax.abs().sum(-1)
        take &= (pr.min(-1).values <= r) & (pr.max(-1).values >= -r)
    take |= cnt[own] == 1
    flat = (cell[:, 2] * n + cell[:, 1]) * n + cell[:, 0]
    rep = torch.full((n ** 3,), -1, dtype=torch.int64, device=dev)
    rep.scatter_reduce_(0, flat[take], own[take], "amax")
    # the cascades: probes, rays through the voxels, merged from the top
    pix = 2 * math.tan(s.camera.fov_y_deg * math.pi / 360) / H
    b = lambda k: p.kInterval * (4 ** k - 1) / 3  # noqa: E731
    probes, rays = [], []
    for c in range(p.cascades):
        ts, res = p.P << c, 4 << min(c, p.resCap)
        tx, ty = -(-W // ts), -(-H // ts)
        ix = (torch.arange(tx, device=dev) * ts + ts // 2).clamp(max=W - 1)
        iy = (torch.arange(ty, device=dev) * ts + ts // 2).clamp(max=H - 1)
        x, nn, valid, zc = (a[iy][:, ix].reshape(-1, *a.shape[2:]) for a in (X, N, ok, zz))
        s0 = (x - eye).norm(dim=-1) * pix * p.P
        o = x + nn * (p.lift * s0 * 2 ** c)[:, None]
        f = (torch.arange(res, device=dev, dtype=torch.float64) + 0.5) / res * 2 - 1
        fy, fx = torch.meshgrid(f, f, indexing="ij")
        fz = 1 - fx.abs() - fy.abs()
        t = (-fz).clamp(min=0)
        dirs = unit(torch.stack([fx - torch.where(fx >= 0, t, -t), fy - torch.where(fy >= 0, t, -t), fz], -1)).reshape(-1, 3)
        K = dirs.shape[0]
        ro = (o + nn * p.voxOffset * vs)[:, None, :].expand(-1, K, -1).reshape(-1, 3)
        rd = dirs[None].expand(o.shape[0], -1, -1).reshape(-1, 3)
        t0, t1 = (b(c) * s0).repeat_interleave(K), (b(c + 1) * s0).repeat_interleave(K)
        rad, tr = _walk(ro, rd, t0, t1, p.voxSkip * vs, rep, n, vs, lo, nrm, albedo, emit, sun, sun_e)
        live = valid.repeat_interleave(K)
        rad, tr = torch.where(live[:, None], rad, torch.zeros_like(rad)), torch.where(live, tr, torch.ones_like(tr))
        probes.append((tx, ty, ts, valid, zc, nn, dirs))
        rays.append((rad.reshape(ty * tx, res, res, 3), tr.reshape(ty * tx, res, res)))
    above = None
    for c in range(p.cascades - 1, -1, -1):
        tx, ty, ts, valid, zc, nn, dirs = probes[c]
        rad, tr = rays[c]
        if above is None:
            far = sky.expand_as(rad)
        else:
            ux, uy, us, uv, uz = probes[c + 1][:5]
            avg = above if above.shape[1] == rad.shape[1] else above.reshape(-1, rad.shape[1], 2, rad.shape[1], 2, 3).mean((2, 4))
            i = torch.arange(tx * ty, device=dev)
            gx, gy = (i % tx + 0.5) * ts / us - 0.5, (i // tx + 0.5) * ts / us - 0.5
            far, ws = torch.zeros_like(rad), torch.zeros(tx * ty, device=dev, dtype=torch.float64)
            for k in range(4):
                ox, oy = k & 1, k >> 1
                qx, qy = (gx.floor() + ox).clamp(0, ux - 1).long(), (gy.floor() + oy).clamp(0, uy - 1).long()
                j = qy * ux + qx
                fx, fy = gx - gx.floor(), gy - gy.floor()
                wt = ((fx if ox else 1 - fx) * (fy if oy else 1 - fy) + 1e-4) * (torch.exp(-20 * (uz[j] - zc).abs() / zc) + 1e-4)
                wt = torch.where(uv[j], wt, torch.zeros_like(wt))
                far, ws = far + avg[j] * wt[:, None, None, None], ws + wt
            far = torch.where((valid & (ws > 0))[:, None, None, None], far / ws.clamp(min=1e-300)[:, None, None, None], torch.zeros_like(far))
        above = rad + far * tr[..., None]
    # spherical harmonics of the first cascade's 16 directions, then the pixels
    tx, ty, ts, valid, zc, nn, dirs = probes[0]
    omega = T(fr.oct_solid_angles(4))

    def basis(v):
        x, y, z = v[..., 0], v[..., 1], v[..., 2]
        return torch.stack([0.282095 * torch.ones_like(x), 0.488603 * y, 0.488603 * z, 0.488603 * x, 1.092548 * x * y, 1.092548 * y * z,
                            0.315392 * (3 * z * z - 1), 1.092548 * x * z, 0.546274 * (x * x - y * y)], -1)
    band = T([math.pi] + [2 * math.pi / 3] * 3 + [math.pi / 4] * 5)
    sh = torch.einsum("pdc,d,dk->pkc", above.reshape(-1, 16, 3), omega, basis(dirs)) * band[:, None]
    gx, gy = ((px + 0.5) / ts - 0.5)[None].expand(H, W), ((py + 0.5) / ts - 0.5)[:, None].expand(H, W)
    y, e, ws = basis(N), torch.zeros(H, W, 3, device=dev, dtype=torch.float64), torch.zeros(H, W, device=dev, dtype=torch.float64)
    for k in range(4):
        ox, oy = k & 1, k >> 1
        j = (gy.floor() + oy).clamp(0, ty - 1).long() * tx + (gx.floor() + ox).clamp(0, tx - 1).long()
        fx, fy = gx - gx.floor(), gy - gy.floor()
        nd = (N * nn[j]).sum(-1).clamp(min=0)
        wt = ((fx if ox else 1 - fx) * (fy if oy else 1 - fy) + 1e-4) * (torch.exp(-20 * (zc[j] - zz).abs() / zz) + 1e-4) * (nd ** 4 + 1e-3)
        wt = torch.where(valid[j], wt, torch.zeros_like(wt))
        e, ws = e + torch.einsum("hwkc,hwk->hwc", sh[j], y).clamp(min=0) * wt[..., None], ws + wt
    e = torch.where((ok & (ws > 0))[..., None], e / ws.clamp(min=1e-300)[..., None], torch.zeros_like(e))
    return torch.cat([e, ok[..., None].double()], -1)


def _walk(o, d, t0, t1, skip, rep, n, vs, lo, nrm, albedo, emit, sun, sun_e):
    """Radiance and transmittance of [t0, t1] along every ray: cell by cell to the first occupied voxel."""
    hi = lo + n * vs
    dd = torch.where(d.abs() < 1e-9, torch.full_like(d, 1e-9), d)
    ta, tb = (lo - o) / dd, (hi - o) / dd
    t = torch.maximum(torch.minimum(ta, tb).max(-1).values, t0)
    end = torch.minimum(torch.maximum(ta, tb).min(-1).values, t1)
    rad, tr = torch.zeros_like(o), torch.ones_like(t)
    c = ((o + d * t[:, None] - lo) / vs).floor().clamp(0, n - 1).long()
    st = torch.where(dd > 0, 1, -1)
    live = t < end
    for _ in range(3 * n):
        idx = live.nonzero()[:, 0]
        if not idx.numel():
            break
        ci = c[idx]
        r = rep[(ci[:, 2] * n + ci[:, 1]) * n + ci[:, 0]]
        hit = (r >= 0) & (t[idx] >= skip)
        if hit.any():
            hi_, ri = idx[hit], r[hit]
            N = nrm[ri]
            N = torch.where((N * d[hi_]).sum(-1, keepdim=True) > 0, -N, N)
            rad[hi_] = emit[ri] + albedo[ri] / math.pi * sun_e * (N @ sun).clamp(min=0)[:, None]
            tr[hi_] = 0
        tm = ((ci + (st[idx] > 0)) * vs + lo - o[idx]) / dd[idx]
        t[idx], ax = tm.min(-1)
        c[idx, ax] += st[idx, ax]
        inside = ((c[idx] >= 0) & (c[idx] < n)).all(-1)
        live[idx] = ~hit & inside & (t[idx] < end[idx])
    return rad, tr
