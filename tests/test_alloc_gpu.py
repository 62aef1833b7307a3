"""The ordered brick allocation at the edges of its launch shapes: 1, 4 or 16 pointers per thread by the number of pointers
(levels x G^3), ragged last parts, one part and many, and pointer outputs that are not 16-byte aligned (scalar loads).
Pointers, brick codes and the header counts equal the oracle's; integers, so exactly."""
import ctypes as C

import numpy as np
import pytest

from oracle import bind
from rtgi import _lib, configs, gpu, scenes

pytestmark = pytest.mark.gpu

# levels, G: one part of 64 pointers; 8192 - 64 x 1 and just past 8192 (4 per thread); ragged last part; past 524,288 (16)
SHAPES = [(1, 4), (8, 8), (2, 16), (5, 12), (5, 20), (3, 56), (7, 44)]


def _check(hdr, ptr, code, st, what):
    assert np.array_equal(hdr[[0, 1, 2, 3, 4, 6]], st["hdr"][[0, 1, 2, 3, 4, 6]]), what
    assert np.array_equal(hdr[8:16], st["hdr"][8:16]), what
    assert np.array_equal(ptr, st["ptr"]), what
    nb = int(min(hdr[0], len(code)))
    assert np.array_equal(code[:nb], st["code"][:nb]), what


@pytest.mark.parametrize("levels,G", SHAPES)
@pytest.mark.parametrize("bricks", [4096, 40])   # 40: the pool overflows, bricks are dropped in order
def test_brick_allocation_shapes(levels, G, bricks):
    import torch
    s = scenes.room_scene(0, n_boxes=30)
    v = configs.vox_params({"v0": 0.05, "levels": levels, "G": G, "maxBricks": bricks, "maxVoxels": 1 << 18})
    eye = s.camera.eye
    st = bind.vox_build(s, v.v0, v.levels, v.G, v.maxBricks, v.maxVoxels, eye)
    ctx = gpu.Context(0)
    sg = gpu.SceneGpu(ctx, s)
    vw = gpu.VoxWorld(sg, v)
    try:
        vw.update(eye)
        vw.encode()
        g = vw.read_state()
        _check(g["hdr"], g["ptr"], g["code"], st, "gi_vox_build")
    finally:
        for h in (vw, sg, ctx):
            h.destroy()
    # the caller's own buffers, the pointers one word off 16-byte alignment
    dev = torch.device("cuda", 0)
    pos, nrm = (torch.zeros((a.shape[0], 4), dtype=torch.float32, device=dev) for a in (s.positions, s.normals))
    pos[:, :3], nrm[:, :3] = torch.from_numpy(s.positions).to(dev), torch.from_numpy(s.normals).to(dev)
    tri = torch.from_numpy(np.ascontiguousarray(s.tri, np.uint32).view(np.int32)).to(dev)
    mats = torch.from_numpy(s.material_array().view(np.uint8)).to(dev)
    n = v.levels * v.G ** 3
    words = {"hdr": 64, "ptr": n + 4, "occ": bricks * 16, "base": bricks, "code": bricks, "attr": v.maxVoxels * 4,
             "plane": v.maxVoxels, "sunvis": v.maxVoxels}
    out = {k: torch.zeros(c, dtype=torch.int32, device=dev) for k, c in words.items()}
    p = _lib.GiVoxParams(float(v.v0), v.levels, v.G, v.maxBricks, v.maxVoxels, v.dynBricks, 0)
    at = {k: t.data_ptr() for k, t in out.items()}
    assert at["ptr"] % 16 == 0
    at["ptr"] += 4
    _lib.call("gi_vox_build_noalloc", C.byref(p), (C.c_double * 3)(*[float(x) for x in eye]), pos.data_ptr(), nrm.data_ptr(),
              pos.shape[0], tri.data_ptr(), tri.shape[0], mats.data_ptr(), len(s.materials), at["hdr"], at["ptr"], at["occ"],
              at["base"], at["code"], at["attr"], at["plane"], at["sunvis"], None)
    torch.cuda.synchronize()
    get = lambda k: out[k].cpu().numpy().view(np.uint32)
    _check(get("hdr"), get("ptr")[1:n + 1], get("code"), st, "gi_vox_build_noalloc")
