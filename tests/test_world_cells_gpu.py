"""World probes where a warp's pixels spread over few and many grid cells: the gather's staged cells (more than four a warp, so
several rounds; ragged views; style tags) and registerPixels' cells (eight lanes a cell, strided pixels).  Counters, hash keys,
slots, SH and irradiance equal the oracle's bit for bit, over two solves."""
import numpy as np
import pytest

import test_world_gpu as T
from oracle import bind
from rtgi import configs, frame as fr, gpu, scenes

pytestmark = pytest.mark.gpu

CAPS = [32768, 16384, 8192, 4096, 2048]


@pytest.mark.parametrize("cfg,W,H,stride,toon", [("world-4-voxel-rc2-norel-f32", 61, 43, 1, False),
                                                 ("world-6-voxel-rc2-f16", 37, 21, 1, True),
                                                 ("world-96-voxel-rc2-bf16-f32out", 130, 67, 3, False),
                                                 ("world-5-voxel-rc2-vrel-f32", 70, 33, 2, False)])
def test_cells(cfg, W, H, stride, toon):
    room = scenes.room_scene(0)
    if toon:
        room.materials[2].flags = scenes.FLAG_TOON
        room.materials[0].flags = scenes.FLAG_TOON
    case = T._case("cells", room, W, H, cfg, T.ROOM_VOX, CAPS)
    F = case.frame.copy()
    F.view(np.uint32)[fr.F_RU + 2] = stride
    ctx = gpu.Context(0)
    frames = [(case.scene, F)] * 2
    g = T._gpu_frames(ctx, case, frames)
    ctx.destroy()
    lay = configs.world_layout(case.rc)
    state = bind.WorldState(lay)
    v = case.vox
    for f, gr in enumerate(g):
        st = bind.vox_build(case.scene, v.v0, v.levels, v.G, v.maxBricks, v.maxVoxels, case.scene.camera.eye)
        kw = {}
        if toon:
            _, _, tri = bind.raster_gbuffer(case.scene, F, W, H)
            kw["tag"] = bind.gbuffer_tags(case.scene, tri)
        o = bind.world_solve(st, lay, state, F, gr["depth"], gr["normal"].astype(np.float32), **kw)
        assert not o["counts"][16:24].any()
        T._eq(gr["counts"], o["counts"], f"frame {f} counts")
        T._eq(gr["keys"], o["keys"], f"frame {f} keys")
        occ = o["keys"] != 0
        T._eq(gr["slot_probe"][occ], o["slot_probe"][occ], f"frame {f} slots")
        n0 = min(int(o["counts"][0]), lay["casc"][0]["cap"])
        assert n0 > 8
        T._eq(gr["sh"][:n0, :27], o["sh"][:n0, :27], f"frame {f} SH")
        T._eq(gr["irr"], o["irr"], f"frame {f} irradiance")
