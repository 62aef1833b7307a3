"""The cascade merge where a warp's quads belong to several probes, one probe or part of one: direction maps that stop
growing (rc0, rc1: the upper cascade read at the same resolution), views with fewer probes than a warp holds, ragged tile
counts and every atlas format.  The merged atlas, the SH and the irradiance equal the oracle's bit for bit."""
import numpy as np
import pytest

import gi_cases
from oracle import bind
from rtgi import _lib, configs, frame as fr, gpu, scenes

pytestmark = pytest.mark.gpu

CASES = [("screen-8-voxel-f32-rc0", 5, 7, 5), ("screen-8-voxel-f16-rc1", 4, 33, 17), ("screen-12-voxel-bf16-rc2", 5, 130, 71),
         ("screen-8-voxel-f32", 6, 97, 50), ("screen-16-voxel-f32-f32out-rc0", 3, 64, 200), ("screen-8-voxel-f16-f32out", 1, 45, 45)]


@pytest.mark.parametrize("cfg,cascades,W,H", CASES)
def test_merge_shapes(cfg, cascades, W, H):
    s = scenes.room_scene(1, n_boxes=60)
    p = configs.parse_config(cfg, {"cascades": cascades})
    v = configs.vox_params({"v0": 0.16, "levels": 2, "G": 8, "maxBricks": 1024, "maxVoxels": 1 << 18})
    F = gi_cases._frame(s, W, H, p, sun_e=fr.SUN_E, sky=fr.SKY)
    lay = configs.cascade_layout(p, W, H)
    ctx = gpu.Context(0)
    sg = gpu.SceneGpu(ctx, s)
    vw = gpu.VoxWorld(sg, v)
    rc = gpu.Rc(ctx, p, W, H)
    try:
        rc.set_frame(F)
        rc.render_gbuffer(sg)
        vw.update(s.camera.eye)
        depth = rc.read_buffer(_lib.GI_RC_DEPTH).view(np.float32).reshape(H, W)
        normal = rc.read_buffer(_lib.GI_RC_NORMAL).view(np.float16).reshape(H, W, 4).astype(np.float32)
        st = bind.vox_build(s, v.v0, v.levels, v.G, v.maxBricks, v.maxVoxels, s.camera.eye)
        o = bind.rc_solve(st, lay, F, depth, normal)
        for threads in (64, 256, 512):
            rc.set_tuning(merge_threads=threads)
            rc.solve(vw)
            for name, g in (("rad", rc.read_atlas(_lib.GI_RC_RAD)), ("sh", rc.read_atlas(_lib.GI_RC_SH)), ("irr", rc.read_irradiance())):
                e = np.asarray(o[name], np.float32)
                assert np.array_equal(g.reshape(-1).view(np.uint32), e.reshape(-1).view(np.uint32)), (name, threads)
    finally:
        for h in (rc, vw, sg, ctx):
            h.destroy()
