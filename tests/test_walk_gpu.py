"""The voxel walk's edges: step caps of one to a few (a walk cut in an empty run and inside a brick), the smallest clipmap (one
brick from the window's edge), a pool that drops bricks (cells read at the coarser level) at one and several levels, rays that
start outside the window, and every trace order.  DDA hits with their entry times, step counters and irradiance equal the
oracle's."""
import numpy as np
import pytest

import gi_cases
from oracle import bind
from rtgi import _lib, configs, frame as fr, gpu, scenes

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 4, 64, 4), (2, 2, 4, 128, 3), (3, 3, 16, 8192, 5), (7, 2, 8, 40, 4), (64, 1, 8, 30, 5), (1024, 3, 16, 200, 5)]


@pytest.mark.parametrize("cap,levels,G,bricks,cascades", CASES)
def test_walk(cap, levels, G, bricks, cascades):
    W, H = 75, 50
    s = scenes.room_scene(2, n_boxes=80)
    p = configs.parse_config(f"screen-8-voxel-f32-dda{cap}", {"cascades": cascades})
    p.stats = 1
    v = configs.vox_params({"v0": 0.08, "levels": levels, "G": G, "maxBricks": bricks, "maxVoxels": 1 << 18})
    F = gi_cases._frame(s, W, H, p, sun_e=fr.SUN_E, sky=fr.SKY)
    lay = configs.cascade_layout(p, W, H)
    ctx = gpu.Context(0)
    sg = gpu.SceneGpu(ctx, s)
    vw = gpu.VoxWorld(sg, v)
    rc = gpu.Rc(ctx, p, W, H)
    try:
        rc.set_debug_hits(True)
        rc.set_frame(F)
        rc.render_gbuffer(sg)
        vw.update(s.camera.eye)
        depth = rc.read_buffer(_lib.GI_RC_DEPTH).view(np.float32).reshape(H, W)
        normal = rc.read_buffer(_lib.GI_RC_NORMAL).view(np.float16).reshape(H, W, 4).astype(np.float32)
        st = bind.vox_build(s, v.v0, v.levels, v.G, v.maxBricks, v.maxVoxels, s.camera.eye)
        o = bind.rc_solve(st, lay, F, depth, normal, want_hit=True)
        if bricks in (40, 30, 200):
            assert st["hdr"][2] > 0, "the pool must drop bricks"
        for order in (0, 1, 2, 2):
            rc.set_tuning(trace_order=order)
            rc.solve(vw)
            hits = rc.read_buffer(_lib.GI_RC_HITS).view(np.uint32).reshape(-1, 4)
            assert np.array_equal(hits, o["hit"]), order
            counts = rc.read_counts()
            assert np.array_equal(counts[24:24 + cascades], o["counts"][24:24 + cascades]), order
            assert np.array_equal(counts[32:32 + cascades], o["counts"][32:32 + cascades]), order
            assert np.array_equal(counts[64:64 + cascades], o["counts"][64:64 + cascades]), order
            assert np.array_equal(rc.read_irradiance().view(np.uint32), o["irr"].view(np.uint32)), order
    finally:
        for h in (rc, vw, sg, ctx):
            h.destroy()
