"""The G-buffer raster's lists: warps of pairs from a single triangle (its tiles distinct, one atomic each), from about four and
from dozens (tiles shared, one atomic for the lanes that do), and a list capacity that cuts through such warps.  Depth, normal and
tag equal the oracle's brute-force raster bit for bit."""
import numpy as np
import pytest

import gi_cases
import test_raster_dealt_gpu as T
from oracle import bind
from rtgi import _lib, configs, frame as fr, gpu

pytestmark = pytest.mark.gpu


def check(s, W, H, cap=0, share=0.1):
    p = configs.parse_config("screen-8-voxel-f32", {"cascades": 1})
    F = gi_cases._frame(s, W, H, p, sun_e=fr.SUN_E, sky=fr.SKY)
    ctx = gpu.Context(0)
    sg = gpu.SceneGpu(ctx, s)
    rc = gpu.Rc(ctx, p, W, H)
    try:
        if cap:
            sg.set_raster_capacity(cap)
        rc.set_frame(F)
        for _ in range(2):
            rc.render_gbuffer(sg)
        depth = rc.read_buffer(_lib.GI_RC_DEPTH).view(np.uint32)
        normal = rc.read_buffer(_lib.GI_RC_NORMAL).view(np.float16).reshape(H, W, 4).astype(np.float32)
        tag = rc.read_buffer(_lib.GI_RC_TAG)
    finally:
        for h in (rc, sg, ctx):
            h.destroy()
    d, nn, tri = bind.raster_gbuffer(s, F, W, H)
    assert (np.asarray(d) > 0).mean() > share
    assert np.array_equal(depth, np.asarray(d, np.float32).reshape(-1).view(np.uint32))
    assert np.array_equal(normal[..., :3], np.asarray(nn, np.float32).reshape(H, W, -1)[..., :3])
    assert np.array_equal(tag, np.asarray(bind.gbuffer_tags(s, tri)).reshape(-1))


# boxes of hundreds of tiles, of about eight, of one or two; the last two with lists that end inside a warp's pairs
@pytest.mark.parametrize("n,W,H,size,cap", [(31, 500, 300, 2.0, 0), (600, 256, 144, 0.12, 0), (5000, 256, 144, 0.02, 0),
                                            (600, 256, 144, 0.12, 1003), (257, 333, 97, 0.5, 131)])
def test_pairs(n, W, H, size, cap):
    check(T._soup(n, 3 * n + W, size, False), W, H, cap)
