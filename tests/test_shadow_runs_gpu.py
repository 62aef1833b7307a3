"""The shadow raster's runs of 128 texels and their row rejection: boxes just under, at and over a run's width, boxes of more
than 4096 texels (longer chunks), maps of sizes that are no power of two, and light windows from a part of the triangles' extent
to several times it.  Every texel equals the oracle's brute-force map bit for bit."""
import numpy as np
import pytest

import test_shadow_gpu as T
from oracle import bind
from rtgi import frame as fr, gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,half,seed,n", [(127, 14.0, 5, 700), (128, 9.0, 6, 700), (130, 40.0, 7, 1500),
                                              (517, 6.0, 8, 400), (900, 14.0, 9, 300), (1, 10.0, 10, 50)])
def test_runs(size, half, seed, n):
    s = T._stress_scene(seed, n)
    F = fr.pack_frame(fr.FrameParams(cam=s.camera, width=64, height=64, sun_dir=s.sun_dir,
                                     light_view_proj=fr.scene_sun_view_proj([-half] * 3, [half] * 3, s.sun_dir),
                                     shadow_bias=fr.SHADOW_BIAS, cascades=2))
    ctx = gpu.Context(0)
    sg = gpu.SceneGpu(ctx, s)
    rc = gpu.Rc(ctx, T.gpu_params(), 64, 64)
    try:
        rc.set_frame(F)
        for _ in range(2):
            rc.render_shadow(sg, size)
        got = rc.read_shadow()
    finally:
        for h in (rc, sg, ctx):
            h.destroy()
    ref = bind.shadow_render(s, F, size)
    bad = got.view(np.uint32) != ref.view(np.uint32)
    assert not bad.any(), f"{bad.sum()} texels differ, first at {np.argwhere(bad)[:4].tolist()}"
