"""The shadow raster's groups of chunks: a warp takes 1, 2, 4 or 8 consecutive 128-texel chunks by the number of chunks there
are, crossing from triangle to triangle inside a group.  Scenes whose chunk totals lie on each side of the rule's lines (10,
1,484, 27,905, 47,442, 84,049 and 241,963 chunks), of wide boxes, boxes of less than a chunk and triangles without any texel
between them; every texel equals the oracle's map bit for bit."""
import numpy as np
import pytest

import test_shadow_gpu as T
from oracle import bind
from rtgi import frame as fr, gpu, scenes

pytestmark = pytest.mark.gpu


def _scene(n, spread, seed):
    """n triangles: every third spread over the map, every third small, every third outside it."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(-8, 8, (n, 3))
    ext = np.where(np.arange(n) % 3 == 0, spread, 0.05)[:, None]
    b, c = a + rng.uniform(-1, 1, (n, 3)) * ext, a + rng.uniform(-1, 1, (n, 3)) * ext
    for v in (a, b, c):
        v[np.arange(n) % 3 == 2] += 500.0
    pos = np.stack([a, b, c], 1).reshape(-1, 3).astype(np.float32)
    tri = np.zeros((n, 4), np.uint32)
    tri[:, :3] = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    nrm = np.tile(np.array([0, 1, 0], np.float32), (3 * n, 1))
    return scenes.Scene("shadow-groups", pos, nrm, tri, [scenes.Material("grey", (0.5, 0.5, 0.5, 1.0))],
                        scenes.Camera((0, 5, 20), (0, 0, 0), 60, 0.05), sun_dir=(-0.4, 1.0, 0.3))


# one chunk a group up to 37,887 chunks (148 SMs), two from 37,888, four from 75,776, eight from 151,552
@pytest.mark.parametrize("n,size,spread", [(1, 129, 20.0), (300, 256, 8.0), (600, 512, 14.0), (700, 600, 14.0), (900, 640, 16.0),
                                           (1200, 768, 20.0)])
def test_groups(n, size, spread):
    s = _scene(n, spread, n)
    F = fr.pack_frame(fr.FrameParams(cam=s.camera, width=64, height=64, sun_dir=s.sun_dir,
                                     light_view_proj=fr.scene_sun_view_proj([-12.0] * 3, [12.0] * 3, s.sun_dir),
                                     shadow_bias=fr.SHADOW_BIAS, cascades=2))
    ctx = gpu.Context(0)
    sg = gpu.SceneGpu(ctx, s)
    rc = gpu.Rc(ctx, T.gpu_params(), 64, 64)
    try:
        rc.set_frame(F)
        rc.render_shadow(sg, size)
        got = rc.read_shadow()
    finally:
        for h in (rc, sg, ctx):
            h.destroy()
    ref = bind.shadow_render(s, F, size)
    assert (ref < 1.0).any()
    bad = got.view(np.uint32) != ref.view(np.uint32)
    assert not bad.any(), f"{bad.sum()} texels differ, first at {np.argwhere(bad)[:4].tolist()}"
