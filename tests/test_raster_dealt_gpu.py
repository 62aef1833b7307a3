"""The G-buffer raster where a tile's triangles are dealt out pixel by pixel: thousands of triangles of a few pixels in one tile
(several chunks), boxes from one pixel to the whole tile on both sides of the large / small line, views smaller than a tile,
equal depths (duplicated triangles: the smaller index wins), alpha-masked fragments, and a forced overflow of the lists.  Depth,
normal and tag equal the oracle's brute-force raster bit for bit."""
import numpy as np
import pytest

import gi_cases
from oracle import bind
from rtgi import _lib, configs, frame as fr, gpu, scenes

pytestmark = pytest.mark.gpu


def _soup(n, seed, size, masked):
    rng = np.random.default_rng(seed)
    z = rng.uniform(0.5, 12.0, n)                      # in front of a camera at the origin looking along +x
    c = np.stack([z, z * rng.uniform(-0.4, 0.4, n), z * rng.uniform(-0.6, 0.6, n)], -1)[:, None, :]
    r = (z * size * np.exp(rng.uniform(-2.5, 0.5, n)))[:, None, None]
    pos = (c + rng.uniform(-1, 1, (n, 3, 3)) * r).reshape(-1, 3).astype(np.float32)
    pos[-30:] = pos[:30]                               # ten duplicates
    nr = np.cross(pos[1::3] - pos[0::3], pos[2::3] - pos[0::3])
    nr /= np.maximum(np.linalg.norm(nr, axis=1, keepdims=True), 1e-12)
    tri = np.concatenate([np.arange(3 * n).reshape(-1, 3), rng.integers(0, 2, (n, 1))], 1).astype(np.uint32)
    mats = [scenes.Material("a", (0.7, 0.6, 0.5, 1.0), flags=scenes.FLAG_TOON),
            scenes.Material("b", (0.2, 0.9, 0.4, 0.4 if masked else 1.0), flags=scenes.FLAG_ALPHA_MASK if masked else 0)]
    return scenes.Scene("soup", pos, np.repeat(nr, 3, 0).astype(np.float32), tri, mats,
                        scenes.Camera((0.0, 0.0, 0.0), (1.0, 0.0, 0.0), 60, 0.05), sun_dir=(0.2, 1.0, 0.1))


@pytest.mark.parametrize("n,W,H,size,masked,cap", [(4000, 16, 16, 0.2, False, 0), (6000, 123, 61, 0.03, True, 0),
                                                   (3000, 5, 3, 0.3, False, 0), (2500, 200, 112, 0.15, False, 700),
                                                   (300, 97, 64, 0.6, True, 0)])
def test_dealt_raster(n, W, H, size, masked, cap):
    s = _soup(n, n + W, size, masked)
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
    assert (np.asarray(d) > 0).mean() > 0.1   # the soup covers part of the view
    assert np.array_equal(depth, np.asarray(d, np.float32).reshape(-1).view(np.uint32))
    assert np.array_equal(normal[..., :3], np.asarray(nn, np.float32).reshape(H, W, -1)[..., :3])
    assert np.array_equal(tag, np.asarray(bind.gbuffer_tags(s, tri)).reshape(-1))
