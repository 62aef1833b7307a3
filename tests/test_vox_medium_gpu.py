"""voxBits' big triangles of every handling: groups of 1, 2, 4 and 8 medium items a warp (by how many there are), the largest
medium range and the smallest chunked one, thin ranges along each axis, and alpha-masked materials.  Random triangles of
0.2 to 1.2 m around the camera at 0.1 m voxels; the voxel state equals the oracle's word for word."""
import numpy as np
import pytest

from oracle import bind
from rtgi import configs, gpu, scenes

pytestmark = pytest.mark.gpu


def _soup(n, seed, masked):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-5.5, 5.5, (n, 1, 3))
    size = rng.uniform(0.1, 0.6, (n, 1, 1))
    off = rng.uniform(-1, 1, (n, 3, 3)) * size
    thin = rng.integers(0, 4, n)                      # a third axis flattened for three quarters of them
    for a in range(3):
        off[thin == a, :, a] *= 0.02
    pos = (c + off).reshape(-1, 3).astype(np.float32)
    e1, e2 = pos[1::3] - pos[0::3], pos[2::3] - pos[0::3]
    nr = np.cross(e1, e2)
    nr /= np.maximum(np.linalg.norm(nr, axis=1, keepdims=True), 1e-12)
    tri = np.concatenate([np.arange(3 * n).reshape(-1, 3), rng.integers(0, 2, (n, 1))], 1).astype(np.uint32)
    mats = [scenes.Material("a", (0.7, 0.6, 0.5, 1.0)),
            scenes.Material("b", (0.2, 0.9, 0.4, 0.4 if masked else 1.0), flags=scenes.FLAG_ALPHA_MASK if masked else 0)]
    return scenes.Scene("soup", pos, np.repeat(nr, 3, 0).astype(np.float32), tri, mats,
                        scenes.Camera((0.1, 0.2, 0.3), (1, 0, 0), 60, 0.05))


@pytest.mark.parametrize("n,masked", [(300, False), (6000, True), (16000, False), (40000, False), (70000, False)])
def test_big_triangles(n, masked):
    s = _soup(n, n, masked)
    v = configs.vox_params({"v0": 0.1, "levels": 3, "G": 16, "maxBricks": 12288, "maxVoxels": 1 << 22})
    st = bind.vox_build(s, v.v0, v.levels, v.G, v.maxBricks, v.maxVoxels, s.camera.eye)
    ctx = gpu.Context(0)
    sg = gpu.SceneGpu(ctx, s)
    vw = gpu.VoxWorld(sg, v)
    try:
        vw.update(s.camera.eye)
        for _ in range(2):
            vw.encode()
        g = vw.read_state()
    finally:
        for h in (vw, sg, ctx):
            h.destroy()
    nb, nv = int(min(g["hdr"][0], v.maxBricks)), int(min(g["hdr"][1], v.maxVoxels))
    assert g["hdr"][3] == 0 and int(g["hdr"][16:24].sum()) > n // 2
    assert np.array_equal(g["hdr"], st["hdr"])
    for k, m in (("ptr", None), ("occ", nb * 16), ("base", nb), ("rep", nb * 512), ("attr", nv * 4)):
        assert np.array_equal(g[k][:m], st[k][:m]), k
    assert np.array_equal(g["plane"][:nv].view(np.uint32), st["plane"][:nv].view(np.uint32))
