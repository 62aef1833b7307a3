"""The search of each voxel's brick by a whole warp (resolveAttr, bnInject) at its edges: fewer than 32 bricks and past 32 and
33 x 32 of them, bricks of one voxel (a warp passes 32 bricks) and of hundreds, and a voxel pool that ends inside them.  The
attributes equal the oracle's word for word."""
import numpy as np
import pytest

from oracle import bind
from rtgi import configs, gpu, scenes

pytestmark = pytest.mark.gpu


def _specks(n, size):
    """n triangles of the given size, each inside its own brick (0.4 m at 0.05 m voxels) of a 16^3 grid around the origin"""
    rng = np.random.default_rng(n)
    cell = rng.permutation(14 ** 3)[:n]
    c = np.stack([cell % 14, cell // 14 % 14, cell // 196], 1) - 7 + 0.5
    pos = (c[:, None, :] * 0.4 + rng.uniform(-1, 1, (n, 3, 3)) * size).reshape(-1, 3).astype(np.float32)
    nr = np.cross(pos[1::3] - pos[0::3], pos[2::3] - pos[0::3])
    nr /= np.maximum(np.linalg.norm(nr, axis=1, keepdims=True), 1e-12)
    tri = np.concatenate([np.arange(3 * n).reshape(-1, 3), np.zeros((n, 1), int)], 1).astype(np.uint32)
    return scenes.Scene("specks", pos, np.repeat(nr, 3, 0).astype(np.float32), tri, [scenes.Material("a", (0.7, 0.6, 0.5, 1.0))],
                        scenes.Camera((0.1, 0.2, 0.3), (1, 0, 0), 60, 0.05))


@pytest.mark.parametrize("n,size,levels,pool", [(1, 0.001, 1, 4096), (31, 0.001, 1, 4096), (33, 0.15, 1, 4096), (1056, 0.001, 1, 1 << 16),
                                                (1100, 0.02, 2, 1 << 16), (2700, 0.15, 3, 1 << 18), (2700, 0.001, 1, 1111)])
def test_voxel_bricks(n, size, levels, pool):
    s = _specks(n, size)
    v = configs.vox_params({"v0": 0.05, "levels": levels, "G": 16, "maxBricks": 8192, "maxVoxels": pool})
    eye = (0.0, 0.0, 0.0)
    st = bind.vox_build(s, v.v0, v.levels, v.G, v.maxBricks, v.maxVoxels, eye)
    ctx = gpu.Context(0)
    sg = gpu.SceneGpu(ctx, s)
    vw = gpu.VoxWorld(sg, v)
    try:
        vw.update(eye)
        vw.encode()
        g = vw.read_state()
    finally:
        for h in (vw, sg, ctx):
            h.destroy()
    nb = int(min(g["hdr"][0], v.maxBricks))
    fits = st["base"][:nb] != 0xffffffff   # a brick that does not fit the pool whole has no attributes
    ends = st["base"][:nb][fits] + np.unpackbits(st["occ"][:nb * 16].view(np.uint8)).reshape(nb, -1).sum(1)[fits]
    nv = int(ends.max())
    assert nb >= n and nv > min(n, pool) - 512
    assert np.array_equal(g["hdr"], st["hdr"])
    for k, m in (("base", nb), ("attr", nv * 4)):
        assert np.array_equal(g[k][:m], st[k][:m]), k
    assert np.array_equal(g["plane"][:nv].view(np.uint32), st["plane"][:nv].view(np.uint32))
