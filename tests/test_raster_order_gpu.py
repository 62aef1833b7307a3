"""The G-buffer raster's walk of a tile's large triangles front to back: hundreds of sheets that cover the tile, whose depth bounds
lie closer than the 256 units in the last place that the order resolves, further apart, or exactly on one another, in random
order; and boxes on both sides of the large / small line.  Depth, normal and tag equal the oracle's bit for bit."""
import numpy as np
import pytest

import test_raster_dealt_gpu as T
from test_raster_lists_gpu import check
from rtgi import scenes

pytestmark = pytest.mark.gpu


def _sheets(n, step, half, seed):
    """n triangles across the view axis at distances 3 + k step, in random order, each tilted a little and moved sideways."""
    rng = np.random.default_rng(seed)
    x = 3.0 + step * rng.permutation(n)
    tilt = rng.uniform(-2.0, 2.0, (n, 2)) * step
    c = rng.uniform(-0.2, 0.2, (n, 2)) * half
    yz = np.array([[-1.0, -1.0], [1.0, -1.0], [0.0, 1.4]])[None] * half + c[:, None, :]
    pos = np.concatenate([x[:, None, None] + (yz * tilt[:, None, :]).sum(-1, keepdims=True), yz], -1).reshape(-1, 3).astype(np.float32)
    nr = np.cross(pos[1::3] - pos[0::3], pos[2::3] - pos[0::3])
    nr /= np.maximum(np.linalg.norm(nr, axis=1, keepdims=True), 1e-12)
    tri = np.concatenate([np.arange(3 * n).reshape(-1, 3), rng.integers(0, 2, (n, 1))], 1).astype(np.uint32)
    mats = [scenes.Material("a", (0.7, 0.6, 0.5, 1.0), flags=scenes.FLAG_TOON), scenes.Material("b", (0.2, 0.9, 0.4, 1.0))]
    return scenes.Scene("sheets", pos, np.repeat(nr, 3, 0).astype(np.float32), tri, mats,
                        scenes.Camera((0.0, 0.0, 0.0), (1.0, 0.0, 0.0), 60, 0.05), sun_dir=(0.2, 1.0, 0.1))


@pytest.mark.parametrize("n,step,half,W,H", [(700, 1e-6, 4.0, 16, 16), (700, 1e-3, 4.0, 33, 17), (255, 0.0, 4.0, 16, 16),
                                             (257, 2e-5, 0.4, 64, 48), (513, 1e-4, 0.9, 40, 40)])
def test_sheets(n, step, half, W, H):
    check(_sheets(n, step, half, n), W, H, share=0.02)   # a sheet of half width 0.4 covers 2.4 % of the view


@pytest.mark.parametrize("size", [0.1, 0.2, 0.35])   # boxes around 80 pixels of a tile
def test_line(size):
    check(T._soup(1500, 77, size, True), 48, 32)
