"""The world gather's two ways to its probes in one view: warps of up to four grid cells (staged) beside warps of more (read one by
one), with and without style tags, in views narrower and wider than a warp's 4 x 8 tile.  Counters, hash keys, slots, SH and
irradiance equal the oracle's bit for bit, over two solves."""
import pytest

import test_world_cells_gpu as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg,W,H,toon", [("world-48-voxel-rc2-f32", 150, 61, True), ("world-24-voxel-rc2-norel-f16", 97, 55, True),
                                          ("world-16-voxel-rc2-bf16", 121, 67, False), ("world-24-voxel-rc2-f16-f32out", 3, 50, False),
                                          ("world-24-voxel-rc2-f32-irr16", 41, 5, True)])
def test_gather(cfg, W, H, toon):
    T.test_cells(cfg, W, H, 1, toon)
