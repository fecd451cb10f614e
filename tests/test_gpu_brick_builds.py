"""Occupancy bricks of volumes of every proportion: long and thin along one
axis, flat, small, rows and slices that need several blocks, for the word
reads and the byte reads, against the layout's definition."""
import numpy as np
import pytest

from helpers import bricks_from_voxels
from voxeltoy_gb300 import Context, Scene
from voxeltoy_gb300 import _lib as L
from voxeltoy_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bctx():
    c = Context()
    yield c
    c.close()


@pytest.mark.parametrize("res", [
    (1, 1, 1), (5, 3, 2), (24, 24, 24), (4, 40, 4), (120, 9, 130), (131, 70, 93), (128, 65, 12),   # x, y, z
    (9000, 1, 1), (8192, 2, 3), (1, 9000, 1), (2, 3, 9000), (60000, 5, 1), (1048574, 1, 1), (1, 1048574, 1),
    (1, 1, 524286), (4, 1, 524286),
])
@pytest.mark.parametrize("shape", [(2, 2, 2), (1, 2, 3), (4, 1, 1)])
def test_bricks(bctx, res, shape):
    rng = np.random.default_rng(sum(res))
    vox = (rng.random(res[::-1]) < 0.2).astype(np.uint8)
    vox[-1, -1, -1] = 3                                     # the largest entry in the last voxel
    palette = [S.lambert(0.5)] * 3
    sc = Scene.dense(bctx, vox, palette)
    try:
        sc.set_brick_shape(shape)
        assert np.array_equal(sc.bricks(), bricks_from_voxels(vox, shape))
    finally:
        sc.close()
    with pytest.raises(L.VtError):
        Scene.dense(bctx, vox, palette[:2])
