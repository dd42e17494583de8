"""The rasteriser's ways through a triangle's box (a lane, a warp, tiles, a full tile list) against
the oracle's image: quads from below a pixel to beyond the screen, image sizes at the tile edges,
and image buffers off the alignment of the tile list that is kept in them.
"""
import ctypes

import numpy as np
import pytest

from gpu_util import ctx_for, dev_bytes, to_dev, to_np

pytestmark = pytest.mark.gpu


def quads(count, rng, size):
    """count faces with corners around random centres, `size` the largest half extent in NDC."""
    v = np.zeros((count, 4), dtype=[("p", "f4", 3), ("t", "f4", 2), ("f", "u4")])
    centre = rng.uniform(-1.2, 1.2, (count, 1, 2))
    half = size * rng.random((count, 1, 1)) ** 3
    corner = np.array([[-1, -1], [1, -1], [-1, 1], [1, 1]]) * rng.choice([-1, 1], (count, 1, 2))
    v["p"][..., :2] = centre + half * (corner + rng.uniform(-0.3, 0.3, (count, 4, 2)))
    v["p"][..., 2] = rng.uniform(-0.05, 1.05, (count, 1)) + rng.uniform(-0.1, 0.1, (count, 4))
    v["t"] = [[0, 0], [1, 0], [0, 1], [1, 1]]
    v["f"] = rng.integers(0, 6, (count, 1))
    index = 4 * np.arange(count, dtype=np.uint32)[:, None] + np.array([0, 2, 1, 3, 1, 2], np.uint32)
    return v, index


@pytest.mark.parametrize("width,height,count,size", [
    (1, 1, 40, 2.0), (33, 31, 500, 2.0), (64, 64, 3000, 3.0), (257, 130, 4000, 0.5),
    (640, 360, 300, 3.0), (511, 1, 200, 1.0)])
@pytest.mark.parametrize("offset", [0, 5])
def test_raster_matches_oracle(vox, oracle, width, height, count, size, offset):
    rng = np.random.default_rng(width * 7 + count)
    v, index = quads(count, rng, size)
    view = np.eye(4, dtype=np.float32).reshape(16)
    view[11] = 0.25  # w = 1 + z / 4: perspective
    cfg = vox.make_config(chunk_size=16)
    want = oracle.raster(list(view), v.tobytes(), index.tobytes(), count, width, height, cfg.texture_index)
    ctx = ctx_for(vox, cfg)
    d0, d1 = to_dev(np.frombuffer(v.tobytes(), np.uint8)), to_dev(np.frombuffer(index.tobytes(), np.uint8))
    keys, rgba = dev_bytes(width * height * 8), dev_bytes(width * height * 4 + 16, fill=0x5A)
    m = (ctypes.c_float * 16)(*[float(x) for x in view])
    for _ in range(2):
        st = vox.lib().vox_raster(ctx._h, ctypes.addressof(m), d0.data_ptr(), d1.data_ptr(), count, width,
                                  height, keys.data_ptr(), rgba.data_ptr() + offset)
        assert st == vox.VOX_OK
        ctx.sync()
        got = to_np(rgba)
        assert np.array_equal(got[offset:offset + width * height * 4], np.asarray(want).reshape(-1))
        assert (got[:offset] == 0x5A).all() and (got[offset + width * height * 4:] == 0x5A).all()
    ctx.close()
