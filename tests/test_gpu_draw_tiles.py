"""The draw list over several tiles of 256 chunks, and the frustum test's corner lanes, at counts
around a tile and over many: records against numpy, from the visibility that the frustum test
gives for the same chunks (checked against the oracle elsewhere, and here for a sample).
"""
import numpy as np
import pytest

from gpu_util import ctx_for, dev_bytes, to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [0, 1, 255, 256, 257, 3001, 70000])
@pytest.mark.parametrize("layout", [0, 1])
def test_draw_list_matches_numpy(vox, oracle, count, layout):
    rng = np.random.default_rng(count)
    cfg = vox.make_config(chunk_size=16, layout=layout)
    ctx = ctx_for(vox, cfg)
    coords = rng.integers(-60, 60, (max(count, 1), 3)).astype(np.int32)
    faces = rng.integers(0, 4, max(count, 1)) * rng.integers(0, 300, max(count, 1))
    offs = np.concatenate([[0], np.cumsum(faces)]).astype(np.uint64)
    eye = (8.0, 30.0, -4.0)
    planes = vox.frustum_planes(vox.camera_matrix(eye, (0.7, -0.2, 0.6)))
    d_coords, d_offs = to_dev(coords), to_dev(offs)
    visible, draws, n_draws = dev_bytes(max(count, 1), fill=9), dev_bytes(20 * max(count, 1), fill=7), dev_bytes(4)
    for _ in range(2):
        ctx.frustum_cull(planes, d_coords, count, visible)
        ctx.draw_list(planes, d_coords, d_offs, count, draws, n_draws)
        ctx.sync()
    vis = to_np(visible)[:count] == 1
    sample = rng.integers(0, max(count, 1), 200) if count else []
    for i in sample:
        assert vis[i] == oracle.frustum_contains(planes, tuple(int(v) for v in coords[i]), 16)
    at = np.flatnonzero(vis & (faces[:count] > 0))
    assert int(to_np(n_draws).view(np.uint32)[0]) == len(at)
    want = np.zeros((len(at), 5), np.uint32)
    if layout == 0:
        want[:, 0], want[:, 1] = 6 * faces[at], 1
        want[:, 2], want[:, 3] = 6 * offs[at], 4 * offs[at]
    else:
        want[:, 0], want[:, 1], want[:, 4] = 6, faces[at], offs[at]
    got = to_np(draws).view(np.uint8)
    assert np.array_equal(got[:20 * len(at)].view(np.uint32).reshape(-1, 5), want)
    assert (got[20 * len(at):20 * count] == 7).all()
    ctx.close()
