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


@pytest.mark.parametrize("count", [200, 1024, 1025, 5000])
def test_draw_list_in_a_recorded_graph(vox, count):
    """A recorded call against a direct one, replayed after a larger call of the same context."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(count)
    stream = torch.cuda.Stream()
    ctx = vox.Context(vox.make_config(chunk_size=16), stream=stream.cuda_stream)
    big = 400000
    coords = to_dev(rng.integers(-60, 60, (big, 3)).astype(np.int32))
    offs = to_dev(np.concatenate([[0], np.cumsum(rng.integers(0, 9, big))]).astype(np.uint64))
    planes = vox.frustum_planes(vox.camera_matrix((8.0, 30.0, -4.0), (0.7, -0.2, 0.6)))
    want, draws, many = (dev_bytes(20 * k, fill=7) for k in (count, count, big))
    n_want, n_draws = dev_bytes(4), dev_bytes(4)
    torch.cuda.synchronize()
    ctx.draw_list(planes, coords, offs, count, want, n_want)
    ctx.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        ctx.draw_list(planes, coords, offs, count, draws, n_draws)
    ctx.draw_list(planes, coords, offs, big, many, dev_bytes(4))
    ctx.sync()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(to_np(n_draws)[:4], to_np(n_want)[:4])  # (behind them nothing is written)
    assert np.array_equal(to_np(draws)[:20 * count], to_np(want)[:20 * count])
    ctx.close()
