"""The draw list's tickets and look-back words are its own: lists and batches of one context that run
at the same time, the batches replayed by a caller's graph on another stream.
"""
import numpy as np
import pytest

from gpu_util import dev_bytes, to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,n", [(300, 40), (5000, 900), (70000, 2000)])
def test_draw_lists_beside_replayed_batches(vox, count, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(count)
    main, other = torch.cuda.Stream(), torch.cuda.Stream()
    cfg = vox.make_config(chunk_size=16, kind=vox.GEN_HEIGHTMAP, octaves=2, frequency=1 / 40, amplitude=20.0,
                          base_height=8.0, seed=3)
    ctx = vox.Context(cfg, stream=main.cuda_stream)
    side = int(np.ceil(np.sqrt(n)))
    c = to_dev(np.array([(i % side, 0, i // side) for i in range(n)], np.int32))
    m = to_dev(np.full(n, 15, np.uint8))
    room = 6 * 256 * n
    o0, o1, offs = dev_bytes(room * 96, fill=1), dev_bytes(room * 24, fill=1), to_dev(np.zeros(n + 1, np.uint64))
    coords = to_dev(rng.integers(-60, 60, (count, 3)).astype(np.int32))
    faces = rng.integers(0, 4, count) * rng.integers(0, 300, count)
    d_offs = to_dev(np.concatenate([[0], np.cumsum(faces)]).astype(np.uint64))
    planes = vox.frustum_planes(vox.camera_matrix((8.0, 30.0, -4.0), (0.7, -0.2, 0.6)))
    rounds = 60
    draws, numbers = dev_bytes(rounds * 20 * count, fill=7), dev_bytes(4 * rounds, fill=7)
    to_np(draws)  # waits: everything above is in place

    ctx.gen_mesh_batch(c, m, n, o0, o1, room, offs)
    ctx.draw_list(planes, coords, d_offs, count, draws, numbers)
    ctx.sync()
    want = [to_np(t).copy() for t in (o0, o1, offs)]
    total = int(to_np(numbers).view(np.uint32)[0])
    records = to_np(draws)[:20 * total].copy()
    assert 0 < total < count and int(want[2][n]) <= room
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=main):
        ctx.gen_mesh_batch(c, m, n, o0, o1, room, offs)
    for t in (o0, o1):
        t.fill_(1)
    draws.fill_(7)
    torch.cuda.synchronize()
    for r in range(rounds):
        with torch.cuda.stream(other):
            graph.replay()
        ctx.draw_list(planes, coords, d_offs, count, draws[20 * count * r:], numbers[4 * r:])
    torch.cuda.synchronize()
    ctx.sync()
    for t, w in zip((o0, o1, offs), want):
        assert np.array_equal(to_np(t), w)
    h, hn = to_np(draws).reshape(-1)[:rounds * 20 * count].reshape(rounds, -1), to_np(numbers).view(np.uint32)
    for r in range(rounds):
        assert hn[r] == total, r
        assert np.array_equal(h[r, :20 * total], records), r
    ctx.close()
