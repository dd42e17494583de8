"""Launches that may begin before the one ahead of them has ended (vox_mesh, vox_frustum_cull,
vox_draw_list) read what that one writes: producers and consumers queued back to back, with other data
each round, without a wait in between, against the oracle.
"""
import numpy as np
import pytest

from gpu_util import ctx_for, dev_bytes, to_dev, to_np

pytestmark = pytest.mark.gpu

ROUNDS = 200


@pytest.mark.parametrize("n,pool", [(16, 3000), (32, 1500), (64, 200)])
def test_mesh_of_occupancy_just_packed(vox, oracle, n, pool):
    """vox_cubes_to_occ of a pool whose last chunk changes every round, then vox_mesh of that chunk,
    with the one before it as a neighbour."""
    cfg = vox.make_config(chunk_size=n, kind=vox.GEN_HEIGHTMAP, octaves=3, frequency=1 / 24,
                          amplitude=0.7 * n, base_height=n / 2.0, seed=11)
    kinds = 5
    cubes = [oracle.generate_cubes(cfg, (3 * k, 0, -k), 0) for k in range(kinds)]
    want = [oracle.mesh_chunk(cfg, (1, 2, 3), cubes[k], [cubes[(k + 1) % kinds]] + [None] * 5) for k in range(kinds)]
    per = n ** 3
    ctx = ctx_for(vox, cfg)
    words = ctx.sizes.occ_words_per_chunk
    ring = [dev_bytes(pool * per, fill=2) for _ in range(kinds)]
    for k in range(kinds):
        ring[k][(pool - 2) * per:(pool - 1) * per] = to_dev(cubes[(k + 1) % kinds])
        ring[k][(pool - 1) * per:pool * per] = to_dev(cubes[k])
    occ = dev_bytes(pool * words * 4, fill=0xEE)
    last, side = (occ[(pool - i) * words * 4:(pool - i + 1) * words * 4] for i in (1, 2))
    room = max(w[2] for w in want)
    stride0, stride1 = (room * 96 + 15) // 16 * 16, (room * 24 + 15) // 16 * 16
    rounds = min(ROUNDS, (1 << 30) // stride0)
    o0, o1 = dev_bytes(rounds * stride0, fill=5), dev_bytes(rounds * stride1, fill=5)
    counts = to_dev(np.zeros(rounds, np.uint64))
    to_np(counts)  # waits: everything above is in place
    for r in range(rounds):
        ctx.cubes_to_occ(ring[r % kinds], pool, occ)
        ctx.mesh(last, [side] + [None] * 5, (1, 2, 3), o0[r * stride0:], o1[r * stride1:], room, counts[r:])
    ctx.sync()
    h0, h1, hc = to_np(o0), to_np(o1), to_np(counts)
    for r in range(rounds):
        w0, w1, faces = want[r % kinds]
        assert int(hc[r]) == faces, r
        assert np.array_equal(h0[r * stride0:r * stride0 + faces * 96], w0), r
        assert np.array_equal(h1[r * stride1:r * stride1 + faces * 24], w1), r
    ctx.close()


@pytest.mark.parametrize("cull_first", [False, True])
@pytest.mark.parametrize("count", [100, 700, 3000])
def test_draw_list_of_a_batch_just_issued(vox, oracle, count, cull_first):
    """A batch, the frustum test of its coordinates and the draw list on its face offsets; the batches
    of two generations of coordinates take turns in the same buffers."""
    torch = pytest.importorskip("torch")
    cfg = vox.make_config(chunk_size=16, kind=vox.GEN_HEIGHTMAP, octaves=2, frequency=1 / 40, amplitude=20.0,
                          base_height=8.0, seed=3)
    side = int(np.ceil(np.sqrt(count)))
    sets = [np.array([(x + dx, y, z - 9) for z in range(side) for x in range(side)], np.int32)[:count]
            for dx, y in ((-side // 2, 0), (400, 1))]
    planes = vox.frustum_planes(vox.camera_matrix((8.0, 30.0, -4.0), (0.7, -0.2, 0.6)))
    wide = np.array([0, 0, 0, 1] * 6, np.float32)  # every corner is inside: d = 1
    ctx = ctx_for(vox, cfg)
    given = [to_dev(c) for c in sets]
    coords, offs = to_dev(sets[0]), to_dev(np.zeros(count + 1, np.uint64))
    faces = [oracle.gen_mesh_digests(cfg, c, [0] * count, counts_only=True)[0] for c in sets]
    room = int(max(f.sum() for f in faces))
    masks = to_dev(np.zeros(count, np.uint8))
    o0, o1 = dev_bytes(room * 96), dev_bytes(room * 24)
    draws = torch.full((ROUNDS, count, 5), -7, dtype=torch.int32, device="cuda")
    numbers = torch.full((ROUNDS,), -7, dtype=torch.int32, device="cuda")
    visible = torch.full((ROUNDS, count), 9, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for r in range(ROUNDS):
        pl = wide if r % 3 else planes
        coords.copy_(given[r % 2])  # in stream order, ahead of the batch
        ctx.gen_mesh_batch(coords, masks, count, o0, o1, room, offs)
        if cull_first:
            ctx.frustum_cull(pl, coords, count, visible[r])
        ctx.draw_list(pl, coords, offs, count, draws[r], numbers[r:])
    ctx.sync()
    h, hn, hv = draws.cpu().numpy(), numbers.cpu().numpy(), visible.cpu().numpy()
    seen = [np.array([oracle.frustum_contains(planes, tuple(int(v) for v in c), 16) for c in s]) for s in sets]
    for r in range(ROUNDS):
        f = faces[r % 2].astype(np.int64)
        start = np.concatenate([[0], np.cumsum(f)])
        vis = np.ones(count, bool) if r % 3 else seen[r % 2]
        if cull_first:
            assert np.array_equal(hv[r] == 1, vis), r
        at = np.flatnonzero(vis & (f > 0))
        rec = np.stack([6 * f[at], np.ones_like(at), 6 * start[at], 4 * start[at], np.zeros_like(at)], 1)
        assert hn[r] == len(at), r
        assert np.array_equal(h[r, :len(at)], rec), r
        assert (h[r, len(at):] == -7).all(), r
    ctx.close()
