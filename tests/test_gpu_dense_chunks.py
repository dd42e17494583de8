"""Chunks with more faces than a face list takes, in batches of more parts than the GPU has warps: the
runs of such chunks are shared among warps. Mixed with listed and empty chunks, in one launch and in
slabs, with an output that ends inside a chunk, repeated without a wait, and replayed from a graph;
byte for byte against the look-back schedule (another kernel, checked against the oracle).
"""
import numpy as np
import pytest

from gpu_util import ctx_for, dev_bytes, to_dev
from test_gpu_face_lists import chunk

pytestmark = pytest.mark.gpu

# isolated voxels (6 faces each): the most that are listed (9 N^2 faces at 16^3, else what a slot holds;
# an 8^3 chunk has room for 64, which are always listed)
LISTED = {8: 53, 16: 384, 32: 1144, 64: 5461}


def outputs(ctx, count, cap):
    import torch
    b1 = ctx.sizes.bytes_per_face_out1
    return (torch.zeros(count + 1, dtype=torch.int64, device="cuda"),
            dev_bytes(cap * ctx.sizes.bytes_per_face_out0 + 64, fill=0xAB), dev_bytes(cap * b1 + 64, fill=0xCD))


def same(got, want):
    import torch
    torch.cuda.synchronize()
    return all(torch.equal(g, w) for g, w in zip(got, want))


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("n,count", [(8, 3), (8, 9000), (16, 1300), (32, 230), (64, 1), (64, 20)])
def test_dense_chunks_match_lookback(vox, n, layout, count):
    import torch
    rng = np.random.default_rng(n + count)
    kinds = ["random", LISTED[n], LISTED[n] + 1, "random", "slab", "empty", "random", "full"]
    ctx = ctx_for(vox, vox.make_config(chunk_size=n, layout=layout))
    pool = to_dev(np.zeros((len(kinds), ctx.sizes.occ_words_per_chunk), np.uint32))
    ctx.cubes_to_occ(to_dev(np.concatenate([chunk(k, n, rng) for k in kinds])), len(kinds), pool)
    slots = to_dev(rng.integers(0, len(kinds), count).astype(np.int32) if count > 1 else np.zeros(1, np.int32))
    nbrs = to_dev(rng.integers(-1, len(kinds), (count, 6)).astype(np.int32))
    coords = to_dev(rng.integers(-999, 999, (count, 3)).astype(np.int32))
    d = ctx.tuning()

    def mesh(schedule, cap, out, slab=0):
        ctx.set_tuning(d.threads, d.stage_faces, 0, schedule, slab)
        ctx.mesh_batch(pool, len(kinds), slots, nbrs, coords, count, out[1],
                       out[2] if layout == 0 else None, cap, out[0])

    offs = torch.zeros(count + 1, dtype=torch.int64, device="cuda")
    mesh(vox.SCHEDULE_LOOKBACK, 1, (offs, dev_bytes(256), dev_bytes(256)))
    ctx.sync(raise_on_error=False)
    total = int(offs[count])
    for cap in (total, total - total // 3):
        want = outputs(ctx, count, cap)
        mesh(vox.SCHEDULE_LOOKBACK, cap, want)
        status = ctx.sync(raise_on_error=False)
        assert status == (vox.VOX_OK if cap == total else vox.VOX_ERR_CAPACITY)
        for slab in (0, max(1, count // 3)):
            got = [outputs(ctx, count, cap) for _ in range(3)]
            torch.cuda.synchronize()
            for out in got:
                mesh(vox.SCHEDULE_OVERLAP, cap, out, slab)
            assert ctx.sync(raise_on_error=False) == status
            assert all(same(out, want) for out in got), (cap, slab)
            del got
    ctx.close()


@pytest.mark.parametrize("layout", [0, 1])
def test_dense_chunks_of_a_replayed_graph(vox, layout):
    import torch
    n, count = 16, 1100
    cfg = vox.make_config(chunk_size=n, layout=layout, kind=vox.GEN_DENSITY, octaves=1, frequency=0.61,
                          y_ref=0.0, y_scale=1 / 200, seed=9)
    ctx = ctx_for(vox, cfg)
    # from dense noise (y around 0) over thinner to air
    coords = to_dev(np.array([(i % 11, (i // 11) % 20 - 6, i // 220) for i in range(count)], np.int32))
    cap = 16 * n * n * count
    want, got = outputs(ctx, count, cap), outputs(ctx, count, cap)
    d = ctx.tuning()
    ctx.set_tuning(d.threads, d.stage_faces, 0, vox.SCHEDULE_LOOKBACK)
    ctx.gen_mesh_batch(coords, None, count, want[1], want[2] if layout == 0 else None, cap, want[0])
    ctx.sync()
    ctx.set_tuning(d.threads, d.stage_faces, 0, vox.SCHEDULE_OVERLAP)
    graph = ctx.capture_graph(coords, None, count, got[1], got[2] if layout == 0 else None, cap, got[0])
    for _ in range(3):
        for t, fill in zip(got[1:], (0xAB, 0xCD)):
            t.fill_(fill)
        torch.cuda.synchronize()
        for _ in range(5):
            graph.launch()
        ctx.sync()
        assert same(got, want)
    del graph
    ctx.close()
