"""The face-list launches of the overlap schedule at their edges, byte for byte against the
look-back schedule (another kernel, checked against the oracle): face counts on both sides of a
list's capacity, chunks without faces, batches on both sides of an offset group (32 chunks), an
output that ends inside a chunk, origins on both sides of the exact float translation.
"""
import numpy as np
import pytest

from gpu_util import ctx_for, dev_bytes, to_dev, to_np

pytestmark = pytest.mark.gpu

# isolated voxels (6 faces each) that just fit a list of 32-bit codes
FITS = {8: 64, 16: 467, 32: 1144, 64: 5461}


def chunk(kind, n, rng):
    cubes = np.full((n, n, n), 2, np.uint8)  # [y][z][x]
    if kind == "full":
        cubes[:] = 0
    elif kind == "random":
        cubes[rng.random((n, n, n)) < 0.5] = 0
    elif kind == "slab":
        cubes[:n // 3] = 0
    elif kind != "empty":  # that many isolated voxels
        at = rng.permutation((n // 2) ** 3)[:kind]
        h = n // 2
        cubes[2 * (at // (h * h)), 2 * ((at // h) % h), 2 * (at % h)] = 0
    return cubes.reshape(-1)


def mesh(vox, ctx, schedule, pool, n, count, slots, nbrs, coords, cap):
    t = ctx.tuning()
    ctx.set_tuning(t.threads, t.stage_faces, 0, schedule)
    b0, b1 = ctx.sizes.bytes_per_face_out0, ctx.sizes.bytes_per_face_out1
    o0, o1 = dev_bytes(cap * b0 + 64, fill=0xAB), dev_bytes(cap * b1 + 64, fill=0xCD)
    offs = to_dev(np.zeros(count + 1, np.uint64))
    ctx.mesh_batch(pool, n, slots, nbrs, coords, count, o0, o1 if b1 else None, cap, offs)
    status = ctx.sync(raise_on_error=False)
    return status, to_np(offs), to_np(o0), to_np(o1)


@pytest.mark.parametrize("n", [8, 16, 32, 64])
@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("count", [1, 32, 45])
def test_lists_match_lookback(vox, n, layout, count):
    rng = np.random.default_rng(n + count)
    kinds = ["slab", FITS[n], FITS[n] + 1 if n > 8 else 40, "empty", "random", "full", 1]
    cfg = vox.make_config(chunk_size=n, layout=layout)
    ctx = ctx_for(vox, cfg)
    cubes = to_dev(np.concatenate([chunk(k, n, rng) for k in kinds]))
    pool = to_dev(np.zeros((len(kinds), ctx.sizes.occ_words_per_chunk), np.uint32))
    ctx.cubes_to_occ(cubes, len(kinds), pool)
    which = np.arange(count) % len(kinds) if count > 1 else np.array([4])
    slots = to_dev(which.astype(np.int32))
    nbrs = to_dev(rng.integers(-1, len(kinds), (count, 6)).astype(np.int32))
    near, far = (1 << 23) // n - 2, (1 << 24) // n + 3  # below and above 2^23 - 64 in size
    xyz = np.stack([np.full(count, near) + np.arange(count) % 4, -np.arange(count),
                    np.where(np.arange(count) % 5 == 0, -far, np.arange(count))], 1)
    coords = to_dev(xyz.astype(np.int32))
    args = (pool, len(kinds), count, slots, nbrs, coords)
    _, offs, _, _ = mesh(vox, ctx, vox.SCHEDULE_LOOKBACK, *args, 1)
    total = int(offs[-1])
    for cap in (total, total - 1 - total // 3):
        want = mesh(vox, ctx, vox.SCHEDULE_LOOKBACK, *args, cap)
        got = mesh(vox, ctx, vox.SCHEDULE_OVERLAP, *args, cap)
        assert got[0] == want[0] == (vox.VOX_OK if cap == total else vox.VOX_ERR_CAPACITY)
        for g, w in zip(got[1:], want[1:]):
            assert np.array_equal(g, w)
    ctx.close()
