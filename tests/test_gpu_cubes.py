"""Cube/occupancy conversions at the edges of their wide accesses: every chunk size, counts
that end inside a thread block's units, and cube buffers off the 16-byte alignment."""
import numpy as np
import pytest

from gpu_util import ctx_for, to_dev, to_np, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 16, 32, 64])
@pytest.mark.parametrize("count", [1, 3, 33])
@pytest.mark.parametrize("offset", [0, 1, 8])
def test_conversions_match_numpy(vox, n, count, offset):
    torch = torch_cuda()
    rng = np.random.default_rng(n * 100 + count * 10 + offset)
    cubes = rng.choice(np.array([0, 1, 2, 3, 130, 255], np.uint8), size=count * n ** 3)
    solid = cubes != 2
    words = max(1, n // 32)
    bits = np.packbits(solid.reshape(-1, min(n, 32)), axis=1, bitorder="little")
    want = np.zeros((count * n * n * words, 4), np.uint8)
    want[:, :bits.shape[1]] = bits
    ctx = ctx_for(vox, vox.make_config(chunk_size=n))
    buf = to_dev(np.full(cubes.size + 32, 7, np.uint8))
    buf[offset:offset + cubes.size] = to_dev(cubes)
    occ = to_dev(np.zeros(want.shape[0] + 4, np.uint32))
    torch.cuda.synchronize()
    ctx.cubes_to_occ(buf.data_ptr() + offset, count, occ)
    ctx.sync()
    got = to_np(occ).view(np.uint32)
    assert np.array_equal(got[:want.shape[0]], want.reshape(-1).view(np.uint32))
    assert not got[want.shape[0]:].any()
    back = to_dev(np.full(cubes.size + 32, 7, np.uint8))
    ctx.occ_to_cubes(occ, count, back.data_ptr() + offset)
    ctx.sync()
    out = to_np(back)
    assert np.array_equal(out[offset:offset + cubes.size], np.where(solid, 0, 2))
    assert (out[:offset] == 7).all() and (out[offset + cubes.size:] == 7).all()
    ctx.close()
