"""Cave voxels of 32^3 chunks that a single rounding decides (17 of the 8 * 10^8 voxels of 24,576
chunks of the layers around the surface): an evaluation that fuses a product of the packed
interpolation with its sum has the other sign at each of them. Generation and meshing apart: the
occupancy against the oracle's, meshes of the oracle's occupancy, and the fused batch. A world voxel
does not depend on the size of the chunk that holds it, so the other sizes have to agree too.
"""
import numpy as np
import pytest

from gpu_util import ctx_for, dev_bytes, gpu_gen_mesh, gpu_generate, to_dev, to_np

pytestmark = pytest.mark.gpu

PLACES = [(818235696, (-20094, 278, -33404)), (20032162, (38468, 264, -31349)), (20032162, (38662, 284, -31179)),
          (39371367, (-5990, 260, 60764)), (332966094, (-44320, 233, 30933)), (332966094, (-44114, 233, 31209)),
          (605238300, (46623, 276, 32508)), (313334186, (-49891, 240, 23712)), (313334186, (-49888, 240, 23712)),
          (313334186, (-49882, 240, 23712)), (313334186, (-49604, 247, 23979)), (30597843, (22198, 246, -3107)),
          (234782789, (22877, 282, 28798)), (898466117, (15171, 270, 47331)), (779959138, (32271, 227, -3653)),
          (779959138, (32260, 246, -3429)), (178225236, (62859, 258, 24027))]


def _config(vox, n, seed):
    return vox.make_config(chunk_size=n, kind=vox.GEN_DENSITY, seed=1 + seed % 1000003, octaves=3, frequency=1 / 96,
                           lacunarity=2.0, gain=0.5, y_ref=256.0, y_scale=1 / 64)


@pytest.mark.parametrize("seed,place", PLACES)
def test_surface_voxels_next_to_zero(vox, oracle, seed, place):
    n = 32
    cfg = _config(vox, n, seed)
    x, y, z = (v // n for v in place)
    # the chunk of the place and its lateral neighbours, in the order of vox_mesh's halo
    chunks = [(x, y, z), (x - 1, y, z), (x + 1, y, z), (x, y, z - 1), (x, y, z + 1)]
    cubes = [oracle.generate_cubes(cfg, c, 0) for c in chunks]
    occ = np.stack([oracle.cubes_to_occ(n, c) for c in cubes])
    assert np.array_equal(gpu_generate(vox, cfg, chunks), occ)

    w0, w1, faces = oracle.mesh_chunk(cfg, chunks[0], cubes[0], cubes[1:] + [None, None])
    ctx = ctx_for(vox, cfg)
    d_occ = to_dev(occ.view(np.int32))
    o0, o1, count = dev_bytes(faces * 96, fill=1), dev_bytes(faces * 24, fill=1), to_dev(np.zeros(1, np.uint64))
    ctx.mesh(d_occ[0], [d_occ[1], d_occ[2], d_occ[3], d_occ[4], None, None], chunks[0], o0, o1, faces, count)
    ctx.sync()
    assert int(to_np(count)[0]) == faces
    assert np.array_equal(to_np(o0, faces * 96), w0) and np.array_equal(to_np(o1, faces * 24), w1)
    ctx.close()

    b0, b1, boffs = oracle.gen_mesh_batch(cfg, chunks, [15] * 5)
    g0, g1, offs, _ = gpu_gen_mesh(vox, cfg, chunks, [15] * 5, cap=int(boffs[-1]))
    assert np.array_equal(offs, boffs) and np.array_equal(g0, b0) and np.array_equal(g1, b1)

    solid = int(occ[0][(place[1] % n) * n + place[2] % n] >> (place[0] % n)) & 1
    for m in (8, 16, 64):
        words = gpu_generate(vox, _config(vox, m, seed), [tuple(v // m for v in place)])[0]
        lx, ly, lz = (v % m for v in place)
        assert (int(words[(ly * m + lz) * max(1, m // 32) + lx // 32]) >> (lx % 32)) & 1 == solid, m
