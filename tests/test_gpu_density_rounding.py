"""Density samples that a single rounding decides: at each place the exact FP32 evaluation is an
ulp or two from zero, and one with a fused multiply-add in the packed interpolation has the
other sign. Occupancy and meshes against the oracle, for every chunk size.
"""
import numpy as np
import pytest

from gpu_util import gpu_gen_mesh, gpu_generate

pytestmark = pytest.mark.gpu

PLACES = [(326384298, (78890, 280, -39472)), (200995867, (-110689, 252, -80702)), (360881139, (102240, 260, 79541)),
          (1060197637, (94361, 249, 101599)), (173047027, (94149, 243, -57851))]


@pytest.mark.parametrize("n", [8, 16, 32, 64])
@pytest.mark.parametrize("seed,place", PLACES)
def test_samples_next_to_zero(vox, oracle, n, seed, place):
    cfg = vox.make_config(chunk_size=n, kind=vox.GEN_DENSITY, seed=1 + seed % 1000003, octaves=3, frequency=1 / 96,
                          lacunarity=2.0, gain=0.5, y_ref=256.0, y_scale=1 / 64, cull_mode=vox.CULL_FULL6)
    # the chunk of the place, and the ones whose lateral halo planes hold it
    chunks = [tuple((v + d) // n for v, d in zip(place, step))
              for step in ((0, 0, 0), (n, 0, 0), (-n, 0, 0), (0, 0, n), (0, 0, -n))]
    got = gpu_generate(vox, cfg, chunks)
    for i, c in enumerate(chunks):
        assert np.array_equal(got[i], oracle.cubes_to_occ(n, oracle.generate_cubes(cfg, c, i))), c
    w0, w1, woffs = oracle.gen_mesh_batch(cfg, chunks, [63] * len(chunks))
    g0, g1, offs, _ = gpu_gen_mesh(vox, cfg, chunks, [63] * len(chunks), cap=max(int(woffs[-1]), 1))
    assert np.array_equal(offs, woffs) and np.array_equal(g0, w0) and np.array_equal(g1, w1)
