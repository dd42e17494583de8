"""Density chunks whose samples are decided cell by cell without evaluating them
(gen_density): chunk layers from far below to far above the surface, halo planes at the rims,
noise that rarely and that nearly always decides a cell, the inverted rule, a height term that
vanishes or falls, and coordinates beyond the limits of the bounds. Byte for byte against the
oracle, which evaluates every sample.
"""
import numpy as np
import pytest

from gpu_util import gpu_gen_mesh, gpu_generate

pytestmark = pytest.mark.gpu

CASES = {
    "caves": dict(octaves=3, frequency=1 / 96, y_ref=256.0, y_scale=1 / 64),
    "smooth": dict(octaves=2, frequency=1 / 300, y_ref=20.0, y_scale=1 / 32, solid_below_zero=1),
    "fine": dict(octaves=4, frequency=1 / 40, y_ref=40.0, y_scale=1 / 16),
    "flat": dict(octaves=2, frequency=1 / 80, y_ref=0.0, y_scale=0.0),
    "falling": dict(octaves=3, frequency=1 / 128, gain=-0.7, y_ref=100.0, y_scale=-1 / 50),
    "uneven": dict(octaves=3, frequency=0.05, lacunarity=0.5, gain=2.5, solid_below_zero=1),
}


def layers(n, cfg):
    """Chunks over the heights where the density can change sign, and one far off."""
    mid = int(cfg.gen.y_ref) // n
    step = max(1, 48 // n)
    out = [(3 * i - 4, mid + step * i, 5 - 2 * i) for i in range(-3, 4)]
    return out + [(-70000 // n, mid, 70000 // n), (20_000_000 // n, mid, -3), (1, mid + 4000 // n, 1)]


@pytest.mark.parametrize("n", [8, 16, 32, 64])
@pytest.mark.parametrize("name", sorted(CASES))
def test_cells_match_oracle(vox, oracle, n, name):
    kw = dict(kind=vox.GEN_DENSITY, seed=31 + n, chunk_size=n, cull_mode=vox.CULL_FULL6, **CASES[name])
    cfg = vox.make_config(**kw)
    coords = layers(n, cfg)
    got = gpu_generate(vox, cfg, coords)
    for i, c in enumerate(coords):
        assert np.array_equal(got[i], oracle.cubes_to_occ(n, oracle.generate_cubes(cfg, c, i))), c
    rng = np.random.default_rng(n)
    masks = [63] + [int(v) for v in rng.integers(0, 64, len(coords) - 1)]
    w0, w1, woffs = oracle.gen_mesh_batch(cfg, coords, masks)
    g0, g1, offs, _ = gpu_gen_mesh(vox, cfg, coords, masks, cap=max(int(woffs[-1]), 1))
    assert np.array_equal(offs, woffs)
    assert np.array_equal(g0, w0) and np.array_equal(g1, w1)
