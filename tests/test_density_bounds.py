"""The two properties of Perlin's noise that let the density generator skip samples
(dens_bounds in csrc/vox_device.cuh), from the formulas: the largest magnitude of a value and of
a second derivative along an axis, over every choice of the corner gradients. The gradient set
and the formulas are symmetric in the axes, so one axis stands for the three.
"""
import itertools

import numpy as np

GRADS = np.array([g for g in itertools.product((-1, 0, 1), repeat=3) if np.abs(g).sum() == 2], float)


def fade(t):
    return t * t * t * (t * (t * 6 - 15) + 10)


def test_largest_value_and_curvature():
    steps = 100
    g = np.linspace(0.0, 1.0, steps + 1)
    y, z = np.meshgrid(g, g, indexing="ij")
    value = curve = 0.0
    for x in g:
        u, u1, u2 = fade(x), 30 * x**2 * (1 - x) ** 2, 60 * x * (1 - x) * (1 - 2 * x)
        val, cur = np.zeros_like(y), np.zeros_like(y)
        for b, c in itertools.product((0, 1), repeat=2):
            w = (fade(y) if b else 1 - fade(y)) * (fade(z) if c else 1 - fade(z))
            near, far = (np.stack([gx * (x - a) + gy * (y - b) + gz * (z - c) for gx, gy, gz in GRADS])
                         for a in (0, 1))
            # a value is the weighted sum of the corners' dot products
            val += w * ((1 - u) * np.abs(near).max(0) + u * np.abs(far).max(0))
            # n'' = u'' (B - A) + 2 u' (B' - A'), A and B the near and far columns; the choices
            # at their corners are independent
            slope = 2 * u1 * GRADS[:, 0, None, None]
            ta, tb = u2 * near + slope, u2 * far + slope
            cur += w * np.maximum(tb.max(0) - ta.min(0), ta.max(0) - tb.min(0))
        value, curve = max(value, val.max()), max(curve, cur.max())
    assert curve < 12.1  # the generator counts with 13
    # between grid points, for one choice of gradients, a value exceeds its trilinear
    # interpolation by at most 3 axes * 13 / 8 * step^2; the generator counts with 1.037
    assert value + 3 * 13.0 / 8 / steps**2 < 1.037
