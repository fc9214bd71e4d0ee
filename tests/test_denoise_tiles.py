"""The a-trous filter at the edges of its tiles (16 x 16 lattice points, two rows a thread), against the FP64 oracle;
the display bytes whose FP32 estimate lies next to a step, against FP64."""
import os
import sys

import numpy as np
import pytest

import mypbr_gb300 as mp

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import oracle as orc  # noqa: E402
import post_oracle  # noqa: E402


# one pixel, one short of and past a tile's rows and columns, odd heights (a thread's second row outside)
@pytest.mark.gpu
@pytest.mark.parametrize("width,height", [(1, 1), (3, 1), (1, 3), (15, 16), (16, 17), (17, 15), (33, 31), (70, 129)])
def test_gpu_denoiser_matches_oracle_at_tile_edges(width, height):
    rng = np.random.default_rng(width * 1000 + height)
    alb = rng.uniform(0.1, 0.9, (height, width, 3))
    nrm = rng.normal(size=(height, width, 3)) * 0.05 + np.array([0.0, 0.0, 1.0])
    nrm /= np.linalg.norm(nrm, axis=2, keepdims=True)
    rad = alb * rng.uniform(0.5, 1.5, (height, width, 1))
    var = np.full((height, width), 0.05)
    out = np.empty_like(rad)
    mp.denoise(rad, alb, nrm, var, width, height, out)
    want = orc.denoise(rad, alb, nrm, var)
    # five FP32 iterations of 25 weighted taps: each weight carries a few 2^-24 of relative error times its
    # exponent (at most about 10 where it counts), each sum 25 roundings: 5 x (10 x 4 + 25) x 2^-24 = 2e-5
    assert np.all(np.abs(out - want) <= 2e-5 * np.abs(want) + 1e-9)


@pytest.mark.gpu
def test_display_bytes_next_to_every_step():
    """Values within 1e-3 to 1e-12 of the 256 steps of the sRGB curve, and far from them."""
    steps = np.arange(1, 256) / 256.0
    at = np.where(steps <= 0.04045, steps / 12.92, ((steps + 0.055) / 1.055) ** 2.4)
    values = [at * (1.0 + sign * eps) for eps in (1e-3, 3e-5, 1e-5, 1e-6, 1e-8, 1e-12) for sign in (-1, 1)]
    values += [np.linspace(0.0, 1.2, 255), np.array([0.0, -1.0, 0.0031308, 0.0031309, 0.998, 0.999, 1.0, 50.0])]
    flat = np.concatenate([np.ravel(v) for v in values])
    flat = np.concatenate([flat, np.zeros(-len(flat) % 3)])
    frame = flat.reshape(1, -1, 3)
    _, rgb = mp.display(frame, mp.display_opts())
    assert np.array_equal(rgb, post_oracle.to_byte(frame))
