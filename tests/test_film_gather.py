"""The 4 x 4 films of renders at sizes where the tiled gather of the samples can go wrong.

Every pixel's (R, G, B, W) sums of a render against an FP64 restatement: the samples' raster
positions from the renderer's counter-based draws (one cell of the sample window per pixel index),
the filters of HdrRgbFilm::addRgbSample (HdrRgbFilm.cpp:82-123, SampleFilter.cpp:12-59), and a camera
that sees nothing but a constant environment, whose radiance the samples carry up to the rounding of
the environment's bilinear lookup (4 products and 3 sums in FP32). The GPU
evaluates the weights in FP32: an axis factor is within 3e-7 of its FP64 value (the Blackman-Harris
window's cosines of rounded arguments up to 6 pi), a weight within 1e-6, and at most 25 samples per
sample index reach a pixel.
"""

import numpy as np
import pytest

import scenes
from test_film_reference_cases import FILTERS, HALF

NAMES = {"gaussian": "gaussian", "mn": "mitchell-netravali", "bh": "blackman-harris"}
RADIANCE = (0.25, 1.0, 4.0)


def _mix64(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _raster(width, height, spp, seed, first_sample):
    """Raster positions [spp, height, width, 2] float32 of the samples (regen_kernel's draws)."""
    with np.errstate(over="ignore"):
        path = np.arange(width * height * spp, dtype=np.uint64) + np.uint64(first_sample * width * height)
        base = _mix64(path ^ _mix64(np.array([seed], np.uint64)))
        u = [(_mix64(base + np.uint64(dim) * np.uint64(0xD1B54A32D192ED03)) >> np.uint64(40)).astype(np.float32)
             * np.float32(1.0 / 16777216.0) for dim in (0, 1)]
    out = np.empty((spp, height, width, 2), np.float32)
    for a, size in enumerate((width, height)):
        cell = np.arange(width if a == 0 else height, dtype=np.float32)
        cell = cell[None, None, :] if a == 0 else cell[None, :, None]
        scale = np.float32((size - 1.0 + 2.0 * HALF) / size)
        out[..., a] = np.float32(0.5 - HALF) + (cell + u[a].reshape(spp, height, width)) * scale
    return out


def _weights(name, width, height, raster):
    """FP64 sum of the filter weights that reach each pixel."""
    pad = 3
    w = np.zeros((height + 2 * pad, width + 2 * pad))
    c = raster.reshape(-1, 2).astype(np.float64) - 0.5
    first = np.ceil(c - HALF).astype(np.int64)
    for dy in range(5):
        for dx in range(5):
            p = first + (dx, dy)
            d = p - c
            f = np.where((np.abs(d) <= HALF).all(1), FILTERS[NAMES[name]](d[:, 0], d[:, 1]), 0.0)
            inside = (p[:, 0] >= -pad) & (p[:, 0] < width + pad) & (p[:, 1] >= -pad) & (p[:, 1] < height + pad)
            np.add.at(w, (p[inside, 1] + pad, p[inside, 0] + pad), f[inside])
    return w[pad:-pad, pad:-pad]


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(NAMES))
@pytest.mark.parametrize("width,height,spp", [(1, 1, 3), (2, 17, 5), (31, 15, 2), (32, 16, 4), (33, 17, 1), (100, 1, 9),
                                              (64, 63, 3), (257, 130, 2)])
def test_gathered_film_matches_restatement(gpu_lib, name, width, height, spp):
    import photon_gpu

    behind = np.array([[[0.0, 0.0, -5.0], [0.1, 0.0, -5.0], [0.0, 0.1, -5.0]]], np.float32)
    scene = scenes.Scene("sky", width, height, spp, 1, cam_pos=(0.0, 0.0, 0.0), cam_dir=(0.0, 0.0, 1.0),
                         cam_up=(0.0, 1.0, 0.0), fov_deg=40.0, env_radiance=RADIANCE,
                         groups=[scenes.MeshGroup(behind, scenes.Material("matte"))])
    with photon_gpu.RenderScene(scene) as rs:
        rs.set_filter(name)
        rs.render(spp, max_bounces=1, seed=9)
        rs.render(2, max_bounces=1, seed=9, first_sample=spp)   # a second pass adds to the film
        sums = rs.film()[1]
    want = (_weights(name, width, height, _raster(width, height, spp, 9, 0))
            + _weights(name, width, height, _raster(width, height, 2, 9, spp)))
    np.testing.assert_allclose(sums[..., 3], want, rtol=0, atol=1e-6 * 25 * (spp + 2))
    # the radiances are powers of two: the channels are the same sums up to the order of the additions
    for k in (0, 2):
        np.testing.assert_allclose(sums[..., k] / RADIANCE[k], sums[..., 1], rtol=1e-12, atol=1e-12)
    if name != "mn":   # (weights of both signs)
        np.testing.assert_allclose(sums[..., 1], sums[..., 3], rtol=7 * 2.0 ** -24)
