"""The 4 x 4 films around 65,536 pixels a side, up to which the film gathers its samples by tile and beyond
which it splats them: W sums against the FP64 restatement of test_film_gather.py, with its bound."""

import numpy as np
import pytest

import scenes
from test_film_gather import NAMES, RADIANCE, _raster, _weights


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(NAMES))
@pytest.mark.parametrize("width,height", [(65536, 1), (1, 65536), (65519, 17), (65537, 1), (2, 65537), (65569, 16)])
def test_wide_and_high_films_match_restatement(gpu_lib, name, width, height):
    import photon_gpu

    behind = np.array([[[0.0, 0.0, -5.0], [0.1, 0.0, -5.0], [0.0, 0.1, -5.0]]], np.float32)
    scene = scenes.Scene("sky", width, height, 2, 1, cam_pos=(0.0, 0.0, 0.0), cam_dir=(0.0, 0.0, 1.0),
                         cam_up=(0.0, 1.0, 0.0), fov_deg=40.0, env_radiance=RADIANCE,
                         groups=[scenes.MeshGroup(behind, scenes.Material("matte"))])
    with photon_gpu.RenderScene(scene) as rs:
        rs.set_filter(name)
        rs.render(2, max_bounces=1, seed=9)
        sums = rs.film()[1]
    want = _weights(name, width, height, _raster(width, height, 2, 9, 0))
    np.testing.assert_allclose(sums[..., 3], want, rtol=0, atol=1e-6 * 25 * 2)
    for k in (0, 2):   # powers of two: the same sums up to the order of the additions
        np.testing.assert_allclose(sums[..., k] / RADIANCE[k], sums[..., 1], rtol=1e-12, atol=1e-12)
