"""Closest and any hit at ray counts around the resident warps and lanes of a launch, where the rays a
warp holds change from one to a full warp: a ray's answer is its own, whatever the launch."""

import numpy as np
import pytest

import scenes

# 148 SMs x 8 blocks x 4 warps hold a ray each, and 32 times as many rays fill them
WARPS = 148 * 8 * 4


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 33, WARPS - 1, WARPS, WARPS + 1, 2 * WARPS + 7, 31 * WARPS + 5, 32 * WARPS, 32 * WARPS + 1])
def test_hits_do_not_depend_on_the_launch(gpu_lib, n):
    import photon_gpu

    tris = np.concatenate([g.tris for g in scenes.slit_room(num_boxes=300).groups])
    rng = np.random.default_rng(7)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.uniform(0.2, 3.8, (n, 3))
    d = rng.normal(size=(n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = rng.uniform(0.5, 20.0, n)
    with photon_gpu.Geometry(tris) as g:
        whole = g.closest(rays)
        occluded = g.occluded(rays)
        some = np.unique(np.concatenate([[0, n - 1], rng.integers(0, n, 64)]))
        for i in some:   # one ray per launch
            one = g.closest(rays[i:i + 1])
            for a, b in zip(whole, one):
                np.testing.assert_array_equal(a[i:i + 1], b)
            assert occluded[i] == g.occluded(rays[i:i + 1])[0] == (one[0][0] >= 0)
