"""Renders as two wavefronts beyond the single-scene default: several scenes with the wavefronts' boundary
inside one of them, the other estimators, the refine modes, and previews while both run."""

import dataclasses
import threading
import time

import numpy as np
import pytest

import scenes
from test_progressive import _engine


@pytest.mark.gpu
@pytest.mark.parametrize("estimator", ["bvpt", "bvptdl"])
@pytest.mark.parametrize("sample_filter", ["box", "mn"])
def test_estimators_give_one_wavefronts_film(gpu_lib, estimator, sample_filter):
    import photon_gpu

    est = {"bvpt": photon_gpu.BVPT, "bvptdl": photon_gpu.BVPTDL}[estimator]
    films, rays = [], []
    for capacity in (1024, 1 << 20):
        with photon_gpu.RenderScene(scenes.cornell_glossy(45, 23, 5, 8)) as rs:
            rs.set_launch(capacity=capacity)
            rs.set_filter(sample_filter)
            r = rs.render(5, max_bounces=8, seed=31, estimator=est)
            films.append(rs.film()[1])
            rays.append((r["rays"], r["shadow_rays"]))
    assert rays[0] == rays[1]
    # the same paths; the FP64 film adds them up in another order
    np.testing.assert_allclose(films[0], films[1], rtol=1e-11, atol=1e-11 * np.abs(films[1]).max())


@pytest.mark.gpu
@pytest.mark.parametrize("spp", [(3, 5, 1), (1, 1, 4), (40, 1, 1)])
def test_several_scenes_give_one_wavefronts_films(gpu_lib, spp):
    import photon_gpu

    sc = [scenes.cornell(33, 31, 1, 8), scenes.cornell_glossy(40, 40, 1, 8),
          dataclasses.replace(scenes.batch_scene(0), width=48, height=30)]
    sc[1].env_image = None
    sc[1].env_radiance = (0.5, 0.6, 0.7)
    films = []
    for capacity in (1024, 1 << 20):
        rss = [photon_gpu.RenderScene(s) for s in sc]
        try:
            rss[0].set_launch(capacity=capacity)   # (the first scene's pool serves all)
            photon_gpu.render_scenes_wavefront(rss, list(spp), max_bounces=8, seed=33)
            films.append([rs.film()[1] for rs in rss])
        finally:
            for rs in rss:
                rs.close()
    for a, b in zip(*films):
        assert np.array_equal(a[..., 3], b[..., 3])
        np.testing.assert_allclose(a, b, rtol=1e-11, atol=1e-11 * np.abs(b).max())


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["manual", "empirical", "iterative"])
def test_refine_modes_give_one_wavefronts_film(gpu_lib, tmp_path, mode):
    """2^22 paths are two pools of the default size: one call against two calls of half the samples."""
    frames = []
    for calls, spp in ((1, 64), (2, 32)):
        path = tmp_path / str(calls)
        path.mkdir()
        eng = _engine(path, scenes.cornell(256, 256, spp, 5))
        eng.set_surface_refine(mode)
        for _ in range(calls):
            eng.render()
        frames.append(eng.frame())
        eng.close()
    # float32 frames of FP64 sums that differ by the order of 64 additions
    np.testing.assert_allclose(frames[0], frames[1], rtol=2.0 ** -23, atol=0)


@pytest.mark.gpu
def test_previews_of_two_wavefronts_weigh_every_pixel(gpu_lib, tmp_path):
    """A matte ground under a constant sky, BVPT: every path that sees the ground brings its albedo, every
    other one the sky's radiance, so a pixel that sees one of them has the same value whatever samples have
    finished -- if its W counts exactly those. One sample too many or too few would be 1/256 of W at most
    256 samples in; the values' own FP32 arithmetic is below 1e-5."""
    import photon_gpu

    ground = np.array([[[-900.0, 0.0, -900.0], [-900.0, 0.0, 900.0], [900.0, 0.0, 900.0]],
                       [[-900.0, 0.0, -900.0], [900.0, 0.0, 900.0], [900.0, 0.0, -900.0]]], np.float32)
    scene = scenes.Scene("ground", 256, 256, 512, 3, cam_pos=(0.0, 3.0, 0.0), cam_dir=(0.0, 0.0, 1.0),
                         cam_up=(0.0, 1.0, 0.0), fov_deg=60.0, env_radiance=(1.0, 1.0, 1.0), estimator="bvpt",
                         groups=[scenes.MeshGroup(ground, scenes.Material("matte", albedo=(0.5, 0.25, 0.75)))])
    eng = _engine(tmp_path, scene)
    eng.render()   # (the graphs are built)
    previews, stop = [], threading.Event()

    def poller():
        while not stop.is_set():
            r = eng.poll_region()
            if r is not None and r[4] == photon_gpu.REGION_UPDATING:
                previews.append(eng.peek())
            else:
                time.sleep(0.0001)

    eng.poll_regions(256)
    eng.clear_film()
    t = threading.Thread(target=poller)
    t.start()
    try:
        eng.render()
    finally:
        stop.set()
        t.join()
    final = eng.frame()
    eng.close()
    ground_px = np.all(np.abs(final - (0.5, 0.25, 0.75)) < 1e-4, axis=2)
    sky_px = np.all(np.abs(final - 1.0) < 1e-4, axis=2)
    assert ground_px.sum() > 20000 and sky_px.sum() > 20000
    assert previews and any(not np.array_equal(p, final) for p in previews)
    for p in previews:
        np.testing.assert_allclose(p[ground_px], np.broadcast_to((0.5, 0.25, 0.75), final.shape)[ground_px], rtol=1e-4)
        np.testing.assert_allclose(p[sky_px], 1.0, rtol=1e-4)
