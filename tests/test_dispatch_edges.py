"""Sizes at which a dispatch changes its path, each against the general path or the oracle.

* Host ray queries: results up to 256 KB come back through one page-locked copy, larger ones
  straight into the caller's arrays; a batch's answers are its rays' own, however it is cut.
* The guiding network's forward pass spreads tiles of 128 rows over teams and SMs: rows are
  independent, so a row's output does not depend on the batch around it.
* The tensor-core backward pass keeps several tiles' gradients per CTA beyond 128 x 148 samples:
  against the FP32 CUDA-core backward (the bar of test_guide.py).
* Scenes of matte surfaces shade in slot order, others by class lists: a Cornell box gives the same
  film when a conductor that no path can reach makes it shade by class.
* A scene's loop graph serves all its renders of one shape, and is built again for another: a
  scene that has rendered other things before gives the film of a fresh one.
"""

import dataclasses

import numpy as np
import pytest

import scenes
from oracle import guide_ref as ref


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.uniform(5.0, 550.0, (n, 3))
    d = rng.normal(size=(n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 7] = rng.uniform(10.0, 2000.0, n)
    return rays


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 13106, 13107, 13108, 65535, 65536])
def test_host_queries_do_not_depend_on_the_batch(gpu_lib, n):
    import photon_gpu

    tris = np.concatenate([g.tris for g in scenes.cornell().groups])
    rays = _rays(n, 3)
    with photon_gpu.Geometry(tris) as g:
        prim, t, bary = g.closest(rays)
        occluded = g.occluded(rays)
        for part in np.array_split(np.arange(n), max(1, n // 5000)):
            p, tt, b = g.closest(rays[part])
            np.testing.assert_array_equal(prim[part], p)
            np.testing.assert_array_equal(t[part], tt)
            np.testing.assert_array_equal(bary[part], b)
            np.testing.assert_array_equal(occluded[part], g.occluded(rays[part]))
    np.testing.assert_array_equal(occluded != 0, prim >= 0)


def _params(seed):
    rng = np.random.default_rng(seed)
    parts = ref.unpack(ref.init_params(seed, out_scale=1.0))
    for name in ("b0", "b1", "b2", "b3", "b4"):
        parts[name] = rng.normal(0.0, 0.1, parts[name].shape)
    return ref.pack(parts)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 128, 129, 128 * 148, 128 * 148 + 1, 128 * 148 * 3 + 130, 128 * 148 * 4 + 1, 150_001])
def test_forward_rows_do_not_depend_on_the_batch(gpu_lib, n):
    import photon_gpu

    params = _params(5)
    f = np.random.default_rng(n).random((n, 7), dtype=np.float32)
    raw = photon_gpu.guide_forward(params, f)
    mix = photon_gpu.guide_mixture(params, f)
    rows = np.unique(np.concatenate([np.arange(min(n, 300)), np.arange(max(0, n - 300), n),
                                     np.random.default_rng(1).integers(0, n, 500)]))
    np.testing.assert_array_equal(raw[rows], photon_gpu.guide_forward(params, f[rows]))
    np.testing.assert_array_equal(mix[rows], photon_gpu.guide_mixture(params, f[rows]))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 129, 128 * 148, 128 * 148 + 1, 60_007])
def test_backward_over_several_tiles_per_cta(gpu_lib, n):
    import photon_gpu

    params = _params(6)
    rng = np.random.default_rng(n)
    f = rng.random((n, 7), dtype=np.float32)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    w = rng.random(n) + 0.1
    loss_tc, g_tc = photon_gpu.guide_gradients(params, f, d, w)
    loss_cc, g_cc = photon_gpu.guide_gradients(params, f, d, w, cuda_cores=True)
    assert np.all(np.isfinite(g_tc))
    assert abs(loss_tc - loss_cc) <= 1e-5 * abs(loss_cc) + 1e-6
    o = 0
    for name, shape in ref.SHAPES:
        k = int(np.prod(shape))
        a, b = g_tc[o:o + k], g_cc[o:o + k]
        assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b), name
        o += k


@pytest.mark.gpu
@pytest.mark.parametrize("estimator", ["bneept", "bvpt"])
@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (33, 31, 3), (128, 96, 40)])
def test_slot_order_and_class_order_shade_the_same_film(gpu_lib, estimator, width, height, spp):
    import photon_gpu

    est = {"bneept": photon_gpu.BNEEPT, "bvpt": photon_gpu.BVPT}[estimator]
    plain = scenes.cornell(width, height, spp, 8)
    far = np.array([[[278.0, 273.0, -9e4], [279.0, 273.0, -9e4], [278.0, 274.0, -9e4]]], np.float32)
    classed = dataclasses.replace(plain, groups=plain.groups + [
        scenes.MeshGroup(far, scenes.Material("conductor", roughness=0.3, f0=(0.9, 0.9, 0.9)))])
    sums = []
    for sc in (plain, classed):
        with photon_gpu.RenderScene(sc) as rs:
            rs.render(spp, max_bounces=8, estimator=est, seed=11)
            sums.append(rs.film()[1])
    # the same paths; the FP64 film adds them up in another order (at most 1e5 additions of 2^-53 each)
    np.testing.assert_allclose(sums[0], sums[1], rtol=1e-11, atol=0)


@pytest.mark.gpu
def test_graph_reuse_gives_a_fresh_scenes_film(gpu_lib):
    import photon_gpu

    scene = scenes.cornell_glossy(48, 40, 8, 8)
    shapes = [dict(spp=8, max_bounces=8, seed=1), dict(spp=1, max_bounces=8, seed=2, first_sample=3),
              dict(spp=700, max_bounces=8, seed=3),   # a larger pool than before
              dict(spp=8, max_bounces=2, seed=4), dict(spp=8, max_bounces=8, seed=1, estimator=photon_gpu.BVPT),
              dict(spp=8, max_bounces=8, seed=1)]
    with photon_gpu.RenderScene(scene) as used:
        for shape in shapes:
            for sample_filter in ("box", "mn"):
                used.set_filter(sample_filter)   # (clears the film)
                used.render(**shape)
                with photon_gpu.RenderScene(scene) as fresh:
                    fresh.set_filter(sample_filter)
                    fresh.render(**shape)
                    want = fresh.film()[1]
                got = used.film()[1]
                np.testing.assert_allclose(got, want, rtol=1e-11, atol=1e-11 * np.abs(want).max())
        used.set_filter("box")
        used.profile(16, 8, seed=5)   # plain launches between graph launches
        used.render(**shapes[0])
        with photon_gpu.RenderScene(scene) as fresh:
            fresh.render(**shapes[0])
            np.testing.assert_allclose(used.film()[1], fresh.film()[1], rtol=1e-11, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("sample_filter", ["box", "bh"])
@pytest.mark.parametrize("width,height,spp", [(32, 32, 1), (32, 32, 2), (33, 31, 2), (45, 23, 5), (64, 33, 7)])
def test_two_wavefronts_give_one_wavefronts_film(gpu_lib, sample_filter, width, height, spp):
    """Renders of at least two pools of paths run as two wavefronts: pools of 1,024 paths (the smallest)
    against one that holds them all, and the ray counts."""
    import photon_gpu

    scene = scenes.cornell_glossy(width, height, spp, 8)
    films, rays = [], []
    for capacity in (1024, 1 << 20):
        with photon_gpu.RenderScene(scene) as rs:
            rs.set_launch(capacity=capacity)
            rs.set_filter(sample_filter)
            r = rs.render(spp, max_bounces=8, seed=21)
            films.append(rs.film()[1])
            rays.append((r["rays"], r["shadow_rays"]))
    assert rays[0] == rays[1]
    np.testing.assert_allclose(films[0], films[1], rtol=1e-11, atol=1e-11 * np.abs(films[1]).max())


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [1, 0])
@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (33, 31, 1), (45, 23, 3)])
def test_guided_vertices_do_not_depend_on_their_row(gpu_lib, width, height, spp, depth):
    """A guided vertex' row of the network is its place in the lists of its class: pools of 1,024 paths,
    whose queues mix vertices of several bounces, against one that holds all paths; the network is frozen."""
    import photon_gpu

    scene = scenes.cornell_glossy(width, height, spp, 8)
    films, guided = [], []
    for capacity in (1024, 1 << 20):
        with photon_gpu.RenderScene(scene) as rs:
            rs.set_launch(capacity=capacity)
            rs.set_guiding(True, False)
            rs.set_guiding_depth(depth)
            rs.render(spp, max_bounces=8, seed=23)
            films.append(rs.film()[1])
            guided.append(rs.guide_info()["guided_vertices"])
    assert guided[0] == guided[1]
    np.testing.assert_allclose(films[0], films[1], rtol=1e-11, atol=1e-11 * np.abs(films[1]).max())
