"""Renders of one scene that differ from call to call: sample counts, depths, one or two wavefronts, guided
or not. A switch gives the film of a fresh scene, and costs no rebuilding of what the scene keeps."""

import statistics
import time

import numpy as np
import pytest

import scenes


def _render(rs, shape):
    import photon_gpu

    rs.set_guiding(shape.get("guided", False), False)   # (the network stays as initialised)
    rs.set_guiding_depth(shape.get("guided_depth", 1))
    rs.render(shape["spp"], max_bounces=shape["depth"], seed=shape["seed"],
              estimator=photon_gpu.BVPT if shape.get("bvpt") else photon_gpu.BNEEPT)


@pytest.mark.gpu
def test_switching_shapes_gives_a_fresh_scenes_film(gpu_lib):
    import photon_gpu

    scene = scenes.cornell_glossy(45, 23, 8, 8)   # 1,035 paths per sample
    shapes = [dict(spp=1, depth=8), dict(spp=9, depth=8), dict(spp=2, depth=3), dict(spp=2, depth=8, guided=True),
              dict(spp=5, depth=4, guided=True), dict(spp=5, depth=4, guided=True, guided_depth=0), dict(spp=3, depth=8, bvpt=True),
              dict(spp=40, depth=8), dict(spp=1, depth=1)]
    for capacity in (1024, 4096):   # sample counts on both sides of two pools of paths
        with photon_gpu.RenderScene(scene) as used:
            used.set_launch(capacity=capacity)
            for k, shape in enumerate(shapes + shapes[::-1] + shapes):
                shape = dict(shape, seed=k)
                used.clear()
                _render(used, shape)
                with photon_gpu.RenderScene(scene) as fresh:
                    fresh.set_launch(capacity=capacity)
                    _render(fresh, shape)
                    want = fresh.film()[1]
                # the same paths; the FP64 film adds them up in another order
                np.testing.assert_allclose(used.film()[1], want, rtol=1e-11, atol=1e-11 * np.abs(want).max())


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [[dict(spp=1, depth=8), dict(spp=2, depth=8)], [dict(spp=1, depth=4), dict(spp=1, depth=8)],
                                    [dict(spp=1, depth=d) for d in (2, 3, 4, 5, 6, 7)],
                                    [dict(spp=4, depth=8), dict(spp=4, depth=8, guided=True)]])
def test_alternating_shapes_cost_what_each_costs(gpu_lib, shapes):
    """Medians of 40 calls each, alternating against each shape on its own: a graph that is captured and
    instantiated anew, or a pool laid out anew, would add more than half of such a short call (bound: 30 % and
    30 us)."""
    import photon_gpu

    def timed(rs, sequence):
        out = []
        for k, shape in enumerate(sequence):
            t = time.perf_counter()
            _render(rs, dict(shape, seed=k))
            out.append(time.perf_counter() - t)
        return out

    with photon_gpu.RenderScene(scenes.cornell(64, 48, 1, 8)) as rs:
        alone = []
        for shape in shapes:
            timed(rs, [shape] * 5)
            alone.append(statistics.median(timed(rs, [shape] * 40)))
        mixed = timed(rs, shapes * 40)
        mixed = [statistics.median(mixed[k::len(shapes)]) for k in range(len(shapes))]
    for a, m in zip(alone, mixed):
        assert m <= 1.3 * a + 30e-6, (alone, mixed)
