"""Device memory that the library holds between calls: at most 512 MiB of per-call memory, none once the
last geometry or scene is gone, and none that an allocation of the library itself would miss.

Free memory is the device's own count (cudaMemGetInfo through torch); the slack of 64 MiB is for the
driver's granularity and for kernels loaded on the way."""

import numpy as np
import pytest

import scenes

MIB = 1 << 20
KEPT = 512 * MIB
SLACK = 64 * MIB


def _free():
    import torch

    return torch.cuda.mem_get_info()[0]


def _rays(n):
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = (278.0, 273.0, -800.0)
    rays[:, 6], rays[:, 7] = 1.0, 1e30
    return rays


def _geometry():
    import photon_gpu

    return photon_gpu.Geometry(np.concatenate([g.tris for g in scenes.cornell().groups]))


@pytest.mark.gpu
def test_a_large_query_gives_its_memory_back(gpu_lib):
    before_geometry = None
    for _ in range(2):   # (the first round loads the kernels)
        before_geometry = _free()
        with _geometry() as g:
            g.closest(_rays(16))
            before = _free()
            g.closest(_rays(16_000_000))   # 60 bytes of device memory each: 920 MiB
            assert before - _free() <= KEPT + SLACK
            g.closest(_rays(4_000_000))    # kept for the next call
            g.closest(_rays(16))
            assert before - _free() <= KEPT + SLACK
    assert before_geometry - _free() <= SLACK


@pytest.mark.gpu
def test_the_last_scene_takes_the_kept_memory_along(gpu_lib):
    import photon_gpu
    from oracle import guide_ref as ref

    params, feat = ref.init_params(1), np.full((1_000_000, 7), 0.5, np.float32)
    photon_gpu.guide_mixture(params, feat[:10])
    with photon_gpu.RenderScene(scenes.cornell(8, 8, 1, 2)) as rs:
        rs.render(1, max_bounces=2)
    before = _free()
    with photon_gpu.RenderScene(scenes.cornell(8, 8, 1, 2)):
        photon_gpu.guide_mixture(params, feat)
    assert before - _free() <= SLACK


@pytest.mark.gpu
def test_kept_memory_makes_room_for_a_scene(gpu_lib):
    """A path pool of 2^20 slots (some 340 MiB) where only the kept memory of a query leaves room for it."""
    import photon_gpu
    import torch

    scene = scenes.cornell(1024, 1024, 1, 2)
    with photon_gpu.RenderScene(scene) as rs:
        rs.set_launch(capacity=1 << 20)
        rs.render(1, max_bounces=2)
    with _geometry() as g, photon_gpu.RenderScene(scene) as rs:
        rs.set_launch(capacity=1 << 20)
        g.closest(_rays(16))
        torch.cuda.empty_cache()
        hog = torch.empty(_free() - 680 * MIB, dtype=torch.uint8, device="cuda")
        try:
            g.closest(_rays(7_000_000))   # 400 MiB, kept
            rs.render(1, max_bounces=2)
        finally:
            del hog
            torch.cuda.empty_cache()
