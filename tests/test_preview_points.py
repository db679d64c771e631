"""Progress points of short renders: a render that takes more than eight iterations of the render loop
publishes its first preview after eight, also when sixteen would be its end."""

import pytest

import scenes
from test_progressive import _engine


@pytest.mark.gpu
@pytest.mark.parametrize("width,height,depth", [(64, 48, 8), (129, 97, 11)])
def test_short_render_publishes_a_preview(gpu_lib, tmp_path, width, height, depth):
    import photon_gpu

    eng = _engine(tmp_path, scenes.cornell(width, height, 1, depth))   # a pool holds all paths
    eng.render()
    status = [r[4] for r in eng.poll_regions(64)]
    iterations = eng.profile(2, 1)["iterations"]
    eng.close()
    assert 9 <= iterations <= 16, iterations
    assert status == [photon_gpu.REGION_UPDATING, photon_gpu.REGION_FINISHED]
