"""Exhaustive rays: a slot that finishes takes the block's next ray, so what a ray
gives cannot depend on how many others it is traced with.  Each ray of a large
call against the same ray in calls of eight (one block, one ray to a slot)."""
import numpy as np
import pytest

from test_gpu_rays import some_rays, trace_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1185, 4003])
def test_exhaustive_rays_do_not_depend_on_their_number(cuda, count):
    from stratum_hyperdetail_b200.views import View
    v = View(64, 64)
    v.set_pose(77, (5, 0, 0xFFFFFFF9, 0xFFFFFFFF), (0.0, 2.0, 0.0), 0.0, 0.0)
    rays = some_rays(count)
    got = trace_rays(v, rays, True)
    want = np.concatenate([trace_rays(v, rays[i:i + 8], True) for i in range(0, count, 8)])
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
