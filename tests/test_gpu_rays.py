"""Arbitrary rays against the oracle at the counts where the work split changes
(rays to a warp, rays and lots to a block, refills) and with rays that graze,
miss, start outside the city's slab, run along an axis or are not normalised;
hierarchy and exhaustive forms, every word bit for bit."""
import numpy as np
import pytest

import oracle_lib as ol
from test_gpu_streaming import trace_rays

pytestmark = pytest.mark.gpu


def some_rays(n):
    rng = np.random.default_rng(n)
    ro = np.stack([rng.uniform(-700, 700, n), rng.uniform(0.2, 90.0, n), rng.uniform(-700, 700, n)], 1)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    kind = rng.integers(0, 10, n)
    d[kind == 0, 0] = 0.0
    d[kind == 1, 2] = -0.0
    d[kind == 2, 1] = 0.0
    ro[kind == 3, 1] += 400.0
    ro[kind == 4, 1] = -20.0
    d[kind == 5] *= rng.uniform(0.1, 3.0, (int((kind == 5).sum()), 1))
    d[kind == 6] = [0.0, -1.0, 0.0]
    return np.concatenate([ro, d, rng.uniform(0.0, 0.01, (n, 1))], 1).astype(np.float32)


@pytest.mark.parametrize("exhaustive,count", [(False, n) for n in (1, 31, 32, 33, 2500, 9000)]
                         + [(True, n) for n in (1, 7, 8, 9, 1300)])
def test_rays_against_oracle(cuda, oracle, exhaustive, count):
    from stratum_hyperdetail_b200.views import View
    origin = (0xFFFFFFF0, 0, 90, 0)
    v = View(64, 64)
    v.set_pose(4321, origin, (0.0, 2.0, 0.0), 0.0, 0.0)
    o = ol.setup_pose(oracle, 4321, (0.0, 2.0, 0.0), 0.0, 0.0, 64, 64, origin=origin)
    rays = some_rays(count)
    got = trace_rays(v, rays, exhaustive)
    want = oracle.trace_rays(o.World, o.Nodes, o.Origin, rays, exhaustive)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert count < 100 or (want[:, 1] >= 0).sum() > count // 10
