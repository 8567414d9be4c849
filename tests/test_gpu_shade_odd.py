"""Shading where its shortcuts must not be taken, against the oracle: hits at an
infinite distance, whose noise is no number (so is the colour, unless fog covers it
or the material has no noise), and a table with masses below the ground."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
from stratum_hyperdetail_b200 import call, ptr

pytestmark = pytest.mark.gpu
W, H = 150, 91


def both_ways(v, o, oracle):
    """Linear of the drop-in, of the batched pass, and of the oracle, for v's Hit and Surface."""
    from stratum_hyperdetail_b200.batch import Batch
    s = torch.cuda.current_stream().cuda_stream
    hit, surface = v.Hit.clone(), v.Surface.clone()
    call("stratum_shadePixels", ptr(v.World), ptr(v.Origin), ptr(v.C), ptr(hit), ptr(surface), ptr(v.Linear), W, H, 0, H, s)
    dropin = v.Linear.cpu().numpy().copy()
    b = Batch([v], group_cache=0)
    b.trace()
    v.Hit.copy_(hit)
    v.Surface.copy_(surface)
    b.shade()
    batched = v.Linear.cpu().numpy()
    want = np.zeros(W * H * 4, np.float32)
    oracle.shade(o.World, o.Origin, o.C, hit.cpu().numpy(), surface.cpu().numpy(), want, W, H)
    return dropin, batched, want


def setup(oracle, pos, pitch):
    from stratum_hyperdetail_b200.views import View
    v = View(W, H)
    v.set_pose(7, (3, 0, 4, 0), pos, 0.6, pitch)
    v.C[19] = 1.0
    o = ol.setup_pose(oracle, 7, pos, 0.6, pitch, W, H, origin=(3, 0, 4, 0))
    call("stratum_tracePrimary", ptr(v.World), ptr(v.Nodes), ptr(v.Origin), ptr(v.C), ptr(v.Hit), ptr(v.Surface), W, H, 0, H,
         torch.cuda.current_stream().cuda_stream)
    return v, o


@pytest.mark.parametrize("t", [float("inf"), -float("inf"), float("nan"), 1e38])
def test_hits_that_are_not_finite(cuda, oracle, t):
    with ol.device_angles(oracle):
        v, o = setup(oracle, (17.0, 30.0, 0.0), -0.3)
        far = torch.from_numpy(np.random.default_rng(1).random(W * H) < 0.5).cuda()
        v.Hit.view(-1, 4)[:, 0][far] = t
        hits = v.Hit.view(-1, 4)[:, 1].cpu().numpy() != -10000
        dropin, batched, want = both_ways(v, o, oracle)
    no_number = np.isnan(want.reshape(-1, 4)[:, :3]).any(1)
    assert (no_number & hits).sum() > 1000
    for got in (dropin, batched):
        assert np.array_equal(np.isnan(got), np.isnan(want))


def test_masses_below_the_ground(cuda, oracle):
    with ol.device_angles(oracle):
        v, o = setup(oracle, (17.0, 2.0, 0.0), 0.0)
        rows = o.World.reshape(-1, 16)
        rows[np.random.default_rng(2).integers(0, 16384, 8000), 2] = -40.0
        v.World.copy_(torch.from_numpy(o.World))
        dropin, batched, want = both_ways(v, o, oracle)
    for got in (dropin, batched):
        assert np.abs(got - want).max() < 1e-4
