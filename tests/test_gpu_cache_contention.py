"""Warps that come to the same groups while these are being cached: several views of
one camera share one table and one group cache, from cold to filled, with room for
none, a few and all of the groups; every frame equals the uncached one."""
import ctypes as ct

import pytest
import torch

import stratum_hyperdetail_b200 as sb

pytestmark = pytest.mark.gpu
W, H = 200, 113


@pytest.mark.parametrize("order", [1, 3])
@pytest.mark.parametrize("entries", [1, 37, 900, 30000])
def test_views_that_share_a_cache(cuda, entries, order):
    from stratum_hyperdetail_b200.views import View
    v = View(W, H)
    v.set_pose(5, (3, 0, 4, 0), (17.0, 30.0, 0.0), 0.6, -0.3)
    v.C[19] = 1.0
    n = 6
    s = torch.cuda.current_stream().cuda_stream

    def trace(times):
        hit = torch.zeros(n, W * H * 4, device="cuda")
        surface = torch.zeros_like(hit)
        rec = (sb.ViewRecord * n)()
        for i, r in enumerate(rec):
            for k in ("C", "Origin", "I", "World", "Tags", "Nodes", "Queue", "Linear", "History", "Pixels", "Groups"):
                setattr(r, k, sb.ptr(getattr(v, k)))
            r.Hit, r.Surface, r.width, r.height = sb.ptr(hit[i]), sb.ptr(surface[i]), W, H
        table = torch.frombuffer(bytearray(bytes(rec)), dtype=torch.uint8).cuda()
        size = int(sb.lib().stratum_batchScratchBytes(n))
        scratch = torch.zeros(size, dtype=torch.uint8, device="cuda")
        tune = sb.Tune(64, 1, order)
        for _ in range(times):
            hit.fill_(-5.0)
            surface.fill_(-5.0)
            sb.call("stratum_traceViews", sb.ptr(table), n, sb.ptr(scratch), size, ct.byref(tune), s)
            torch.cuda.synchronize()
            yield hit.clone(), surface.clone()

    want = next(trace(1))
    v.enable_group_cache(entries)
    for got in trace(11):  # a full cache starts again after eight
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert (want[0] == want[0][0]).all()
