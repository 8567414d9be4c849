"""The block-pooled trace over more views than 11 and 12 bits number: every view of
one camera shows what the first shows, and what the per-warp trace shows."""
import ctypes as ct

import pytest
import torch

import stratum_hyperdetail_b200 as sb

pytestmark = pytest.mark.gpu
W, H = 8, 4


@pytest.mark.parametrize("n,threads", [(2048, 64), (2050, 128), (4099, 64)])
def test_pooled_trace_of_many_views(cuda, n, threads):
    from stratum_hyperdetail_b200.views import View
    v = View(W, H)
    v.set_pose(5, (3, 0, 4, 0), (17.0, 2.0, 0.0), 0.6, 0.05)
    v.C[19] = 1.0
    frames = [(torch.zeros(n, W * H * 4, device="cuda"), torch.zeros(n, W * H * 4, device="cuda")) for _ in range(2)]
    for order, (hit, surface) in zip((0, 2), frames):
        rec = (sb.ViewRecord * n)()
        for i, r in enumerate(rec):
            for k in ("C", "Origin", "I", "World", "Tags", "Nodes", "Queue", "Linear", "History", "Pixels"):
                setattr(r, k, sb.ptr(getattr(v, k)))
            r.Hit, r.Surface = hit.data_ptr() + i * W * H * 16, surface.data_ptr() + i * W * H * 16
            r.width, r.height = W, H
        table = torch.frombuffer(bytearray(bytes(rec)), dtype=torch.uint8).cuda()
        size = int(sb.lib().stratum_batchScratchBytes(n))
        scratch = torch.zeros(size, dtype=torch.uint8, device="cuda")
        tune = sb.Tune(threads, 1, order)
        sb.call("stratum_traceViews", sb.ptr(table), n, sb.ptr(scratch), size, ct.byref(tune),
                torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    assert (frames[0][0][0, 1::4] >= 0).sum() > W * H // 2
    for plain, pooled in zip(*frames):
        assert (plain == plain[0]).all()
        assert torch.equal(pooled, plain)
