"""Strips around the size from which the drop-in trace draws no band of narrow tiles in
them (0.6 of the blocks the device holds: 710 columns of 64 rows on 148 SMs), and their
last, shorter strips: the same bits as the whole frame."""
import pytest
import torch

from stratum_hyperdetail_b200 import call, ptr
from stratum_hyperdetail_b200.views import View

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(704, 130), (720, 130), (1024, 96), (1184, 65), (1185, 129)])
@pytest.mark.parametrize("pitch", [0.0, -0.7])
def test_strips_equal_the_frame(cuda, w, h, pitch):
    v = View(w, h)
    v.set_pose(99, (3, 0, 4, 0), (17.0, 25.0, 3.0), 0.4, pitch)
    v.C[19] = 1.0
    s = torch.cuda.current_stream().cuda_stream
    got = []
    for rows in (h, 64, 16):
        v.Hit.zero_()
        v.Surface.zero_()
        for y in range(0, h, rows):
            call("stratum_tracePrimary", ptr(v.World), ptr(v.Nodes), ptr(v.Origin), ptr(v.C), ptr(v.Hit), ptr(v.Surface),
                 w, h, y, min(rows, h - y), s)
        got.append((v.Hit.clone(), v.Surface.clone()))
    assert (got[0][0].view(-1, 4)[:, 0] > 0).all()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert torch.equal(a.view(torch.int32), b.view(torch.int32))
