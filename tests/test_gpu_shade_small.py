"""Strips on both sides of the line between one shading launch and two (32 tiles an SM:
4,736 on 148), procedural and with the surrogate: a frame shaded at once has the same bits
as in strips of 8 rows."""
import pytest
import torch

from stratum_hyperdetail_b200 import call, ptr
from stratum_hyperdetail_b200.views import View, shade_launches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("surrogate", [False, True])
@pytest.mark.parametrize("w,h", [(1, 1), (7, 3), (65, 33), (512, 296), (512, 297), (513, 296), (640, 361)])
def test_small_and_large_strips_agree(cuda, w, h, surrogate):
    v = View(w, h)
    v.set_pose(99, (3, 0, 4, 0), (17.0, 12.0, 3.0), 0.4, -0.1)
    v.frame()
    s = torch.cuda.current_stream().cuda_stream
    net = [torch.zeros(n, device="cuda") for n in (291, 291, 291, 32)]
    call("stratum_initNeural", *map(ptr, net), 5, s)
    net[3][4] = 1.0
    v.C[16] = 1.0
    got = []
    for rows in (h, 8):
        v.Linear.fill_(-1.0)
        for y in range(0, h, rows):
            common = [ptr(t) for t in (v.World, v.Origin, v.C, v.Hit, v.Surface, v.Linear)]
            if surrogate:
                call("stratum_shadePixelsNeural", *common, ptr(net[0]), ptr(net[3]), w, h, y, rows, s)
            else:
                call("stratum_shadePixels", *common, w, h, y, rows, s)
        got.append(v.Linear.clone())
    assert torch.equal(got[0].view(torch.int32), got[1].view(torch.int32))
    assert (got[0].view(-1, 4)[:, 3] == 1.0).all()


def test_launch_counts(cuda):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert [shade_launches(8 * k, 4, "cuda") for k in (1, 32 * sms, 32 * sms + 1)] == [1, 1, 2]
