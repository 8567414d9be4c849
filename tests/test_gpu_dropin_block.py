"""The drop-in trace's block table: warps of a block that come to one group together
build it once, those that come later read it, and groups beyond the table's
entries are built by each warp.  Blocks alone, ragged and many, from a pose
with few groups to a block and from one with more than the table holds, against
the oracle bit for bit; again and again, since the order of the warps varies."""
import numpy as np
import pytest

import oracle_lib as ol
from test_gpu_batch_oracle import check, host_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(16, 16), (17, 15), (40, 50), (160, 90)])
@pytest.mark.parametrize("pos,pitch", [((17.0, 1.7, 0.0), 0.0), ((0.0, 300.0, 0.0), -0.5), ((0.0, 900.0, 0.0), -1.2)])
def test_block_table(cuda, oracle, w, h, pos, pitch):
    from stratum_hyperdetail_b200.views import View
    v = View(w, h)
    v.set_pose(0x5EED, (0, 0, 0, 0), pos, 0.6, pitch)
    with ol.device_angles(oracle):
        o = ol.setup_pose(oracle, 0x5EED, pos, 0.6, pitch, w, h, origin=(0, 0, 0, 0))
        second = np.zeros(w * h, np.float32)
        want = ol.render(oracle, o, w, h, second=second)
    for _ in range(4):
        v.C[19] = 0.0
        v.History.zero_()
        v.frame()
        check(f"{w}x{h}", host_frame(v), want, second)
