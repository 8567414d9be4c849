"""Shading and resolve where the shortcuts change over, against the oracle: frames
so small or far that every frequency weight falls to 0, so close that none does,
looking into the sun, from above every roof, and with the contact-occlusion taps
reaching over creases and silhouettes; batched and drop-in, colour to 1e-5."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
from test_gpu_batch_oracle import check, host_frame

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pos,yaw,pitch,w,h", [
    ((17.0, 1.7, 0.0), 0.0, 0.0, 40, 9), ((13.2, 5.0, 0.0), -1.2, 0.1, 97, 301), ((0.0, 300.0, 0.0), 0.6, -0.9, 120, 67),
    ((17.0, 30.0, 0.0), -1.02, 0.45, 64, 64), ((16.0, 0.3, 15.0), 2.2, -0.3, 83, 200), ((10.0, 12.0, 10.0), 0.8, -1.4, 51, 77)])
def test_shading_changeovers(cuda, oracle, pos, yaw, pitch, w, h):
    from stratum_hyperdetail_b200.batch import Batch
    from stratum_hyperdetail_b200.views import View
    v = View(w, h)
    v.set_pose(2024, (4, 0, 9, 0), pos, yaw, pitch)
    with ol.device_angles(oracle):
        o = ol.setup_pose(oracle, 2024, pos, yaw, pitch, w, h, origin=(4, 0, 9, 0))
        second = np.zeros(w * h, np.float32)
        want = ol.render(oracle, o, w, h, second=second)
    for draw in (v.frame, Batch([v]).frame):
        v.C[19] = 0.0
        v.History.zero_()
        draw()
        torch.cuda.synchronize()
        got = host_frame(v)
        check("shading", got, want, second)
        # transcendentals differ by a few ulp between the two; a term left out would not
        for name in ("Linear", "History"):
            assert np.abs(got[name] - want[name]).max() < 1e-4, name
