"""Frames whose rays run along the axes, and whole frames against strips.

A warp's rays are culled as one packet by the range of their inverse
directions; straight ahead along an axis that range spans both signs and the
guarded inverse of a zero component, and straight down every lot's boxes are
entered from above.  Each frame is compared with the oracle bit for bit, batched
(records from the grammar, then from the group cache) and through the drop-in
entry points (whole frame and 64-row strips)."""
import math

import numpy as np
import pytest
import torch

import oracle_lib as ol
from test_gpu_batch_oracle import check, host_frame

pytestmark = pytest.mark.gpu

SIZES = [(33, 17), (61, 241), (8, 65)]


@pytest.mark.parametrize("yaw,pitch,height", [
    (0.0, 0.0, 1.7), (math.pi / 2, 0.0, 12.0), (math.pi, 0.0, 3.0), (-math.pi / 2, -0.4, 40.0), (0.7, -1.53, 120.0)])
def test_axis_aligned_packets(cuda, oracle, yaw, pitch, height):
    from stratum_hyperdetail_b200.batch import Batch
    from stratum_hyperdetail_b200.views import View
    for k, (w, h) in enumerate(SIZES):
        origin, pos = (5 * k, 0, 8 * k, 0), (17.0 if k != 1 else 0.0, height, 0.0 if k != 1 else -17.5)
        v = View(w, h)
        v.set_pose(77 + k, origin, pos, yaw, pitch)
        with ol.device_angles(oracle):
            o = ol.setup_pose(oracle, 77 + k, pos, yaw, pitch, w, h, origin=origin)
            second = np.zeros(w * h, np.float32)
            want = ol.render(oracle, o, w, h, second=second)
        v.frame()
        check(f"{w}x{h} frame", host_frame(v), want, second)
        whole = host_frame(v)
        v.C[19] = 0.0
        v.History.zero_()
        v.frame_parts()
        parts = host_frame(v)
        for name in whole:
            assert np.array_equal(whole[name].view(np.uint32), parts[name].view(np.uint32)), name
        b = Batch([v], (64, 1, 1))
        for again in range(2):
            v.C[19] = 0.0
            v.History.zero_()
            b.frame()
            check(f"{w}x{h} batched {again}", host_frame(v), want, second)


@pytest.mark.parametrize("w,h,pitch", [(320, 180, 0.0), (640, 360, 0.9), (641, 363, -0.9), (1283, 121, -0.05), (5, 700, 0.02)])
def test_band_and_strips_draw_every_pixel_alike(cuda, w, h, pitch):
    """The horizon inside, above and below the frame, bands of none, some and all
    of its rows: whole frame, 64-row strips (no band) and batched, bit for bit."""
    from stratum_hyperdetail_b200.batch import Batch
    from stratum_hyperdetail_b200.views import View
    v = View(w, h)
    v.set_pose(99, (3, 0, 4, 0), (17.0, 25.0, 3.0), 0.4, pitch)
    kept = None
    b = Batch([v], (64, 2, 0))
    for draw in (v.frame, v.frame_parts, b.frame):
        v.C[19] = 0.0
        for t in (v.Hit, v.Surface, v.Linear, v.History, v.Pixels):
            t.zero_()
        draw()
        got = host_frame(v)
        if kept is None:
            kept = got
            assert (got["Hit"].reshape(-1, 4)[:, 0] > 0).all()  # every pixel was written
        for name in kept:
            assert np.array_equal(kept[name].view(np.uint32), got[name].view(np.uint32)), (draw, name)
