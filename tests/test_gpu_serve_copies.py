"""Frames reach a request's memory whole: sizes around the helper threads' 1 MiB
pieces, requests queued behind one another on a session, many sessions at once, and
requests without a buffer; each frame equals the session's device frame."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (512, 512), (513, 512), (512, 511), (1024, 769)])
def test_served_frames_are_whole(cuda, w, h):
    from stratum_hyperdetail_b200.server import Pose, Server
    srv = Server(8 << 30, 4, 3, group_cache=1024)
    sids = [srv.open(50 + i, w, h) for i in range(6)]
    for step in range(3):
        out = [np.full(w * h, 0x01020304, np.uint32) for _ in sids]
        first = [np.zeros(w * h, np.uint32) for _ in sids]
        poses = [Pose.make((i, 0, step, 0), (17.0, 2.0 + i, 0.0), 0.3 * i, 0.0) for i in range(len(sids))]
        rids = []
        for i, s in enumerate(sids):  # two queued on each session: the second accumulates on the first
            rids.append(srv.submit(s, poses[i], 1, first[i]))
            rids.append(srv.submit(s, poses[i], 2, out[i] if i != 3 else None))
        for r in rids:
            assert srv.wait_status(r, 60000) == 0
        for i, s in enumerate(sids):
            px, _ = srv.read(s)
            if i != 3:
                assert np.array_equal(out[i], px), (step, i)
            assert (first[i] >> 24 == 255).all()
    srv.close()
