"""The hierarchy build against the oracle where its eight-lot units and its two
ways of bounding a group can go wrong: queue lengths around the unit and tables
of edited rows (dimensions no described lot has, next to described ones)."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
from gpu_lib import s, u32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [0, 1, 7, 8, 9, 63, 1185])
@pytest.mark.parametrize("edited", [False, True])
def test_build_of_queues_and_edited_rows(cuda, oracle, count, edited):
    from stratum_hyperdetail_b200 import call, ptr
    o = ol.setup_pose(oracle, 1234, (0.0, 2.0, 0.0), 0.0, 0.0, 64, 64, origin=(20, 0, 3, 0))
    rng = np.random.default_rng(count)
    world = o.World.reshape(-1, 16).copy()
    if edited:
        for word, value in ((0, 3.0), (1, 30.0), (2, 5.0), (3, 4.0), (3, 3.0), (5, 7.0), (7, 1.0), (8, 2.0)):
            world[rng.integers(0, 16384, 2500), word] = value
    queue = np.zeros(16385, np.uint32)
    queue[0] = count
    queue[1:count + 1] = rng.permutation(16384)[:count]
    o.World[:] = world.reshape(-1)
    o.Queue[:] = queue
    o.Nodes[:] = -7.0
    oracle.build_bounds(o.Queue, o.World, o.Nodes)
    W, Q = torch.from_numpy(world.reshape(-1)).cuda(), torch.from_numpy(queue.view(np.int32)).cuda()
    for drop_in in (False, True):
        N = torch.full((16384 * 128 * 8,), -7.0, device="cuda")
        if drop_in:
            for c in range(8):
                call("stratum_buildGroupBounds", ptr(Q), ptr(W), ptr(N), c * 2048, s())
                for first in (32, 16, 8, 4, 2, 1):
                    call("stratum_reduceGroupBounds", ptr(Q), ptr(N), first, c * 2048, s())
        else:
            call("stratum_buildBVH", ptr(Q), ptr(W), ptr(N), s())
        torch.cuda.synchronize()
        assert np.array_equal(u32(N), o.Nodes.view(np.uint32))
